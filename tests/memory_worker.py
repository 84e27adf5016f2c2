"""Device memory of single calls, each in a process of its own (started by test_gpu_s_memory.py): what a call may take, and
what it does when little is left."""
import ctypes as C
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from conftest import load_package  # noqa: E402

pkg = load_package()
MB = 1 << 20


def free_bytes():
    rt = C.CDLL("libcudart.so.12")
    f, t = C.c_size_t(0), C.c_size_t(0)
    assert rt.cudaMemGetInfo(C.byref(f), C.byref(t)) == 0
    return f.value


def velocity():
    """Velocity calls need the acoustic weights alone, and no copies of the decoder's (6 GB)."""
    eng = pkg.Engine(kv_cache_max=64)
    x, h = pkg.synth_f32(36, 5, "mem.x"), pkg.synth_f32(3072, 5, "mem.h")

    def calls():
        before = free_bytes()
        v = [eng.predict_velocity(x, h, t) for t in (0.0, 0.25, 0.5)]     # launches, capture, graph
        assert before - free_bytes() < 64 * MB, (before, free_bytes())
        return np.stack(v)

    eng.upload(pkg.SynthModel(seed=77, decoder=False, audio_table=False), decoder=False, acoustic=True)
    alone = calls()
    eng.upload(pkg.SynthModel(seed=77, acoustic=False, audio_table=False, dec_layers=1), decoder=True, acoustic=False)
    assert np.array_equal(calls(), alone)                                 # the same launches on the same weights


def step():
    """The decoder step needs none of the copies (6 GB), and what it gives does not depend on whether they are there."""
    eng = pkg.Engine(kv_cache_max=64)
    eng.upload(pkg.SynthModel(seed=77, dec_layers=1), audio_table=True)
    x = pkg.synth_f32((9, 3072), 5, "mem.rows", 0.0, 0.5)
    before = free_bytes()
    alone = [eng.llm_forward(e, p) for p, e in enumerate(x)]
    assert before - free_bytes() < 64 * MB, (before, free_bytes())
    eng.prefill(x, 40)
    for _ in range(3):                                                    # launches, capture, graph, if it were one
        assert all(np.array_equal(eng.llm_forward(e, p), a) for p, (e, a) in enumerate(zip(x, alone)))


def take(eng, leave):
    """All of the device's memory but `leave` bytes."""
    p = eng.L.tts_cuda_alloc(free_bytes() - leave)
    assert p and free_bytes() < leave + 64 * MB
    return p


def copies():
    """A prefill that finds no room for the decoder's tile-contiguous copies does without, and keeps none of them."""
    eng = pkg.Engine(kv_cache_max=64)
    eng.upload(pkg.SynthModel(seed=77, acoustic=False, audio_table=False, dec_layers=1), decoder=True, acoustic=False)
    x = pkg.synth_f32((9, 3072), 5, "mem.rows", 0.0, 0.5)
    full = take(eng, 2048 * MB)
    before, rows = free_bytes(), []
    for _ in range(2):
        eng.prefill(x, 0)
        assert before - free_bytes() < 64 * MB, (before, free_bytes())
        rows.append(np.stack([eng.kv_read(l, 0, 9) for l in (0, 25)]))
    assert np.array_equal(*rows)
    eng.L.tts_cuda_free_ptr(full)
    eng.prefill(x, 0)
    got = np.stack([eng.kv_read(l, 0, 9) for l in (0, 25)])
    assert np.linalg.norm(got - rows[0]) < 1e-4 * np.linalg.norm(got)     # sums in other orders


def far():
    """Prompt rows behind more cache rows than a grid's y axis has places, against the decoder step row by row. The earlier
    rows that count are a few on both sides: keys large enough that the zeros between them have no weight. Scores of up
    to 20 as two-term products (2^-16 of a product's size) set the limit."""
    first, n = 65537, 3
    eng = pkg.Engine(kv_cache_max=first + 63)
    eng.upload(pkg.SynthModel(seed=77, acoustic=False, audio_table=False, dec_layers=2), decoder=True, acoustic=False)
    for at in (0, first - 100):
        for l in range(26):
            eng.kv_write(l, at, pkg.synth_f32((100, 1024), 100 * l + 1, f"far.k{at}", 0.0, 5.0), pkg.synth_f32((100, 1024), 100 * l + 2, f"far.v{at}"))
    x = pkg.synth_f32((n, 3072), 5, "far.rows", 0.0, 0.5)
    eng.prefill(x, first)
    got = [eng.kv_read(l, first, n) for l in (0, 1, 25)]
    for i in range(n):
        eng.llm_forward(x[i], first + i)
    for l, (k, v) in zip((0, 1, 25), got):
        k2, v2 = eng.kv_read(l, first, n)
        assert np.linalg.norm(k - k2) < 1e-3 * np.linalg.norm(k2) and np.linalg.norm(v - v2) < 1e-3 * np.linalg.norm(v2), l


def short():
    """A prompt with less and less memory left: smaller blocks of rows, then the streaming kernel; the same cache rows, up to
    the order of sums and 16-bit halves, as with room for all."""
    n, small = 600, 200
    eng = pkg.Engine(kv_cache_max=640)
    eng.upload(pkg.SynthModel(seed=77, acoustic=False, audio_table=False, dec_layers=2), decoder=True, acoustic=False)
    x = pkg.synth_f32((n, 3072), 5, "short.rows", 0.0, 0.5)

    def rows(m):
        eng.kv_write(25, 0, np.zeros((n, 1024), np.float32), np.zeros((n, 1024), np.float32))
        eng.prefill(x[:m], 0)
        return np.concatenate(eng.kv_read(25, 0, m), axis=1)

    eng.prefill(x[:5], 0)                             # the decoder's copies are made
    full, got = take(eng, 200 * MB), []
    for leave, m in ((30, small), (60, small), (100, n), (130, n), (200, n)):
        eng.L.tts_cuda_free_ptr(full)
        full = take(eng, leave * MB)
        got.append((leave, rows(m)))
    eng.L.tts_cuda_free_ptr(full)
    want = rows(n)
    for leave, g in got:
        w = want[:len(g)]
        assert np.linalg.norm(g - w) < 1e-4 * np.linalg.norm(w), (leave, len(g))


def blocks():
    """A prompt of more rows than go through a layer at once: the same bits as those blocks in calls of their own, and up to
    the order of sums the rows of calls cut elsewhere."""
    eng = pkg.Engine(kv_cache_max=4500)
    eng.upload(pkg.SynthModel(seed=77, acoustic=False, audio_table=False, dec_layers=2), decoder=True, acoustic=False)
    for n, calls in ((2300, (2048, 252)), (2048 + 40, (2048, 40)), (2048 + 256 + 9, (2048, 256, 9)), (4400, (2048, 2048, 304 - 48, 48))):
        x = pkg.synth_f32((n, 3072), 5, "blocks.rows", 0.0, 0.5)

        def rows(sizes):
            at = 0
            for m in sizes:
                eng.prefill(x[at:at + m], at)
                at += m
            assert at == n
            return np.stack([np.concatenate(eng.kv_read(l, 0, n), axis=1) for l in (0, 1, 25)])

        whole = rows((n,))
        assert np.array_equal(rows(calls), whole), calls
        other = rows((700, n - 700))
        for l in range(3):
            assert np.linalg.norm(other[l] - whole[l]) < 1e-4 * np.linalg.norm(whole[l]), (n, l)


if __name__ == "__main__":
    {"velocity": velocity, "step": step, "copies": copies, "far": far, "short": short, "blocks": blocks}[sys.argv[1]]()
    print("OK")
