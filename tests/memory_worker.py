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


if __name__ == "__main__":
    {"velocity": velocity}[sys.argv[1]]()
    print("OK")
