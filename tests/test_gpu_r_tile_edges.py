"""Kernels at the edges of their tiles and of the rules that choose them, against the plain statements and the oracle."""
import numpy as np
import pytest

import lm_plain as plain
from lm_models import LIMIT, Case, attention, config, delta, error, feed, latent, tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 16, 17, 32, 33, 64, 65])
def test_float32_gemm_rows(pkg, tmp_path, rows):
    """Portions on both sides of the change from the skinny GEMM to the row-block one (16 and 17 rows) and of what a tile takes;
    widths that are no whole blocks of 64 columns and that split K. The limit is the 32-bit mode's: summation order."""
    c = Case(pkg, tmp_path, config([delta(ff=1300), attention(ff=60)], width=1100, vocab=301), seed=rows)
    toks = tokens(c.cfg, rows + 70, rows)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("float32") as lm:
        s = lm.open()
        assert error(feed(lm, s, toks, [rows, 70]), want) < LIMIT["float32"]


@pytest.mark.parametrize("width", [5120, 8200])
def test_float32_wide_few_rows(pkg, tmp_path, width):
    """A gated feed-forward of the 32-bit mode keeps one K split, so that each of a launch's ten sums takes 8 and 13 blocks of 64
    columns here. The logits are no further off than in portions of 17 rows, whose sums take two blocks: both within the
    mode's limit, which is twenty times what they show."""
    c = Case(pkg, tmp_path, config([delta(heads=2, kv_heads=1, dim=32, vdim=32, ff=200)], width=width, vocab=101), seed=3)
    toks = tokens(c.cfg, 34, 15)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("float32") as lm:
        for sizes in ([1], [5], [16], [17]):
            s = lm.open()
            assert error(feed(lm, s, toks, sizes), want) < LIMIT["float32"], sizes
            lm.release(s)


@pytest.mark.parametrize("rows", [65, 96, 97, 128, 129, 255, 256, 257, 300])
def test_row_block_gemm_rows(pkg, tmp_path, rows):
    """Rows on both sides of the row blocks' edges; matrices of one tile, of odd numbers of tiles and of tiles that are
    not full, alone and with an activation in the epilogue. The limit is the two-term products'."""
    c = Case(pkg, tmp_path, config([attention(ff=60, window=0), delta(ff=330)], width=392, vocab=301), seed=rows)
    toks = tokens(c.cfg, rows, rows)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("bfloat16") as lm:
        assert error(lm.step(lm.open(), toks, range(rows)), want) < LIMIT["bfloat16"]


PROMPT_ATTENTION = {
    # heads of one, two and three 64-column blocks, sizes that end inside a step of 16; pairs that fill a tile of 128
    # unevenly; windows and kept tokens on both sides of a 64-key tile
    "128": attention(heads=8, kv_heads=2, dim=128, vdim=128, window=0, rot=64, scale=0.09, softcap=0, ff=0),
    "64_8": attention(heads=4, kv_heads=4, dim=64, vdim=8, window=65, keep=3, ff=0),
    "72_128": attention(heads=6, kv_heads=2, dim=72, vdim=128, window=64, keep=64, scale=0.12, ff=0),
    "24_72": attention(heads=5, kv_heads=1, dim=24, vdim=72, window=63, keep=1, ff=0),
    "8_64": attention(heads=3, kv_heads=3, dim=8, vdim=64, window=130, keep=70, rot=8, ff=0),
    # whole columns of 64, so that tiles come by TMA, on rings that wrap inside a tile
    "64_128_wraps": attention(heads=4, kv_heads=2, dim=64, vdim=128, window=100, keep=5, ff=0),
    "128_64_wraps": attention(heads=6, kv_heads=2, dim=128, vdim=64, window=90, keep=0, scale=0.09, ff=0),
    "latent_128_64_wraps": latent(heads=2, dim=64, rot_dim=64, vdim=64, kv_rank=72, window=100, scale=0.09, ff=0),
    "latent_192_128_wraps": latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=64, window=77, scale=0.08, ff=0),
    "latent_192_128": latent(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=64, window=0, scale=0.08, ff=0),
    "latent_136_72": latent(heads=3, dim=72, rot_dim=64, vdim=72, window=65, scale=0.09, ff=0),
    "latent_176_16": latent(heads=2, dim=168, rot_dim=8, vdim=16, window=64, scale=0.08, ff=0),
    "latent_88_64": latent(heads=3, dim=80, rot_dim=8, vdim=64, window=127, scale=0.1, ff=0),
    "latent_16_8": latent(heads=7, dim=8, rot_dim=8, vdim=8, window=129, ff=0),
}


@pytest.mark.parametrize("name", list(PROMPT_ATTENTION))
def test_prompt_attention_tiles(pkg, tmp_path, name):
    """Row tiles, key tiles and head sizes of the prompt attention. The limit is the two-term products'."""
    c = Case(pkg, tmp_path, config([PROMPT_ATTENTION[name]]), seed=len(name))
    toks = tokens(c.cfg, 420, 4)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("bfloat16", block_rows=256) as lm:
        for sizes in ([420], [65, 128, 17, 33], [31, 63]):
            s = lm.open()
            assert error(feed(lm, s, toks, sizes), want) < LIMIT["bfloat16"], sizes
            lm.release(s)


@pytest.mark.parametrize("dim,rot_dim", [(128, 64), (168, 8), (120, 64)])
@pytest.mark.parametrize("window", [0, 130])
def test_heads_of_three_blocks(pkg, tmp_path, dim, rot_dim, window):
    """Heads of 192, 176 and 184, whose low query halves lie in shared memory: one to seven key tiles, the last of one key, of 63 and
    whole, by TMA (192) and without, full and nearly empty row tiles."""
    c = Case(pkg, tmp_path, config([latent(heads=2, dim=dim, rot_dim=rot_dim, vdim=128, kv_rank=64, window=window, scale=0.08, ff=0)]), seed=dim)
    toks = tokens(c.cfg, 449, 16)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("bfloat16", block_rows=256) as lm:
        for sizes in ([64], [127, 129], [63, 65, 128], [255, 194], [191, 17, 241]):
            s = lm.open()
            assert error(feed(lm, s, toks, sizes), want) < LIMIT["bfloat16"], sizes
            lm.release(s)


@pytest.mark.parametrize("dtype", list(LIMIT))
@pytest.mark.parametrize("heads,kv_heads,dim,change", [(64, 64, 8, 320), (40, 20, 16, 640), (3, 1, 20, 1280), (80, 80, 8, 160), (10, 2, 16, 160)])
def test_one_token_attention_changes_kernel(pkg, tmp_path, heads, kv_heads, dim, change, dtype):
    """Tokens one at a time on both sides of the length from which an unwindowed layer takes the kernel for many keys (none of
    its own for few in the last two), beside a layer whose window keeps it where it is; the device's own loop makes the
    change at the same token."""
    c = Case(pkg, tmp_path, config([attention(heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, window=0, rot=8, ff=0),
                                    attention(heads=4, kv_heads=2, dim=16, vdim=16, window=70, keep=3, rot=8, ff=0)]), seed=dim)
    n = change - 9
    toks = tokens(c.cfg, n + 20, 12)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open(dtype) as lm:
        s = lm.open()
        assert error(lm.step(s, toks[:n], [n - 1]), want[n - 1:n]) < LIMIT[dtype]
        assert error(feed(lm, s, toks[n:], [1]), want[n:]) < LIMIT[dtype]
        lm.release(s)
        s = lm.open()
        loop = lm.generate(s, toks[:n], 20)
        lm.release(s)
        s, host = lm.open(), []
        z = lm.step(s, toks[:n], [n - 1])
        for _ in range(20):
            host.append(int(z[0].argmax()))
            z = lm.step(s, host[-1:], [0])
        assert loop == host


@pytest.mark.parametrize("dtype", list(LIMIT))
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(40, 40, 16, 8), (20, 20, 20, 36), (64, 32, 32, 64), (8, 2, 64, 68), (3, 3, 132, 12), (2, 1, 30, 31)])
def test_few_rows_tiles(pkg, tmp_path, heads, kv_heads, dim, vdim, dtype):
    """A few rows at a time: heads of which a warp takes eight, four, two or one at once, whole and with lanes to spare, on both sides
    of the change from tiles of 32 keys to 64 (at 129 to 193 keys for the first three)."""
    c = Case(pkg, tmp_path, config([attention(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, window=0, rot=4, ff=0)]), seed=dim)
    toks = tokens(c.cfg, 215, 13)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open(dtype) as lm:
        for sizes in ([2], [3, 8, 5, 1, 30], [120, 7]):
            s = lm.open()
            assert error(feed(lm, s, toks, sizes), want) < LIMIT[dtype], sizes
            lm.release(s)


@pytest.mark.parametrize("dim,rot_dim,vdim", [(128, 64, 128), (64, 16, 64), (40, 8, 72)])
@pytest.mark.parametrize("q_rank", [56, 200, 700])
def test_latent_queries_in_parts(pkg, tmp_path, dim, rot_dim, vdim, q_rank):
    """Portions of 17 to 64 rows, whose queries come in one part, in a few and in as many as a K of eleven blocks is split into."""
    c = Case(pkg, tmp_path, config([latent(heads=3, dim=dim, rot_dim=rot_dim, vdim=vdim, q_rank=q_rank, kv_rank=64, window=0, scale=0.08, ff=0)]),
             seed=q_rank)
    toks = tokens(c.cfg, 200, 14)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("bfloat16") as lm:
        for sizes in ([64, 17], [33, 24], [130, 70]):
            s = lm.open()
            assert error(feed(lm, s, toks, sizes), want) < LIMIT["bfloat16"], sizes
            lm.release(s)


@pytest.mark.parametrize("first,rows", [(1, 64), (65, 31), (100, 129), (7, 300)])
def test_prefill_attention_tiles(pkg, engine, synth_model, first, rows):
    """A prompt in two calls against the same rows at once. Both are two-term products; a row's sums end in other
    orders, and what that does to a layer's rows grows over the layers that follow: the limit of the chunking test."""
    x = pkg.synth_f32((first + rows, 3072), 51, "edge.rows", 0.0, 0.5)
    engine.prefill(x, 0)
    whole = [engine.kv_read(l, 0, first + rows) for l in (0, 1, 25)]
    if first:
        engine.prefill(x[:first], 0)
    engine.prefill(x[first:], first)
    for (k1, v1), l in zip(whole, (0, 1, 25)):
        k2, v2 = engine.kv_read(l, 0, first + rows)
        assert np.linalg.norm(k2 - k1) < 1e-4 * np.linalg.norm(k1) and np.linalg.norm(v2 - v1) < 1e-4 * np.linalg.norm(v1), l


@pytest.mark.parametrize("rows", [257, 300, 320])
def test_prefill_last_rows_keep_three_terms(pkg, engine, synth_model, rows):
    """Up to 64 rows behind a multiple of 256 are multiplied with all the bits that 64 rows alone are: the same bits come
    out as from a call of their own."""
    x = pkg.synth_f32((rows, 3072), 52, "last.rows", 0.0, 0.5)
    engine.prefill(x, 0)
    whole = [engine.kv_read(l, 0, rows) for l in (0, 1, 25)]
    engine.prefill(x[:256], 0)
    engine.prefill(x[256:], 256)
    for (k1, v1), l in zip(whole, (0, 1, 25)):
        k2, v2 = engine.kv_read(l, 0, rows)
        assert np.array_equal(k2, k1) and np.array_equal(v2, v1), l


@pytest.mark.parametrize("rows", [2, 8, 9, 16, 17, 48, 64])
@pytest.mark.parametrize("K,N", [(64, 200), (576, 128), (1088, 9600), (3072, 9600)])
def test_skinny_gemm_sums_stay_short(pkg, engine, rows, K, N):
    """Products of one sign: the worst case for sums that are cut off at every step. Up to 16 rows TMEM adds one half of K
    and then the other, 16 columns a step: every cut at most 2^-23 of a sum that is half its final size on the average,
    and the two are added with a rounding, as are the terms. (9600 columns leave no K splits.)"""
    x = np.abs(pkg.synth_f32((rows, K), 53, "sum.x", 0.0, 1.0))
    W = pkg.synth_bf16((N, K), 54, "sum.W") & 0x7FFF
    dx, dW, dy = pkg.DeviceBuffer(x), pkg.DeviceBuffer(W), pkg.DeviceBuffer(nbytes=rows * N * 4)
    engine.L.tts_cuda_linear_bf16(dy.ptr, dx.ptr, None, rows, K, N, dW.ptr)
    got = dy.get((rows, N))
    want = x.astype(np.float64) @ (W.astype(np.uint32) << 16).view(np.float32).astype(np.float64).T
    off = np.abs(got / want - 1.0).max()
    for d in (dx, dW, dy):
        d.free()
    steps = 4 * ((K // 64 + 1) // 2 if rows <= 16 else K // 64)
    assert off < steps / 2 * 2.0 ** -23 + 4 * 2.0 ** -24, off


def _velocity64(t, x, hidden, time):
    """predict_velocity (voxtral_tts_acoustic.c:182-262) in 64 bits: three tokens, three layers, the head of the first."""
    p = "acoustic_transformer"

    def mul(a, name):
        return a @ (t[f"{name}.weight"].astype(np.uint32) << 16).view(np.float32).T.astype(np.float64)

    def rms(a, name):
        return a / np.sqrt((a * a).mean(-1, keepdims=True) + 1e-5) * t[f"{name}.weight"].astype(np.float64)
    angle = (np.float32(time) * t[f"{p}.time_embedding.inv_freq"]).astype(np.float32)
    temb = np.concatenate([np.cos(angle), np.sin(angle)]).astype(np.float64)
    y = np.stack([mul(x.astype(np.float64), f"{p}.input_projection"), mul(temb, f"{p}.time_projection"),
                  mul(hidden.astype(np.float64), f"{p}.llm_projection")])
    for l in range(3):
        n = f"{p}.layers.{l}"
        h = rms(y, f"{n}.attention_norm")
        q, k, v = (mul(h, f"{n}.attention.w{c}") for c in "qkv")
        q, k, v = q.reshape(3, 8, 4, 128), k.reshape(3, 8, 128), v.reshape(3, 8, 128)
        s = np.exp(np.einsum("igrd,jgd->grij", q, k) * 128 ** -0.5)
        o = np.einsum("grij,jgd->igrd", s / s.sum(-1, keepdims=True), v).reshape(3, 4096)
        y = y + mul(o, f"{n}.attention.wo")
        h = rms(y, f"{n}.ffn_norm")
        g = mul(h, f"{n}.feed_forward.w1")
        y = y + mul(g / (1.0 + np.exp(-g)) * mul(h, f"{n}.feed_forward.w3"), f"{n}.feed_forward.w2")
    return mul(rms(y[:1], f"{p}.norm"), f"{p}.acoustic_codebook_output")[0]


@pytest.mark.parametrize("seed,time", [(3, 0.0), (4, 0.5), (5, 6.0 / 7.0)])
def test_velocity_against_64_bits(pkg, engine, synth_model, seed, time):
    """The longest sums in TMEM are 768 columns, 48 steps, each cut at most 2^-23 of a sum that is half its final size on the
    average; fourteen GEMMs follow one another. Products of random signs leave about an eighth of that (with all of K in
    one sum it was 7e-6 to 1e-5)."""
    x, hidden = pkg.synth_f32(36, seed, "v64.x"), pkg.synth_f32(3072, seed, "v64.h")
    want = _velocity64(synth_model.t, x, hidden, time)
    off = np.linalg.norm(engine.predict_velocity(x, hidden, time) - want) / np.linalg.norm(want)
    assert off < 14 * 24 * 2.0 ** -23 / 8, off


@pytest.mark.parametrize("cap", [30.0, 1000.0, 1e5])
def test_prompt_softcap(pkg, tmp_path, cap):
    """Scores far below the cap keep their digits. The limit is the two-term products'."""
    c = Case(pkg, tmp_path, config([attention(dim=64, vdim=64, window=0, softcap=cap, ff=0)]), seed=8)
    toks = tokens(c.cfg, 300, 8)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("bfloat16") as lm:
        assert error(feed(lm, lm.open(), toks, [299, 1]), want) < LIMIT["bfloat16"]


def test_prompt_attention_maxima_that_rise_late(pkg, tmp_path):
    """Rows whose largest score rises by more than 2^8 in a later tile of the same half, where the sums so far are scaled down.
    |q||k| of 98 in two terms is off by 98 * 2^-17 in a score: the limit is two of these."""
    c = Case(pkg, tmp_path, config([attention(heads=4, kv_heads=2, dim=64, vdim=64, window=0, rot=0, scale=0.6, softcap=0, ff=0)]), seed=9)
    toks = tokens(c.cfg, 420, 9)
    w, eps = c.w, c.cfg["norm"]["eps"]
    h = plain.layer_norm(w["embed"][np.array(toks)], w["l0.norm1"], eps)
    q = plain.rms_norm(h @ w["l0.mix.q"].T, w["l0.mix.q.norm"], eps)[:, :64]
    k = plain.rms_norm(h @ w["l0.mix.k"].T, w["l0.mix.k.norm"], eps)[:, :64]
    top = (q[384:] @ k[:384].T * 0.6 / np.log(2.0)).reshape(-1, 3, 2, 64).max(3)      # [row, tile of a half, half]
    assert (top[:, 1:] > top[:, :1] + 8.0).any(2).any(1).sum() > 10
    want = plain.forward(w, c.cfg, toks)[0]
    with c.open("bfloat16") as lm:
        assert error(lm.step(lm.open(), toks, range(420)), want) < 2 * 98 * 2.0 ** -17


@pytest.mark.parametrize("scale,cap", [(-0.2, 0), (-0.2, 15.0), (0.0, 0), (0.0, 15.0)])
def test_prompt_attention_scales(pkg, tmp_path, scale, cap):
    """A negative scale turns the order of the keys around, with a scale of zero all weigh the same."""
    c = Case(pkg, tmp_path, config([attention(dim=64, vdim=64, window=90, scale=scale, softcap=cap, ff=0)]), seed=10)
    toks = tokens(c.cfg, 200, 10)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("bfloat16") as lm:
        assert error(feed(lm, lm.open(), toks, [199, 1]), want) < LIMIT["bfloat16"]


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_rows_that_are_not_finite_stay_behind_their_tile(pkg, tmp_path, bad):
    """A token whose row is not finite spoils the rows that see it, and those before it in its tile of 64 keys at most
    (weights of zero times a value that is not finite)."""
    c = Case(pkg, tmp_path, config([attention(heads=4, kv_heads=4, dim=64, vdim=64, window=0, ff=72), attention(heads=4, kv_heads=2, dim=24, vdim=40)]),
             seed=11)
    toks = np.array(tokens(c.cfg, 400, 11))
    toks[toks == 5] = 6
    with c.open("bfloat16") as lm:
        clean = lm.step(lm.open(), toks.tolist(), range(400))
    c.w["embed"][5] = bad
    c.rewrite()
    toks[300] = 5
    with c.open("bfloat16") as lm:
        got = lm.step(lm.open(), toks.tolist(), range(400))
    assert np.array_equal(got[:256], clean[:256]) and not np.isfinite(got[300]).any()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,rows", [(2048, 40), (2048, 300), (3072, 297), (4096, 300), (1100, 300), (1028, 297), (1024, 300)])
def test_centred_norms_by_width(pkg, tmp_path, dtype, width, rows):
    """Widths that give every thread of the residual kernel equal columns (one barrier a norm) and others, each up to 296
    rows and in the smaller CTAs beyond; rows whose mean is eight times their spread. The limits are those of the types."""
    c = Case(pkg, tmp_path, config([attention(ff=40)], width=width, vocab=101), seed=width + rows)
    c.w["embed"] += 8.0
    c.rewrite()
    toks = tokens(c.cfg, rows, 12)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open(dtype) as lm:
        assert error(lm.step(lm.open(), toks, range(rows)), want) < LIMIT[dtype]
