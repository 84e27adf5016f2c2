/*
 * vb_codec.cu - the audio codec decoder on the GPU: 37 codes per frame -> 24 kHz waveform
 * (tts_codec_decode, voxtral_tts_codec.c:389-510).
 *
 *   codes -> embedding [T, 292] (voxtral_tts_codec.c:276-300)
 *         -> causal conv 292 -> 1024, kernel 3 (voxtral_tts_kernels.c:217-270)
 *         -> 4 stages x 2 transformer layers (voxtral_tts_codec.c:306-383: RMSNorm eps 1e-2, QK norm
 *            over the whole row, ALiBi sliding-window causal attention, voxtral_tts_kernels.c:527-596,
 *            layer scale, SwiGLU) with a stride-2 transposed conv (kernel 4,
 *            voxtral_tts_kernels.c:272-327) after stages 0..2: T -> 2T -> 4T -> 8T rows
 *         -> causal conv 1024 -> 240, kernel 7 -> [8T, 240] = the waveform
 *
 * Rows stay row-major [time, channel] throughout (the reference transposes to channel-first
 * around every convolution). The transformer linears run on the tensor-core GEMMs
 * (vb_tc.cu, vb_tc_rows.cu) with BF16 weights - exact, because the checkpoint's BF16 values were only widened to
 * fp32 by the loader - and the activations as hi + lo BF16 terms. A convolution is a GEMM too,
 *   C[t][oc] = bias[oc] + sum over taps and input channels of X[src(t, tap)][ic] * W[oc][tap][ic],
 * and a stride-2 transposed convolution is one with both output parities as columns,
 *   C[m][parity * 1024 + oc] = sum over 2 taps of X[m - tap][ic] * W[ic][oc][parity + 2 tap],
 * whose row-major result [T][2048] IS the upsampled sequence [2T][1024]. Their (weight-normed)
 * weights are genuine fp32: they are split into W = hi + lo BF16 matrices (16 mantissa bits,
 * relative error 4e-6), stacked as one matrix of 2 N rows, and the kernel that reads the partial
 * results adds the two halves and the bias.
 *
 * A stage's GEMMs take the tile of its own row count and split K until the SMs are busy (5 frames: the
 * down projection had 8 CTAs); the partial results are summed by the kernel that reads them, so that no
 * launch only adds. 97 launches were, 75 are: 5 frames 0.62 -> 0.37 ms, 611 frames 2.55 -> 2.38 ms.
 */
#include "vb_common.cuh"
#include "vb_model.cuh"
#include "vb_tc.cuh"

#include <algorithm>
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <vector>

namespace vb {

namespace {

constexpr int CD = 1024, CH = 4096, CQKV = 3 * CD, CHEADS = 8, CHD = 128;
constexpr int CEMB = 292, CSEM = 256, CSEM_ROWS = 8192, CPATCH = 240, CLAYERS = 8, CSTAGES = 4;
constexpr float CEPS = 1e-2f, CQK_EPS = 1e-6f;
constexpr int kSegment = 16;     /* TMEM sums of at most 1024 columns. 611 frames: 1.7e-5 off 64 bits, 2.44 ms; 2.2e-5 and 2.40 with 2048 */
constexpr int CFSQ = 21, CSPECIAL = 2, CCODES = 37;

struct CodecLayer {
    TcWeight wqkv, wo, w13, w2;
    float *attn_norm = nullptr, *ffn_norm = nullptr, *q_norm = nullptr, *k_norm = nullptr;
    float *attn_scale = nullptr, *ffn_scale = nullptr;
    int window = 0;
};

struct Codec {
    bool ready = false;
    std::vector<void *> allocs;          /* weights */
    float *sem = nullptr;
    /* convolutions as GEMMs: hi BF16 halves of W[N][Kpad], the lo halves below them, bias[N] */
    struct Conv {
        TcWeight w;
        float *bias = nullptr;
        int N = 0, K = 0, Kpad = 0, Cin = 0, taps = 0, mode = 0, left_pad = 0;
    } in_conv, up_conv[3], out_conv;
    CodecLayer L[CLAYERS];
    float *d_slopes = nullptr;
    /* activations, sized for cap_rows = 8 * frames */
    std::vector<void *> act_allocs;
    int cap_frames = 0;
    int *codes = nullptr;
    float *x = nullptr, *qkv = nullptr, *ssq = nullptr;
    float *pcm = nullptr;
    uint16_t *tD = nullptr, *tH = nullptr, *tC = nullptr;
    float *part = nullptr;               /* split-K partials of one GEMM */
    size_t part_cap = 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    float last_ms = 0.0f;
};
Codec g_codec;
int g_block_frames = 0;   /* frames per decode block; 0: the largest the GEMM takes (an option, survives uploads) */

int c_alloc(void **p, size_t bytes, std::vector<void *> *owner) {
    if (cudaMalloc(p, bytes) != cudaSuccess) {
        cudaGetLastError();
        fprintf(stderr, "voxtral_b200: codec: cudaMalloc(%zu bytes) failed\n", bytes);
        *p = nullptr;
        return -1;
    }
    owner->push_back(*p);
    return 0;
}
void c_free(std::vector<void *> *owner) {
    for (void *p : *owner) cudaFree(p);
    owner->clear();
}

/* ---------------------------------------------------------------- upload kernels */

/* dst[r0 + r][c] = BF16(src[r][c]); *inexact counts the values BF16 cannot hold. */
__global__ void to_bf16_kernel(uint16_t *dst, const float *src, size_t n, unsigned *inexact) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t u = __float_as_uint(src[i]);
    if (u & 0xffffu) atomicAdd(inexact, 1u);
    dst[i] = (uint16_t)(u >> 16);
}
/* rows 2i / 2i+1 <- gate row i / up row i (the SwiGLU pair layout of the GEMM epilogue) */
__global__ void to_bf16_interleaved_kernel(uint16_t *dst, const float *gate, const float *up, int rows, int cols,
                                           unsigned *inexact) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols) return;
    const size_t r = i / cols, c = i % cols;
    const uint32_t a = __float_as_uint(gate[i]), b = __float_as_uint(up[i]);
    if ((a | b) & 0xffffu) atomicAdd(inexact, 1u);
    dst[(2 * r) * cols + c] = (uint16_t)(a >> 16);
    dst[(2 * r + 1) * cols + c] = (uint16_t)(b >> 16);
}
/* conv weight [oc][ic][k] -> [oc][k][ic] */
__global__ void conv_w_kernel(float *dst, const float *src, int oc, int ic, int k) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)oc * ic * k) return;
    const int kk = (int)(i % k), c = (int)((i / k) % ic), o = (int)(i / ((size_t)k * ic));
    dst[((size_t)o * k + kk) * ic + c] = src[i];
}
/* transposed-conv weight [ic][oc][k], k = parity + 2 * tap -> [parity][oc][tap][ic] */
__global__ void convt_w_kernel(float *dst, const float *src, int ic, int oc, int k) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)oc * ic * k) return;
    const int kk = (int)(i % k), o = (int)((i / k) % oc), c = (int)(i / ((size_t)k * oc));
    const int parity = kk & 1, tap = kk >> 1, taps = k / 2;
    dst[(((size_t)parity * oc + o) * taps + tap) * ic + c] = src[i];
}

/* ---------------------------------------------------------------- decode kernels */

/* Four values as BF16 terms; `term` elements between the terms, three of them or two. */
VB_DEVINL void put_terms(uint16_t *o, size_t term, int n_terms, const float (&e)[4]) {
    uint16_t t[3][4];
#pragma unroll
    for (int i = 0; i < 4; i++) vb_split3(e[i], t[0][i], t[1][i], t[2][i]);
#pragma unroll
    for (int j = 0; j < 3; j++)
        if (j < n_terms)
            *reinterpret_cast<uint2 *>(o + j * term) = make_uint2(t[j][0] | ((uint32_t)t[j][1] << 16), t[j][2] | ((uint32_t)t[j][3] << 16));
}

/* Where a kernel's values come from: the sum of n split-K partials [rows][ld], `stride` floats apart. A convolution's
 * has its lo half's columns `lo` further on (0: none), and its rows of N columns are rows of 1024 to the reader. */
struct Parts {
    const float *p;
    int n, ld, N, lo;
    size_t stride;
    const float *bias;
};
VB_DEVINL float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
VB_DEVINL float4 parts_sum4(const Parts &g, int m, int c) {
    const int e = m * CD + c, row = g.N == CD ? m : e / g.N, col = g.N == CD ? c : e - row * g.N;
    const float *q = g.p + (size_t)row * g.ld + col;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 t[kTcMaxSplits], u[kTcMaxSplits];
#pragma unroll
    for (int i = 0; i < kTcMaxSplits; i++) {
        t[i] = i < g.n ? vb_ldcg4(q + (size_t)i * g.stride) : zero;
        u[i] = i < g.n && g.lo ? vb_ldcg4(q + (size_t)i * g.stride + g.lo) : zero;
    }
    float4 v = g.bias ? *reinterpret_cast<const float4 *>(g.bias + col) : zero;
#pragma unroll
    for (int i = 0; i < kTcMaxSplits; i++)
        if (i < g.n) v = add4(v, g.lo ? add4(t[i], u[i]) : t[i]);
    return v;
}

/* The operand of the input convolution's GEMM, straight from the codes: terms[m][tap * 292 + ic] of row
 * src(m, tap) of the embedding (voxtral_tts_codec.c:276-300: 256 columns of the semantic table, then the FSQ levels as
 * [-1, 1]), with the convolution's reflect rule (voxtral_tts_kernels.c:246-262: src = m + tap - left_pad; src < 0 ->
 * -src; outside [0, T) -> 0; at the right end nothing reaches beyond). Columns from taps * 292 on are zero.
 * grid = (Kpad / 1024 rounded up, T), 256 threads x 4 columns (292 is a multiple of 4: one tap each). */
__global__ void codec_input_kernel(uint16_t *buf, int rows_pad, int n_terms, int Kpad, const int *codes, const float *sem, int T, int taps,
                                   int left_pad) {
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.y, k = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (k >= Kpad) return;
    float e[4] = {0.f, 0.f, 0.f, 0.f};
    const int tap = k / CEMB, ic = k - tap * CEMB;
    int src = m + tap - left_pad;
    if (src < 0) src = -src;
    if (tap < taps && src < T) {
        const int *fc = codes + src * CCODES;
        if (ic < CSEM) {
            int s = fc[0] - CSPECIAL;
            s = s < 0 ? 0 : (s >= CSEM_ROWS ? CSEM_ROWS - 1 : s);
            const float4 v = __ldg(reinterpret_cast<const float4 *>(sem + (size_t)s * CSEM + ic));
            e[0] = v.x; e[1] = v.y; e[2] = v.z; e[3] = v.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int a = fc[ic + i - CSEM + 1] - CSPECIAL;
                a = a < 0 ? 0 : (a >= CFSQ ? CFSQ - 1 : a);
                e[i] = (float)a * 2.0f / (float)(CFSQ - 1) - 1.0f;
            }
        }
    }
    put_terms(buf + (size_t)m * Kpad + k, (size_t)rows_pad * Kpad, n_terms, e);
}

/* A stage's last feed-forward update, and the operand of the convolution after it: row s, v = x + parts * scale, goes to
 * every place terms[m][tap * 1024 ..] of the rows m that read it.
 * UP, the stride-2 transposed convolution of kernel 4 (voxtral_tts_kernels.c:272-327: no left trim, the last two raw
 * outputs dropped): rows s and s + 1, taps 0 and 1; row 0 has nothing in tap 1.
 * Otherwise the causal convolution with the reflect rule: row s + left_pad - tap, and, mirrored, left_pad - tap - s for
 * s > 0 (the last stage's rows are more than its taps). grid = T, 256 threads x 4 columns. */
template <bool UP>
__global__ void codec_scatter_kernel(uint16_t *buf, int rows_pad, int n_terms, const float *x, const Parts g, const float *scale, int T,
                                     int taps) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.x, c = threadIdx.x * 4, K = taps * CD, left = taps - 1;
    const float4 y = parts_sum4(g, s, c);
    float4 v = *reinterpret_cast<const float4 *>(x + (size_t)s * CD + c);
    if (scale) {
        const float4 f = __ldg(reinterpret_cast<const float4 *>(scale + c));
        v.x += y.x * f.x; v.y += y.y * f.y; v.z += y.z * f.z; v.w += y.w * f.w;
    } else {
        v = add4(v, y);
    }
    const float e[4] = {v.x, v.y, v.z, v.w};
    const size_t term = (size_t)rows_pad * K;
    if constexpr (UP) {
        put_terms(buf + (size_t)s * K + c, term, n_terms, e);
        if (s + 1 < T) put_terms(buf + (size_t)(s + 1) * K + CD + c, term, n_terms, e);
        if (s == 0) {
            const float none[4] = {0.f, 0.f, 0.f, 0.f};
            put_terms(buf + CD + c, term, n_terms, none);
        }
    } else {
        for (int tap = 0; tap < taps; tap++) {
            const int m = s + left - tap, mirror = left - tap - s;
            if (m < T) put_terms(buf + (size_t)m * K + tap * CD + c, term, n_terms, e);
            if (s > 0 && mirror >= 0) put_terms(buf + (size_t)mirror * K + tap * CD + c, term, n_terms, e);
        }
    }
}

/* The output convolution's samples: partials of both halves and the bias. */
__global__ void codec_samples_kernel(float *pcm, const Parts g, int T) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T * g.N / 4) return;
    const int m = i * 4 / g.N, c = i * 4 - m * g.N;
    const float *q = g.p + (size_t)m * g.ld + c;
    float4 v = g.bias ? *reinterpret_cast<const float4 *>(g.bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p = 0; p < g.n; p++) v = add4(v, add4(vb_ldcg4(q + (size_t)p * g.stride), vb_ldcg4(q + (size_t)p * g.stride + g.lo)));
    *reinterpret_cast<float4 *>(pcm + (size_t)m * g.N + c) = v;
}

/* W[N][K] fp32 -> hi[N][Kpad], lo[N][Kpad] BF16 with W = hi + lo up to 2^-17 (hi truncated, lo the
 * rounded remainder), zero beyond K. */
__global__ void split_w_kernel(uint16_t *hi, uint16_t *lo, const float *W, int N, int K, int Kpad) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)N * Kpad) return;
    const int n = (int)(i / Kpad), k = (int)(i % Kpad);
    uint16_t h = 0, l = 0;
    if (k < K) {
        const float w = W[(size_t)n * K + k];
        const uint32_t u = __float_as_uint(w) & 0xffff0000u;
        h = (uint16_t)(u >> 16);
        const float r = w - __uint_as_float(u);
        uint32_t ru = __float_as_uint(r);
        ru += 0x7fffu + ((ru >> 16) & 1u);                     /* round to nearest even */
        l = (uint16_t)(ru >> 16);
    }
    hi[i] = h;
    lo[i] = l;
}

/* Rows -> BF16 terms for the next GEMM, with the residual update folded in:
 *   v = parts (x null), x + parts * scale, or x + parts;  x_out[m] = v;  terms = v * gain,  ssq[m] = sum v^2 (the GEMM
 *   applies 1/sqrt(ssq/K + eps)).  grid = rows, 256 threads x 4 columns. */
__global__ void codec_prepare_kernel(uint16_t *buf, int rows_pad, int n_terms, const float *x, const Parts g, const float *scale,
                                     float *x_out, const float *gain, float *ssq) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[8];
    const int m = blockIdx.x, c = threadIdx.x * 4;
    float4 v = parts_sum4(g, m, c);
    if (x) {
        const float4 r = *reinterpret_cast<const float4 *>(x + (size_t)m * CD + c);
        if (scale) {
            const float4 f = __ldg(reinterpret_cast<const float4 *>(scale + c));
            v = make_float4(r.x + v.x * f.x, r.y + v.y * f.y, r.z + v.z * f.z, r.w + v.w * f.w);
        } else {
            v = add4(r, v);
        }
    }
    *reinterpret_cast<float4 *>(x_out + (size_t)m * CD + c) = v;
    float ss = vb_warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
    const float4 w = __ldg(reinterpret_cast<const float4 *>(gain + c));
    const float e[4] = {v.x * w.x, v.y * w.y, v.z * w.z, v.w * w.w};
    put_terms(buf + (size_t)m * CD + c, (size_t)rows_pad * CD, n_terms, e);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int i = 0; i < 8; i++) t += red[i];
        ssq[m] = t;
    }
}

/* Sums q, k, v out of the partials; QK norm: RMSNorm over the whole 1024-wide q row and k row (tts_qk_norm,
 * voxtral_tts_kernels.c:351-355). A single partial is normed in place (qkv = part), its values left alone.
 * grid = (rows, 3, or 2 in place), 256 threads. */
__global__ void codec_qkv_kernel(float *qkv, const float *part, int n, size_t stride, const float *qw, const float *kw, float eps) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[8];
    const float *w = blockIdx.y == 0 ? qw : blockIdx.y == 1 ? kw : nullptr;
    const size_t at = (size_t)blockIdx.x * CQKV + blockIdx.y * CD + threadIdx.x * 4;
    float4 t[kTcMaxSplits];
#pragma unroll
    for (int i = 0; i < kTcMaxSplits; i++) t[i] = i < n ? vb_ldcg4(part + i * stride + at) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v = t[0];
#pragma unroll
    for (int i = 1; i < kTcMaxSplits; i++)
        if (i < n) v = add4(v, t[i]);
    if (w) {
        const float ss = vb_warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
        __syncthreads();
        float sum = 0.0f;
        for (int i = 0; i < 8; i++) sum += red[i];
        const float inv = 1.0f / sqrtf(sum / (float)CD + eps);
        const float4 g = __ldg(reinterpret_cast<const float4 *>(w + threadIdx.x * 4));
        v.x = v.x * inv * g.x; v.y = v.y * inv * g.y; v.z = v.z * inv * g.z; v.w = v.w * inv * g.w;
    }
    *reinterpret_cast<float4 *>(qkv + at) = v;
}

/* ALiBi sliding-window causal attention (tts_alibi_attention, voxtral_tts_kernels.c:527-596), its result as the terms
 * that the O projection reads: one warp per (row, head), a lane owns 4 of the 128 dims, keys max(0, i - window + 1) .. i
 * in order, four of them requested together. The eight warps of a CTA take eight rows of one head, which share most of
 * their keys in L1. grid = (rows / 8 rounded up, heads). */
__global__ void __launch_bounds__(256) codec_attention_kernel(uint16_t *buf, int rows_pad, int n_terms, const float *qkv, int rows, int window,
                                                              float scale, const float *slopes8) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), h = blockIdx.y, lane = threadIdx.x & 31;
    if (i >= rows) return;
    const float slope = slopes8[h];
    const float *col = qkv + h * CHD + lane * 4;
    const float4 q = *reinterpret_cast<const float4 *>(col + (size_t)i * CQKV);
    int j0 = 0;
    if (window > 0 && i - window + 1 > 0) j0 = i - window + 1;
    float mx = -1e30f, den = 0.0f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int jb = j0; jb <= i; jb += 4) {
        float4 k[4], v[4];
        float s[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float *r = col + (size_t)(jb + u < i ? jb + u : i) * CQKV;
            k[u] = *reinterpret_cast<const float4 *>(r + CD);
            v[u] = *reinterpret_cast<const float4 *>(r + 2 * CD);
            s[u] = q.x * k[u].x + q.y * k[u].y + q.z * k[u].z + q.w * k[u].w;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int u = 0; u < 4; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
        float top = mx;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            s[u] = jb + u <= i ? s[u] * scale + slope * (float)(jb + u - i) : -INFINITY;
            top = fmaxf(top, s[u]);
        }
        const float corr = expf(mx - top);
        mx = top;
        den *= corr;
        o.x *= corr; o.y *= corr; o.z *= corr; o.w *= corr;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float w = expf(s[u] - top);
            den += w;
            o.x += w * v[u].x; o.y += w * v[u].y; o.z += w * v[u].z; o.w += w * v[u].w;
        }
    }
    const float inv = den > 0.0f ? 1.0f / den : 0.0f;
    const float e[4] = {o.x * inv, o.y * inv, o.z * inv, o.w * inv};
    put_terms(buf + (size_t)i * CD + h * CHD + lane * 4, (size_t)rows_pad * CD, n_terms, e);
}

/* ---------------------------------------------------------------- host side */

int up_f32(float **dst, const float *src, size_t n, std::vector<void *> *owner) {
    if (!src) { *dst = nullptr; return 0; }
    if (c_alloc((void **)dst, n * 4, owner)) return -1;
    return cudaMemcpy(*dst, src, n * 4, cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -1;
}

/* fp32 host matrices -> one BF16 device matrix (rows stacked), tile-contiguous for the GEMM. */
int up_matrix(TcWeight *tw, const float *const *parts, const int *part_rows, int n_parts, int cols, bool interleave,
              float *stage, unsigned *inexact, std::vector<void *> *owner, cudaStream_t st) {
    int rows = 0;
    for (int i = 0; i < n_parts; i++) rows += part_rows[i];
    uint16_t *plain = nullptr, *tiled = nullptr;
    if (cudaMalloc((void **)&plain, (size_t)rows * cols * 2) != cudaSuccess) return -1;
    int rc = 0;
    if (interleave) {
        /* two parts of equal height: gate rows and up rows */
        const size_t n = (size_t)part_rows[0] * cols;
        if (cudaMemcpyAsync(stage, parts[0], n * 4, cudaMemcpyHostToDevice, st) != cudaSuccess ||
            cudaMemcpyAsync(stage + n, parts[1], n * 4, cudaMemcpyHostToDevice, st) != cudaSuccess)
            rc = -1;
        if (!rc)
            to_bf16_interleaved_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(plain, stage, stage + n, part_rows[0],
                                                                                  cols, inexact);
    } else {
        size_t off = 0;
        for (int i = 0; i < n_parts && !rc; i++) {
            const size_t n = (size_t)part_rows[i] * cols;
            if (cudaMemcpyAsync(stage, parts[i], n * 4, cudaMemcpyHostToDevice, st) != cudaSuccess) { rc = -1; break; }
            to_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(plain + off, stage, n, inexact);
            off += n;
        }
    }
    if (!rc && c_alloc((void **)&tiled, tc_tiled_bytes(rows, cols), owner)) rc = -1;
    if (!rc && tc_weight_tiled(tw, plain, rows, cols, tiled, st)) rc = -1;
    if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
    cudaFree(plain);
    return rc;
}

/* The tile that a stage of so many rows takes, and the terms its GEMMs read of the activations. */
int pad_of(int rows) { return rows <= 64 ? tc_rows_pad_frame(rows) : tc_rows_pad_any(rows); }
int terms_of(int rows_pad) { return rows_pad < 256 ? kTcTerms : 2; }
int splits_for(int N, int K, int rows) {
    return pad_of(rows) < 256 ? tc_pick_splits(N, K, model().sm_count) : tc_row_splits(N, K, rows, model().sm_count);
}

/* Floats of split-K partials that a block of so many frames needs. */
size_t part_floats(int frames) {
    const Codec &c = g_codec;
    size_t n = 0;
    auto take = [&](int N, int K, int rows) { n = std::max(n, (size_t)splits_for(N, K, rows) * rows * N); };
    take(2 * c.in_conv.N, c.in_conv.Kpad, frames);
    for (int s = 0, rows = frames; s < CSTAGES; s++, rows *= 2) {
        take(CQKV, CD, rows);
        take(CD, CD, rows);
        take(CD, CH, rows);
        const Codec::Conv &cv = s < CSTAGES - 1 ? c.up_conv[s] : c.out_conv;
        take(2 * cv.N, cv.Kpad, rows);
    }
    return n;
}

int ensure_buffers(int frames) {
    Codec &c = g_codec;
    const size_t part = part_floats(frames);
    if (part > c.part_cap) {
        cudaFree(c.part);
        c.part = nullptr;
        c.part_cap = 0;
        if (cudaMalloc((void **)&c.part, sizeof(float) * part) != cudaSuccess) {
            cudaGetLastError();
            c.part = nullptr;
            fprintf(stderr, "voxtral_b200: codec: cudaMalloc(%zu bytes) failed\n", sizeof(float) * part);
            return -1;
        }
        c.part_cap = part;
    }
    if (frames <= c.cap_frames) return 0;
    c_free(&c.act_allocs);
    c.cap_frames = 0;
    const int rows = 8 * frames;
    /* operands: laid out anew for every stage and convolution (rows that a stage has not written hold an earlier one's:
     * finite, and their results are never stored) */
    size_t tD = 0, tH = 0, tC = tc_acts_bytes(pad_of(frames), c.in_conv.Kpad);
    for (int s = 0; s < CSTAGES; s++) {
        const int pad = pad_of(frames << s);
        if (!pad) return -1;
        tD = std::max(tD, tc_acts_bytes(pad, CD));
        tH = std::max(tH, tc_acts_bytes(pad, CH));
        tC = std::max(tC, tc_acts_bytes(pad, s < CSTAGES - 1 ? c.up_conv[s].Kpad : c.out_conv.Kpad));
    }
    int rc = 0;
    rc |= c_alloc((void **)&c.codes, sizeof(int) * (size_t)frames * CCODES, &c.act_allocs);
    rc |= c_alloc((void **)&c.x, sizeof(float) * (size_t)rows * CD, &c.act_allocs);
    rc |= c_alloc((void **)&c.qkv, sizeof(float) * (size_t)rows * CQKV, &c.act_allocs);
    rc |= c_alloc((void **)&c.ssq, sizeof(float) * (size_t)rows, &c.act_allocs);
    rc |= c_alloc((void **)&c.pcm, sizeof(float) * (size_t)rows * CPATCH, &c.act_allocs);
    rc |= c_alloc((void **)&c.tD, tD, &c.act_allocs);
    rc |= c_alloc((void **)&c.tH, tH, &c.act_allocs);
    rc |= c_alloc((void **)&c.tC, tC, &c.act_allocs);
    if (rc) { c_free(&c.act_allocs); return -1; }
    /* rows of the padding are multiplied like any other (their results are never stored): keep them finite */
    cudaMemsetAsync(c.tD, 0, tD, model().st);
    cudaMemsetAsync(c.tH, 0, tH, model().st);
    cudaMemsetAsync(c.tC, 0, tC, model().st);
    c.cap_frames = frames;
    return 0;
}

/* One GEMM into split-K partials. */
int gemm_parts(const TcWeight &w, const TcActs &a, int rows, const float *ssq, Parts *out, cudaStream_t st) {
    TcGemm g;
    g.M = rows; g.segment = kSegment; g.splits = splits_for(w.N, w.K, rows); g.epi = TC_EPI_PARTIAL; g.out = g_codec.part; g.ld_out = w.N;
    g.ssq = ssq; g.ssq_chunks = ssq ? 1 : 0; g.eps = CEPS;
    g.status = &model().d_out->status;
    *out = {g.out, g.splits, w.N, w.N, 0, (size_t)rows * w.N, nullptr};
    return tc_gemm(w, a, g, st);
}

/* x and aD hold the rows of the layer's attention norm; leaves x and the partials of the feed-forward, which the caller
 * adds (times ffn_scale) to x. */
int layer_forward(const CodecLayer &L, const TcActs &aD, const TcActs &aH, int rows, Parts *out, cudaStream_t st) {
    Codec &c = g_codec;
    const int rp = aD.rows_pad, terms = terms_of(rp);
    const float scale = 1.0f / sqrtf((float)CHD);
    Parts p;
    if (gemm_parts(L.wqkv, aD, rows, c.ssq, &p, st)) return -1;
    float *qkv = p.n == 1 ? c.part : c.qkv;
    if (p.n > 1 || L.q_norm || L.k_norm)
        launch_pdl(codec_qkv_kernel, dim3(rows, p.n == 1 ? 2 : 3), dim3(256), 0, st, qkv, p.p, p.n, p.stride, (const float *)L.q_norm,
                   (const float *)L.k_norm, CQK_EPS);
    launch_pdl(codec_attention_kernel, dim3((rows + 7) / 8, CHEADS), dim3(256), 0, st, c.tD, rp, terms, (const float *)qkv, rows, L.window, scale,
               (const float *)c.d_slopes);
    if (gemm_parts(L.wo, aD, rows, nullptr, &p, st)) return -1;
    launch_pdl(codec_prepare_kernel, dim3(rows), dim3(256), 0, st, c.tD, rp, terms, (const float *)c.x, p, (const float *)L.attn_scale, c.x,
               (const float *)L.ffn_norm, c.ssq);
    TcGemm g;
    g.M = rows; g.segment = kSegment; g.splits = 1; g.epi = TC_EPI_SWIGLU_TERMS; g.ld_out = CH; g.ssq = c.ssq; g.ssq_chunks = 1; g.eps = CEPS;
    g.out_terms = c.tH; g.out_rows_pad = rp; g.status = &model().d_out->status;
    if (tc_gemm(L.w13, aD, g, st)) return -1;
    return gemm_parts(L.w2, aH, rows, nullptr, out, st);
}

/* One convolution made ready as a GEMM: weights reordered to [N][taps * Cin] (a transposed
 * convolution: both parities stacked, N = 2 * out_ch, 2 taps each), split into hi / lo BF16
 * matrices one below the other, tiled; bias (repeated per parity). */
int conv_setup(Codec::Conv *cv, const vb200_conv_t &w, float *stage, std::vector<void *> *owner, cudaStream_t st) {
    const bool tr = w.is_transpose != 0;
    const size_t n = (size_t)w.in_ch * w.out_ch * w.kernel;
    cv->Cin = w.in_ch;
    cv->taps = tr ? w.kernel / 2 : w.kernel;
    cv->N = tr ? 2 * w.out_ch : w.out_ch;
    cv->K = cv->taps * w.in_ch;
    cv->Kpad = (cv->K + 63) / 64 * 64;
    cv->mode = tr ? 1 : 0;
    cv->left_pad = tr ? 0 : w.kernel - w.stride;
    float *ordered = stage + n;                                  /* second half of the staging buffer */
    uint16_t *both = nullptr, *tiled = nullptr;
    const size_t nk = (size_t)cv->N * cv->Kpad;
    int rc = 0;
    if (!w.weight || cudaMemcpyAsync(stage, w.weight, n * 4, cudaMemcpyHostToDevice, st) != cudaSuccess) return -1;
    if (tr) convt_w_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ordered, stage, w.in_ch, w.out_ch, w.kernel);
    else conv_w_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ordered, stage, w.out_ch, w.in_ch, w.kernel);
    if (cudaMalloc((void **)&both, nk * 4) != cudaSuccess) rc = -1;
    if (!rc) split_w_kernel<<<(unsigned)((nk + 255) / 256), 256, 0, st>>>(both, both + nk, ordered, cv->N, cv->K, cv->Kpad);
    if (!rc && c_alloc((void **)&tiled, tc_tiled_bytes(2 * cv->N, cv->Kpad), owner)) rc = -1;
    if (!rc && tc_weight_tiled(&cv->w, both, 2 * cv->N, cv->Kpad, tiled, st)) rc = -1;
    if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
    cudaFree(both);
    if (!rc && w.bias) {
        if (c_alloc((void **)&cv->bias, sizeof(float) * cv->N, owner)) return -1;
        for (int p = 0; p < (tr ? 2 : 1) && !rc; p++)
            if (cudaMemcpy(cv->bias + (size_t)p * w.out_ch, w.bias, sizeof(float) * w.out_ch, cudaMemcpyHostToDevice) != cudaSuccess)
                rc = -1;
    }
    return rc;
}

/* One convolution's GEMM on its operand in tC; the reader adds the halves and the bias. */
int conv_run(const Codec::Conv &cv, const TcActs &acts, int T, Parts *out, cudaStream_t st) {
    if (gemm_parts(cv.w, acts, T, nullptr, out, st)) return -1;
    out->N = cv.N; out->lo = cv.N; out->bias = cv.bias;
    return 0;
}

} // namespace

void codec_free_all() {
    Codec &c = g_codec;
    c_free(&c.allocs);
    c_free(&c.act_allocs);
    cudaFree(c.part);
    if (c.e0) cudaEventDestroy(c.e0);
    if (c.e1) cudaEventDestroy(c.e1);
    c = Codec();
}

int codec_upload(const vb200_codec_weights_t *w) {
    Model &m = model();
    Codec &c = g_codec;
    if (!m.inited || !w) return -1;
    codec_free_all();
    if (tc_init()) return -1;
    /* the shapes this decoder is written for (voxtral_tts_codec.c:204-262) */
    const vb200_conv_t &ic = w->input_conv, &oc = w->output_proj;
    bool ok = w->semantic_embedding && ic.in_ch == CEMB && ic.out_ch == CD && ic.kernel == 3 && ic.stride == 1 &&
              !ic.is_transpose && oc.in_ch == CD && oc.out_ch == CPATCH && oc.kernel == 7 && oc.stride == 1 && !oc.is_transpose;
    for (int s = 0; s < CSTAGES - 1 && ok; s++) {
        const vb200_conv_t &u = w->stage_convs[s];
        ok = u.in_ch == CD && u.out_ch == CD && u.kernel == 4 && u.stride == 2 && u.is_transpose && u.weight;
    }
    for (int l = 0; l < CLAYERS && ok; l++) {
        const vb200_codec_layer_t &L = w->transformers[l];
        ok = L.wq && L.wk && L.wv && L.wo && L.w1 && L.w2 && L.w3 && L.attention_norm && L.ffn_norm;
    }
    if (!ok) {
        fprintf(stderr, "voxtral_b200: codec: weights missing or of an unexpected shape\n");
        return -1;
    }
    cudaStream_t st = m.st;
    float *stage = nullptr;
    unsigned *inexact = nullptr;
    if (cudaMalloc((void **)&stage, sizeof(float) * (size_t)2 * CH * CD) != cudaSuccess ||
        cudaMalloc((void **)&inexact, sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(stage);
        return -1;
    }
    cudaMemset(inexact, 0, sizeof(unsigned));
    int rc = 0;
    rc |= up_f32(&c.sem, w->semantic_embedding, (size_t)CSEM_ROWS * CSEM, &c.allocs);
    rc |= conv_setup(&c.in_conv, ic, stage, &c.allocs, st);
    rc |= conv_setup(&c.out_conv, oc, stage, &c.allocs, st);
    for (int s = 0; s < CSTAGES - 1 && !rc; s++) rc |= conv_setup(&c.up_conv[s], w->stage_convs[s], stage, &c.allocs, st);
    for (int l = 0; l < CLAYERS && !rc; l++) {
        const vb200_codec_layer_t &L = w->transformers[l];
        CodecLayer &d = c.L[l];
        const float *qkv[3] = {L.wq, L.wk, L.wv};
        const int r3[3] = {CD, CD, CD};
        const float *gu[2] = {L.w1, L.w3};
        const int r2[2] = {CH, CH};
        const float *one[1];
        const int rD[1] = {CD};
        rc |= up_matrix(&d.wqkv, qkv, r3, 3, CD, false, stage, inexact, &c.allocs, st);
        one[0] = L.wo;
        rc |= up_matrix(&d.wo, one, rD, 1, CD, false, stage, inexact, &c.allocs, st);
        rc |= up_matrix(&d.w13, gu, r2, 2, CD, true, stage, inexact, &c.allocs, st);
        one[0] = L.w2;
        rc |= up_matrix(&d.w2, one, rD, 1, CH, false, stage, inexact, &c.allocs, st);
        rc |= up_f32(&d.attn_norm, L.attention_norm, CD, &c.allocs);
        rc |= up_f32(&d.ffn_norm, L.ffn_norm, CD, &c.allocs);
        rc |= up_f32(&d.q_norm, L.q_norm, CD, &c.allocs);
        rc |= up_f32(&d.k_norm, L.k_norm, CD, &c.allocs);
        rc |= up_f32(&d.attn_scale, L.attn_scale, CD, &c.allocs);
        rc |= up_f32(&d.ffn_scale, L.ffn_scale, CD, &c.allocs);
        d.window = L.window_size;
    }
    float *slopes = nullptr;
    if (!rc) rc = up_f32(&slopes, w->alibi_slopes, CHEADS, &c.allocs);
    c.d_slopes = slopes;
    unsigned bad = 0;
    if (!rc && cudaMemcpy(&bad, inexact, sizeof(unsigned), cudaMemcpyDeviceToHost) != cudaSuccess) rc = -1;
    cudaFree(stage);
    cudaFree(inexact);
    if (!rc && bad) {
        fprintf(stderr, "voxtral_b200: codec: %u transformer weights are not exactly representable in BF16; "
                        "this decoder keeps them as BF16 and refuses to round\n", bad);
        rc = -1;
    }
    if (!rc && (cudaEventCreate(&c.e0) != cudaSuccess || cudaEventCreate(&c.e1) != cudaSuccess)) rc = -1;
    if (rc) {
        codec_free_all();
        return -1;
    }
    c.ready = true;
    return 0;
}

/* One block of at most kTcMaxRows / 8 frames: the samples of frames [skip, n_frames) go to
 * samples_out. */
static int decode_block(const int *codes, int n_frames, int skip, float *samples_out, float *ms) {
    Model &m = model();
    Codec &c = g_codec;
    if (8 * n_frames > kTcMaxRows || skip < 0 || skip >= n_frames) return -1;
    const size_t total = (size_t)(n_frames - skip) * 8 * CPATCH;
    if (ensure_buffers(n_frames)) return -1;
    cudaStream_t st = m.st;
    if (cudaMemcpyAsync(c.codes, codes, sizeof(int) * (size_t)n_frames * CCODES, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return -1;
    cudaEventRecord(c.e0, st);
    int rows = n_frames, rp = pad_of(rows);
    TcActs acts, aD, aH;
    Parts p;
    launch_pdl(codec_input_kernel, dim3((c.in_conv.Kpad + 1023) / 1024, rows), dim3(256), 0, st, c.tC, rp, terms_of(rp), c.in_conv.Kpad,
               (const int *)c.codes, (const float *)c.sem, rows, c.in_conv.taps, c.in_conv.left_pad);
    if (tc_acts(&acts, c.tC, rp, c.in_conv.Kpad) || conv_run(c.in_conv, acts, rows, &p, st)) return -1;
    int l = 0;
    for (int stage = 0; stage < CSTAGES; stage++) {
        rp = pad_of(rows);
        if (tc_acts(&aD, c.tD, rp, CD) || tc_acts(&aH, c.tH, rp, CH)) return -1;
        for (int i = 0; i < 2; i++, l++) {
            /* the convolution's rows, or the layer before's feed-forward update */
            launch_pdl(codec_prepare_kernel, dim3(rows), dim3(256), 0, st, c.tD, rp, terms_of(rp), i ? (const float *)c.x : (const float *)nullptr, p,
                       i ? (const float *)c.L[l - 1].ffn_scale : (const float *)nullptr, c.x, (const float *)c.L[l].attn_norm, c.ssq);
            if (layer_forward(c.L[l], aD, aH, rows, &p, st)) return -1;
        }
        const bool up = stage < CSTAGES - 1;
        const Codec::Conv &cv = up ? c.up_conv[stage] : c.out_conv;
        launch_pdl(up ? codec_scatter_kernel<true> : codec_scatter_kernel<false>, dim3(rows), dim3(256), 0, st, c.tC, rp, terms_of(rp),
                   (const float *)c.x, p, (const float *)c.L[l - 1].ffn_scale, rows, cv.taps);
        if (tc_acts(&acts, c.tC, rp, cv.Kpad) || conv_run(cv, acts, rows, &p, st)) return -1;
        if (up) rows *= 2;      /* [rows][2 x 1024] row-major = [2 rows][1024] */
    }
    launch_pdl(codec_samples_kernel, dim3((rows * CPATCH / 4 + 255) / 256), dim3(256), 0, st, c.pcm, p, rows);
    cudaEventRecord(c.e1, st);
    int status = 0;
    if (cudaMemcpyAsync(samples_out, c.pcm + (size_t)skip * 8 * CPATCH, sizeof(float) * total, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(&status, &m.d_out->status, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    float t = 0.0f;
    cudaEventElapsedTime(&t, c.e0, c.e1);
    *ms += t;
    m.last_status = status;
    if (status) {
        cudaMemset(&m.d_out->status, 0, sizeof(int));
        return -1;
    }
    return 0;
}


/* The decoder only looks back: 2 frames in the input convolution, (window - 1) positions per
 * transformer layer at its stage's rate (2 + 3 + 3.5 + 3.75 frames), one position per transposed
 * convolution, 6/8 of a frame in the output convolution - under 17 frames in all. An utterance
 * longer than one block is therefore decoded block by block with 32 frames of left context whose
 * samples are dropped; what is kept equals the one-piece decode. */
constexpr int kCodecContext = 32;

int codec_set_block_frames(int frames) {
    if (frames < 2 * kCodecContext || frames > kTcMaxRows / 8) return -1;
    g_block_frames = frames;
    return 0;
}

int codec_decode(const int *codes, int n_frames, float *samples_out, int max_samples, int *n_samples) {
    Model &m = model();
    Codec &c = g_codec;
    if (n_samples) *n_samples = 0;
    if (!m.inited || !c.ready || !codes || n_frames < 1 || !samples_out) return -1;
    const long long total = (long long)n_frames * 8 * CPATCH;
    if (total > max_samples) return -1;
    const int block = g_block_frames > 0 ? g_block_frames : kTcMaxRows / 8;
    float ms = 0.0f;
    int pos = n_frames < block ? n_frames : block;
    if (decode_block(codes, pos, 0, samples_out, &ms)) return -1;
    while (pos < n_frames) {
        const int start = pos - kCodecContext;
        const int len = n_frames - start < block ? n_frames - start : block;
        if (decode_block(codes + (size_t)start * CCODES, len, kCodecContext, samples_out + (size_t)pos * 8 * CPATCH, &ms)) return -1;
        pos = start + len;
    }
    c.last_ms = ms;
    if (n_samples) *n_samples = (int)total;
    return 0;
}

float codec_last_ms() { return g_codec.last_ms; }

} // namespace vb
