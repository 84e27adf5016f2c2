/*
 * vb_lm_attn.cu - decoder language models: softmax attention over a ring cache. Query and key
 * norm over the whole projection, rotary positions on a part of the head, optional softcap,
 * optional sliding window with kept first tokens; any head sizes, separate key and value sizes.
 *
 *   lm_attn_prepare  one row per CTA: sums the projection's split-K partials, norms and rotates q
 *                    and k, appends k and v to the cache
 *   lm_attn_generic  fp32 pipes: any sizes, short portions and the 32-bit mode; a register tile of query rows and keys
 *                    a thread (keys split over CTAs, last arrival merges)
 *   lm_attn_step     one token, preparation included; lm_attn_step_group where a cluster per KV head can take it
 *   lm_attn_mma      prompts: tensor cores on hi + lo BF16 halves of q, k, v and the weights (vb_attn_tc.cuh); the
 *                    cache keeps k and v as such halves
 *
 * Keys are visited in two stretches, the kept first tokens and the window; a stretch that is out
 * of reach of all of a CTA's rows is never loaded.
 */
#include "vb_attn_tc.cuh"
#include "vb_tc.cuh"

#include <algorithm>

namespace vb {

namespace {

inline int ok(cudaError_t e) { return e == cudaSuccess ? 0 : -1; }

/* ------------------------------------------------------------------ q, k, v of a row */
constexpr int kPrepThreads = 512;

__global__ void __launch_bounds__(kPrepThreads) lm_attn_prepare_kernel(const LmAttn a) {
    extern __shared__ __align__(16) float prep_smem[];
    __shared__ float red[2][kPrepThreads / 32];
    const int nq = a.heads * a.dim, nk = a.kv_heads * a.dim, nv = a.kv_heads * a.vdim;
    float *buf = prep_smem;                       /* [nq + nk] */
    float *cs = buf + nq + nk;                    /* [rot / 2] cos, then [rot / 2] sin */
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x, tid = threadIdx.x, half = a.rot / 2;
    const int pos = a.dyn->pos + m;
    const size_t row = (size_t)lm_ring_row(a.ring, pos);
    for (int i = tid; i < half; i += kPrepThreads) {
        lm_angle(pos, a.freq[i], a.freq[half + i], a.mag, &cs[i], &cs[half + i]);
    }
    float sq = 0.0f, sk = 0.0f;
    float *Vr = lm_state(a.v, a.dyn) + row * nv;
    if (((nq | nk | a.vdim) & 3) == 0) {
        for (int c = tid * 4; c < nq + nk + nv; c += kPrepThreads * 4) {
            const float4 v = lm_sum4(a.qkv, m, c);
            if (c < nq + nk) {
                const float ss = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                *reinterpret_cast<float4 *>(buf + c) = v;
                if (c < nq) sq += ss; else sk += ss;
            } else {
                const int j = c - nq - nk, d = j % a.vdim;
                kv_put4(Vr + j - d, a.vdim, d, v, a.split);
            }
        }
    } else {
        for (int c = tid; c < nq + nk; c += kPrepThreads) {
            const float v = lm_sum_batch(a.qkv, m, c);
            buf[c] = v;
            if (c < nq) sq += v * v; else sk += v * v;
        }
        for (int c = tid; c < nv; c += kPrepThreads)
            kv_put(Vr + c / a.vdim * a.vdim, a.vdim, c % a.vdim, lm_sum_batch(a.qkv, m, nq + nk + c), a.split);
    }
    sq = vb_warp_sum(sq);
    sk = vb_warp_sum(sk);
    if ((tid & 31) == 0) { red[0][tid >> 5] = sq; red[1][tid >> 5] = sk; }
    __syncthreads();
    sq = sk = 0.0f;
#pragma unroll
    for (int w = 0; w < kPrepThreads / 32; w++) { sq += red[0][w]; sk += red[1][w]; }
    const float rq = 1.0f / sqrtf(sq / (float)nq + a.eps), rk = 1.0f / sqrtf(sk / (float)nk + a.eps);
    float *Kr = lm_state(a.k, a.dyn) + row * nk, *Q = a.q + (size_t)m * nq;
    auto value = [&](int c) {                     /* column c normed and rotated */
        const bool isq = c < nq;
        const int j = isq ? c : c - nq, d = j % a.dim;
        const float *gain = isq ? a.q_gain : a.k_gain;
        const float r = isq ? rq : rk;
        float v = buf[c] * r * __ldg(gain + j);
        if (d < a.rot) {
            const int i = d < half ? d : d - half, other = d < half ? half : -half;
            const float u = buf[c + other] * r * __ldg(gain + j + other);
            v = d < half ? v * cs[i] - u * cs[half + i] : v * cs[i] + u * cs[half + i];
        }
        return v;
    };
    if (((nq | nk | a.dim) & 3) == 0) {
        for (int c = tid * 4; c < nq + nk; c += kPrepThreads * 4) {
            const float4 v = make_float4(value(c), value(c + 1), value(c + 2), value(c + 3));
            const int j = c < nq ? c : c - nq, d = j % a.dim;
            if (c < nq) *reinterpret_cast<float4 *>(Q + j) = v;
            else kv_put4(Kr + j - d, a.dim, d, v, a.split);
        }
    } else {
        for (int c = tid; c < nq + nk; c += kPrepThreads) {
            const int j = c < nq ? c : c - nq, d = j % a.dim;
            if (c < nq) Q[j] = value(c);
            else kv_put(Kr + j - d, a.dim, d, value(c), a.split);
        }
    }
}

/* ------------------------------------------------------------------ any sizes, fp32 pipes */
/* PAIRS (row, query head) pairs of a KV head per CTA, 32 or 64 keys at a time; a thread holds PAIRS / 16 pairs x 2 or 4 keys of the
 * scores, then the same pairs x 4 * NV columns of the result, as packed fp32 pairs, so that a 16-byte read of shared
 * memory serves 4 to 16 multiply-adds. (Scores by dot products of a lane each, results a column a time through shared
 * memory: 390 rows of 16 heads of 128 took 405 us a layer, five rows at 400 keys 70 us.) 64 pairs for prompts, two
 * CTAs an SM at heads of 128; 16 for a few rows, where the keys are split over CTAs and tiles of 64 pairs would be
 * mostly empty. The last split to arrive merges in split order. */
constexpr int kGaThreads = 256, kGaKeys = 64, kGaFewKeys = 32, kGaManyPairs = 64;

/* rows of a multiple of four floats; an odd number of 16-byte pieces, so that eight rows' pieces lie in different banks */
inline __host__ __device__ int ga_ld(int n) { const int v = (n + 3) / 4 + 1; return 4 * (v | 1); }
inline __host__ __device__ int ga_stride(int vdim) { return (vdim + 3) / 4 * 4 + 4; }   /* a pair's partial result: columns, maximum, sum */
inline size_t ga_smem(int pairs, int keys, int dim, int vdim) {
    return sizeof(float) * ((size_t)pairs * ga_ld(dim) + std::max(keys * ga_ld(dim), pairs * (keys + 4)) + (size_t)keys * ((vdim + 3) / 4 * 4));
}

/* n rows of `size` floats or halves into shared memory, rows up to KEYS and columns up to a multiple of four as zeros. A warp takes a
 * row, or the two, four or eight that its lanes have room for (heads of 32 with three lanes in four idle: 25% longer than element
 * by element, 96 heads). A thread requests its loads together: none behind a condition or a conversion. True where a value is not finite. */
template <int KEYS, bool SPLIT, typename Row>
VB_DEVINL bool ga_load(float *to, int ld, int size, int n, const Row &row, int warp, int lane) {
    const int pieces = (size + 3) / 4, across = pieces > 16 ? 32 : pieces > 8 ? 16 : pieces > 4 ? 8 : 4, step = kGaThreads / across;
    const int first = warp * (32 / across) + lane / across;
    bool odd = false;
    for (int c = lane % across; c < pieces; c += across) {
        float4 v[KEYS / 8];
        if ((size & 3) == 0) {
            uint4 raw[KEYS / 8];
#pragma unroll
            for (int i = 0; i < KEYS / 8; i++) raw[i] = kv_raw4<SPLIT>(row(min(first + step * i, n - 1)), size, 4 * c);
#pragma unroll
            for (int i = 0; i < KEYS / 8; i++) v[i] = first + step * i < n ? kv_value4<SPLIT>(raw[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int i = 0; i < KEYS / 8; i++) {
                const int j = first + step * i;
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j >= n) continue;
                const float *head = row(j);
                v[i].x = kv_get(head, size, 4 * c, SPLIT);
                if (4 * c + 1 < size) v[i].y = kv_get(head, size, 4 * c + 1, SPLIT);
                if (4 * c + 2 < size) v[i].z = kv_get(head, size, 4 * c + 2, SPLIT);
                if (4 * c + 3 < size) v[i].w = kv_get(head, size, 4 * c + 3, SPLIT);
            }
        }
#pragma unroll
        for (int i = 0; i < KEYS / 8; i++) {
            const int j = first + step * i;
            if (j >= KEYS) break;
            *(float4 *)(to + (size_t)j * ld + 4 * c) = v[i];
            odd |= !(fabsf(v[i].x) < INFINITY && fabsf(v[i].y) < INFINITY && fabsf(v[i].z) < INFINITY && fabsf(v[i].w) < INFINITY);
        }
    }
    return odd;
}

/* grid = (tiles of pairs, KV heads, key splits) */
template <int PAIRS, int KEYS, int NV, bool SPLIT>
__global__ void __launch_bounds__(kGaThreads) lm_attn_generic_kernel(const LmAttn a, int M) {
    constexpr int TP = PAIRS / 16, TK = KEYS / 16, LDP = KEYS + 4;
    extern __shared__ __align__(16) float ga[];
    __shared__ float wgt[kLmAttnSplits][PAIRS], total[PAIRS];
    __shared__ int last_flag;
    pdl_launch_dependents();
    pdl_wait();
    const int dim = a.dim, vdim = a.vdim, group = a.heads / a.kv_heads, ld = ga_ld(dim), ldv = (vdim + 3) / 4 * 4;
    float *Q = ga, *K = Q + PAIRS * ld, *P = K, *V = K + (KEYS * ld > PAIRS * LDP ? KEYS * ld : PAIRS * LDP);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    const int g = blockIdx.y, p0 = blockIdx.x * PAIRS;
    const int np = M * group - p0 < PAIRS ? M * group - p0 : PAIRS;
    const int pos0 = a.dyn->pos;
    const KeyTiles kt = key_tiles<KEYS>(pos0 + p0 / group, pos0 + (p0 + np - 1) / group, a.window, a.keep);
    const int S_eff = (int)gridDim.z < kt.n_tiles ? (int)gridDim.z : kt.n_tiles;
    const int sp = blockIdx.z;
    if (sp >= S_eff) return;
    const int t0 = (int)((long long)kt.n_tiles * sp / S_eff), t1 = (int)((long long)kt.n_tiles * (sp + 1) / S_eff);
    const float *Kc = lm_state(a.k, a.dyn), *Vc = lm_state(a.v, a.dyn);

    for (int p = warp; p < PAIRS; p += kGaThreads / 32) {
        const float *q = a.q + (size_t)((p0 + p) / group) * a.heads * dim + (size_t)(g * group + (p0 + p) % group) * dim;
        for (int d = lane; d < (dim + 3) / 4 * 4; d += 32) Q[p * ld + d] = p < np && d < dim ? __ldcg(q + d) : 0.0f;
    }
    float mx[TP], den[TP];
    uint64_t o[TP][2 * NV];
    int at[TP];                                  /* positions of this thread's rows */
#pragma unroll
    for (int i = 0; i < TP; i++) {
        mx[i] = -INFINITY;
        den[i] = 0.0f;
        at[i] = pos0 + (p0 + ty * TP + i) / group;
#pragma unroll
        for (int c = 0; c < 2 * NV; c++) o[i][c] = 0ull;
    }

    for (int t = t0; t < t1; t++) {
        int j0, n;
        key_tile<KEYS>(kt, t, &j0, &n);
        __syncthreads();                         /* the last tile is read */
        ga_load<KEYS, SPLIT>(K, ld, dim, n, [&](int j) { return Kc + ((size_t)lm_ring_row(a.ring, j0 + j) * a.kv_heads + g) * dim; }, warp, lane);
        const bool odd = ga_load<KEYS, SPLIT>(V, ldv, vdim, n, [&](int j) { return Vc + ((size_t)lm_ring_row(a.ring, j0 + j) * a.kv_heads + g) * vdim; }, warp, lane);
        const bool any_odd = __syncthreads_or(odd);
        uint64_t acc[TP][TK] = {};
#pragma unroll 4
        for (int d = 0; d < dim; d += 4) {
            ulonglong2 q[TP], k[TK];
#pragma unroll
            for (int i = 0; i < TP; i++) q[i] = *(const ulonglong2 *)(Q + (ty * TP + i) * ld + d);
#pragma unroll
            for (int j = 0; j < TK; j++) k[j] = *(const ulonglong2 *)(K + (tx + 16 * j) * ld + d);
#pragma unroll
            for (int i = 0; i < TP; i++)
#pragma unroll
                for (int j = 0; j < TK; j++) acc[i][j] = vb_f2_fma(q[i].y, k[j].y, vb_f2_fma(q[i].x, k[j].x, acc[i][j]));
        }
        __syncthreads();                         /* weights take the keys' place */
#pragma unroll
        for (int i = 0; i < TP; i++) {
            float s[TK], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < TK; j++) {
                const int key = tx + 16 * j;
                const float2 e = vb_f2_get(acc[i][j]);
                s[j] = (e.x + e.y) * a.scale;
                if (a.softcap > 0.0f) s[j] = a.softcap * tanhf(s[j] / a.softcap);
                if (key >= n || !key_seen(at[i], j0 + key, a.window, a.keep)) s[j] = -INFINITY;
                top = fmaxf(top, s[j]);
            }
#pragma unroll
            for (int u = 8; u > 0; u >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, u));
            const float now = fmaxf(mx[i], top), c = mx[i] > -INFINITY ? expf(mx[i] - now) : 0.0f;
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < TK; j++) {
                const float w = s[j] > -INFINITY ? expf(s[j] - now) : 0.0f;
                P[(ty * TP + i) * LDP + tx + 16 * j] = w;
                sum += w;
            }
#pragma unroll
            for (int u = 8; u > 0; u >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, u);
            den[i] = den[i] * c + sum;
            mx[i] = now;
#pragma unroll
            for (int v = 0; v < 2 * NV; v++) o[i][v] = vb_f2_mul(o[i][v], vb_f2_pack(c, c));
        }
        __syncwarp();                            /* a pair's weights are read by the half warp that wrote them */
        for (int j = 0; j < n; j += 4) {         /* rows from n on are zeros */
            float4 w[TP];
#pragma unroll
            for (int i = 0; i < TP; i++) w[i] = *(const float4 *)(P + (ty * TP + i) * LDP + j);
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int c = 0; c < NV; c++) {
                    const int col = 64 * c + 4 * tx;
                    if (col >= ldv) continue;
                    const ulonglong2 v = *(const ulonglong2 *)(V + (j + u) * ldv + col);
#pragma unroll
                    for (int i = 0; i < TP; i++) {
                        /* zero times what is not finite: only where the key is seen */
                        if (any_odd && !(j + u < n && key_seen(at[i], j0 + j + u, a.window, a.keep))) continue;
                        const float wu = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
                        const uint64_t e = vb_f2_pack(wu, wu);
                        o[i][2 * c] = vb_f2_fma(e, v.x, o[i][2 * c]);
                        o[i][2 * c + 1] = vb_f2_fma(e, v.y, o[i][2 * c + 1]);
                    }
                }
        }
    }

    if (S_eff > 1) {
        /* several CTAs share these pairs: publish the slice, the last arrival merges in slice order */
        const int stride = ga_stride(vdim);
        const size_t tile = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
        float *po = a.scratch + tile * gridDim.z * PAIRS * stride;
#pragma unroll
        for (int i = 0; i < TP; i++) {
            float *mine = po + ((size_t)sp * PAIRS + ty * TP + i) * stride;
#pragma unroll
            for (int c = 0; c < NV; c++)
                if (64 * c + 4 * tx < ldv) *(ulonglong2 *)(mine + 64 * c + 4 * tx) = make_ulonglong2(o[i][2 * c], o[i][2 * c + 1]);
            if (tx == 0) *(float2 *)(mine + ldv) = make_float2(mx[i], den[i]);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            const unsigned t = atomicAdd(&a.tickets[tile], 1u);
            last_flag = t == (unsigned)(S_eff - 1);
            if (last_flag) a.tickets[tile] = 0u;
        }
        __syncthreads();
        if (!last_flag) return;
        __threadfence();
        if (tid < PAIRS) {
            float M0 = -INFINITY, L = 0.0f;
            for (int u = 0; u < S_eff; u++) M0 = fmaxf(M0, __ldcg(po + ((size_t)u * PAIRS + tid) * stride + ldv));
            for (int u = 0; u < S_eff; u++) {
                const float2 e = __ldcg((const float2 *)(po + ((size_t)u * PAIRS + tid) * stride + ldv));
                const float w = e.x > -INFINITY ? expf(e.x - M0) : 0.0f;
                wgt[u][tid] = w;
                L += w * e.y;
            }
            total[tid] = L;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TP; i++) {
            den[i] = total[ty * TP + i];
#pragma unroll
            for (int c = 0; c < 2 * NV; c++) o[i][c] = 0ull;
        }
        for (int u = 0; u < S_eff; u++)
#pragma unroll
            for (int i = 0; i < TP; i++) {
                const float *from = po + ((size_t)u * PAIRS + ty * TP + i) * stride;
                const float wu = wgt[u][ty * TP + i];
                const uint64_t w = vb_f2_pack(wu, wu);
#pragma unroll
                for (int c = 0; c < NV; c++) {
                    if (64 * c + 4 * tx >= ldv) continue;
                    const ulonglong2 v = __ldcg((const ulonglong2 *)(from + 64 * c + 4 * tx));
                    o[i][2 * c] = vb_f2_fma(w, v.x, o[i][2 * c]);
                    o[i][2 * c + 1] = vb_f2_fma(w, v.y, o[i][2 * c + 1]);
                }
            }
    }
#pragma unroll
    for (int i = 0; i < TP; i++) {
        const int p = ty * TP + i, row = (p0 + p) / group, c0 = (g * group + (p0 + p) % group) * vdim;
        if (p >= np) break;
#pragma unroll
        for (int c = 0; c < NV; c++) {
            const int col = 64 * c + 4 * tx;
            const float2 x = vb_f2_get(o[i][2 * c]), y = vb_f2_get(o[i][2 * c + 1]);
            const float e[4] = {x.x / den[i], x.y / den[i], y.x / den[i], y.y / den[i]};
            if ((vdim & 3) == 0) {
                if (col < vdim) lm_put4(a.out, row, c0 + col, e);
            } else {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (col + u < vdim) lm_put(a.out, row, c0 + col + u, e[u]);
            }
        }
    }
}

/* ------------------------------------------------------------------ one token */
constexpr int kSaThreads = 512, kSaWarps = 16;

/* grid = (key splits, KV heads). Every CTA sums the squares of the whole q and k projection itself
 * (a few L2 reads instead of another launch), norms and rotates its own heads, and attends over its
 * share of the visible keys: a warp serves one head of the group on one of 16 / (heads of the group)
 * subsets of the keys, KP keys in flight, a lane four dimensions per step. The last split owns the
 * new token and appends it. ND, NV: 128-wide steps of the key and value sizes. */
template <int ND, int NV, int KP, bool SPLIT>
__global__ void __launch_bounds__(kSaThreads) lm_attn_step_kernel(const LmAttn a, int lanes_h) {
    extern __shared__ __align__(16) float sa[];
    __shared__ float red[2][kSaWarps], sub_m[kSaWarps], sub_l[kSaWarps], wgt[kLmAttnSplits * kSaWarps];
    __shared__ int last_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dim = a.dim, vdim = a.vdim, group = a.heads / a.kv_heads, half = a.rot / 2;
    const int nq = a.heads * dim, nk = a.kv_heads * dim, nv = a.kv_heads * vdim;
    float *raw = sa;                                       /* [group * dim] own q, then [dim] own k */
    float *qs = raw + (group + 1) * dim;                   /* [group][dim] */
    float *os = qs + group * dim;                          /* [16 warps][vdim] */
    float *cs = os + kSaWarps * vdim;                      /* [rot] */
    pdl_launch_dependents();
    pdl_wait();
    const int sp = blockIdx.x, g = blockIdx.y;
    const int pos = a.dyn->pos;
    /* visible keys in order: the kept ones, then the window */
    const int n_keep = a.window > 0 ? (a.keep < pos + 1 ? a.keep : pos + 1) : 0;
    const int w0 = a.window > 0 ? (pos - a.window + 1 > n_keep ? pos - a.window + 1 : n_keep) : 0;
    const int n_keys = n_keep + (pos + 1 - w0);
    int S = (n_keys + 31) / 32;
    if (S > (int)gridDim.x) S = gridDim.x;
    if (sp >= S) return;
    const int x0 = (int)((long long)n_keys * sp / S), x1 = (int)((long long)n_keys * (sp + 1) / S);
    const bool writer = sp == S - 1;

    float sq = 0.0f, sk = 0.0f;
    const int own0 = g * group * dim, own1 = own0 + group * dim, k0 = nq + g * dim, k1 = k0 + dim;
    for (int c = tid * 4; c < nq + nk; c += kSaThreads * 4) {
        const float4 v = lm_sum4(a.qkv, 0, c);
        const float ss = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        if (c < nq) sq += ss; else sk += ss;
        if (c >= own0 && c < own1) *reinterpret_cast<float4 *>(raw + c - own0) = v;
        else if (c >= k0 && c < k1) *reinterpret_cast<float4 *>(raw + group * dim + c - k0) = v;
    }
    float *Kc = lm_state(a.k, a.dyn) + g * dim, *Vc = lm_state(a.v, a.dyn) + g * vdim;
    const size_t new_row = (size_t)lm_ring_row(a.ring, pos);
    if (writer)
        for (int c = tid; c < vdim; c += kSaThreads) kv_put(Vc + new_row * nv, vdim, c, lm_sum_batch(a.qkv, 0, nq + nk + g * vdim + c), SPLIT);
    for (int i = tid; i < half; i += kSaThreads) {
        lm_angle(pos, a.freq[i], a.freq[half + i], a.mag, &cs[i], &cs[half + i]);
    }
    sq = vb_warp_sum(sq);
    sk = vb_warp_sum(sk);
    if (lane == 0) { red[0][warp] = sq; red[1][warp] = sk; }
    __syncthreads();
    sq = sk = 0.0f;
#pragma unroll
    for (int w = 0; w < kSaWarps; w++) { sq += red[0][w]; sk += red[1][w]; }
    const float rq = 1.0f / sqrtf(sq / (float)nq + a.eps), rk = 1.0f / sqrtf(sk / (float)nk + a.eps);
    const int total = (writer ? group + 1 : group) * dim;
    for (int i = tid; i < total; i += kSaThreads) {
        const bool isq = i < group * dim;
        const int d = i % dim;
        const float *gain = isq ? a.q_gain + own0 + i : a.k_gain + g * dim + d;
        const float r = isq ? rq : rk;
        float v = raw[i] * r * __ldg(gain);
        if (d < a.rot) {
            const int j = d < half ? d : d - half, other = d < half ? half : -half;
            const float u = raw[i + other] * r * __ldg(gain + other);
            v = d < half ? v * cs[j] - u * cs[half + j] : v * cs[j] + u * cs[half + j];
        }
        if (isq) qs[i] = v;
        else kv_put(Kc + new_row * nk, dim, d, v, SPLIT);
    }
    __syncthreads();          /* the appended row is visible to this CTA */

    const int hh = warp % lanes_h, sub = warp / lanes_h, subs = kSaWarps / lanes_h;
    float mx = -INFINITY, den = 0.0f, o[NV][4];
#pragma unroll
    for (int i = 0; i < NV; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    if (hh < group) {
        float4 q[ND];
#pragma unroll
        for (int i = 0; i < ND; i++) {
            const int d = i * 128 + lane * 4;
            q[i] = d < dim ? *reinterpret_cast<const float4 *>(qs + hh * dim + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const int first = w0 > a.ring.keep ? (w0 - a.ring.keep) % a.ring.ring : 0;      /* ring place of the window's first key */
        for (int xb = x0 + sub; xb < x1; xb += KP * subs) {
            /* every load of the pass is requested unconditionally (beyond the range: the last key again), so that
             * they are all in flight together */
            float4 kk[KP][ND], vv[KP][NV];
#pragma unroll
            for (int u = 0; u < KP; u++) {
                int x = xb + u * subs;
                x = x < x1 ? x : x1 - 1;
                int r = first + x - n_keep;
                r = x < n_keep ? x : a.ring.keep + (r < a.ring.ring ? r : r - a.ring.ring);
#pragma unroll
                for (int i = 0; i < ND; i++) {
                    const int d = i * 128 + lane * 4;
                    kk[u][i] = kv_get4<SPLIT>(Kc + (size_t)r * nk, dim, d < dim ? d : 0);
                }
#pragma unroll
                for (int i = 0; i < NV; i++) {
                    const int d = i * 128 + lane * 4;
                    vv[u][i] = kv_get4<SPLIT>(Vc + (size_t)r * nv, vdim, d < vdim ? d : 0);
                }
            }
            float s[KP];
#pragma unroll
            for (int u = 0; u < KP; u++) {
                s[u] = 0.0f;
#pragma unroll
                for (int i = 0; i < ND; i++)
                    s[u] += q[i].x * kk[u][i].x + q[i].y * kk[u][i].y + q[i].z * kk[u][i].z + q[i].w * kk[u][i].w;
            }
            /* a lane ends up with the score of one of the pass's keys (32 / KP lanes share one) */
            constexpr int kShare = 32 / KP;
            vb_warp_multi_sum<KP>(s, lane);
            float sc = s[0] * a.scale;
            if (a.softcap > 0.0f) sc = a.softcap * tanhf(sc / a.softcap);
            if (xb + (lane / kShare) * subs >= x1) sc = -INFINITY;
            float top = sc;
#pragma unroll
            for (int off = kShare; off < 32; off <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
            top = fmaxf(top, mx);                         /* the first key of a pass is always there: finite */
            const float c = expf(mx - top), w = expf(sc - top);
            mx = top;
            den = den * c + w;                            /* this lane's key only; added up at the end */
#pragma unroll
            for (int i = 0; i < NV; i++) { o[i][0] *= c; o[i][1] *= c; o[i][2] *= c; o[i][3] *= c; }
#pragma unroll
            for (int u = 0; u < KP; u++) {
                const float wu = __shfl_sync(0xffffffffu, w, u * kShare);
#pragma unroll
                for (int i = 0; i < NV; i++) {
                    o[i][0] = fmaf(wu, vv[u][i].x, o[i][0]);
                    o[i][1] = fmaf(wu, vv[u][i].y, o[i][1]);
                    o[i][2] = fmaf(wu, vv[u][i].z, o[i][2]);
                    o[i][3] = fmaf(wu, vv[u][i].w, o[i][3]);
                }
            }
        }
#pragma unroll
        for (int off = 32 / KP; off < 32; off <<= 1) den += __shfl_xor_sync(0xffffffffu, den, off);
    }
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int d = i * 128 + lane * 4;
        if (d < vdim) *reinterpret_cast<float4 *>(os + warp * vdim + d) = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
    }
    if (lane == 0) { sub_m[warp] = mx; sub_l[warp] = den; }
    __syncthreads();
    /* merge the key subsets of every head, in order */
    const int stride = vdim + 2;
    float *po = a.scratch + (size_t)g * gridDim.x * group * stride;            /* [split][head][vdim + 2] */
    for (int i = tid; i < group * vdim; i += kSaThreads) {
        const int hd = i / vdim, d = i % vdim;
        float M0 = -INFINITY, L = 0.0f, O = 0.0f;
        for (int u = 0; u < subs; u++) M0 = fmaxf(M0, sub_m[u * lanes_h + hd]);
        for (int u = 0; u < subs; u++) {
            const int w = u * lanes_h + hd;
            const float f = sub_m[w] > -INFINITY ? expf(sub_m[w] - M0) : 0.0f;
            L = fmaf(sub_l[w], f, L);
            O = fmaf(os[w * vdim + d], f, O);
        }
        if (S == 1) {
            lm_put(a.out, 0, (g * group + hd) * vdim + d, O / L);
        } else {
            float *mine = po + ((size_t)sp * group + hd) * stride;
            mine[d] = O;
            if (d == 0) { mine[vdim] = M0; mine[vdim + 1] = L; }
        }
    }
    if (S == 1) return;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const unsigned t = atomicAdd(&a.tickets[g], 1u);
        last_flag = t == (unsigned)(S - 1);
        if (last_flag) a.tickets[g] = 0u;
    }
    __syncthreads();
    if (!last_flag) return;
    __threadfence();
    /* weights of the slices per head, then the slices in order */
    if (tid < group) {
        float m[kLmAttnSplits], M0 = -INFINITY, L = 0.0f;
#pragma unroll
        for (int u = 0; u < kLmAttnSplits; u++) m[u] = u < S ? __ldcg(po + ((size_t)u * group + tid) * stride + vdim) : -INFINITY;
#pragma unroll
        for (int u = 0; u < kLmAttnSplits; u++) M0 = fmaxf(M0, m[u]);
#pragma unroll
        for (int u = 0; u < kLmAttnSplits; u++)
            if (u < S) {
                const float f = expf(m[u] - M0);
                L = fmaf(__ldcg(po + ((size_t)u * group + tid) * stride + vdim + 1), f, L);
                wgt[u * kSaWarps + tid] = f;
            }
        sub_l[tid] = L;
    }
    __syncthreads();
    for (int i = tid; i < group * vdim; i += kSaThreads) {
        const int hd = i / vdim, d = i % vdim;
        float t[kLmAttnSplits], O = 0.0f;
#pragma unroll
        for (int u = 0; u < kLmAttnSplits; u++) t[u] = u < S ? __ldcg(po + ((size_t)u * group + hd) * stride + d) : 0.0f;
#pragma unroll
        for (int u = 0; u < kLmAttnSplits; u++)
            if (u < S) O = fmaf(t[u], wgt[u * kSaWarps + hd], O);
        lm_put(a.out, 0, (g * group + hd) * vdim + d, O / sub_l[hd]);
    }
}

inline size_t step_smem(const LmAttn &a) {
    const int group = a.heads / a.kv_heads;
    return sizeof(float) * ((size_t)(2 * group + 1) * a.dim + (size_t)kSaWarps * a.vdim + a.rot + 4);
}

template <int ND, int NV, int KP, bool SPLIT>
int launch_attn_step(const LmAttn &a, int splits, int lanes_h, cudaStream_t st) {
    const size_t smem = step_smem(a);
    static size_t set = 48 * 1024;
    if (smem > set) {
        if (cudaFuncSetAttribute(lm_attn_step_kernel<ND, NV, KP, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        set = smem;
    }
    return ok(launch_pdl(lm_attn_step_kernel<ND, NV, KP, SPLIT>, dim3(splits, a.kv_heads), dim3(kSaThreads), smem, st, a, lanes_h));
}

/* ------------------------------------------------------------------ one token, few query heads a key head */
/* The same for up to four query heads a KV head and heads of up to 128: grid = (key splits, KV heads), the splits of a KV head a
 * cluster; a warp takes eight keys at a time for all heads of the group, and a CTA sends the others' columns of its
 * result into their shared memory (asynchronous stores that count on the receiver's barrier), so that each merges its share
 * in split order. Bound by latency: whatever the kernel before does not make is fetched before the wait for it - the
 * position, the angles, the gains, the first pass of keys and values (earlier steps are complete: a step's first kernel
 * is a plain launch). One warp per head and a merge by the last CTA through global memory: 17 us at 220 keys of 8 x 128. */
constexpr int kSgThreads = 256, kSgWarps = 8, kSgKeys = 8, kSgHeads = 4, kSgDim = 128, kSgSplits = 8, kSgColumns = 8;
constexpr int kSgMost = 160;              /* keys a CTA, at most: lm_attn_step_near */

template <bool SPLIT>
__global__ void __launch_bounds__(kSgThreads, 2) lm_attn_step_group_kernel(const LmAttn a) {
    __shared__ __align__(16) float raw[(kSgHeads + 1) * kSgDim], qs[kSgHeads][kSgDim], ks[kSgDim], vs[kSgDim], cs[kSgDim];
    __shared__ __align__(16) float warp_o[kSgWarps][kSgHeads][kSgDim];
    __shared__ float2 warp_ml[kSgWarps][kSgHeads];         /* maximum, sum */
    __shared__ float4 slices[kSgThreads];                  /* [S][columns of this CTA / 2]: two columns, maximum, sum */
    __shared__ float red[2][kSgWarps];
    __shared__ uint64_t arrived;
    __shared__ volatile int gave_up;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid == 0) {
        vb_mbar_init(&arrived, 1);
        gave_up = 0;
        vb_mbar_init_fence();
        vb_mbar_arrive_expect_tx(&arrived, (uint32_t)sizeof(slices));
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int dim = a.dim, vdim = a.vdim, group = a.heads / a.kv_heads, half = a.rot / 2;
    const int nq = a.heads * dim, nk = a.kv_heads * dim, nv = a.kv_heads * vdim;
    const int sp = blockIdx.x, S = gridDim.x, g = blockIdx.y;
    const int pos = __ldcg(&a.dyn->pos), slot = __ldcg(&a.dyn->slot);
    /* visible keys in order: the kept ones, then the window; the new token is the last */
    const int n_keep = a.window > 0 ? (a.keep < pos + 1 ? a.keep : pos + 1) : 0;
    const int w0 = a.window > 0 ? (pos - a.window + 1 > n_keep ? pos - a.window + 1 : n_keep) : 0;
    const int n_keys = n_keep + (pos + 1 - w0);
    const int x0 = (int)((long long)n_keys * sp / S), x1 = (int)((long long)n_keys * (sp + 1) / S);
    const bool writer = sp == S - 1;
    float *Kc = a.k.base + (size_t)slot * a.k.slab + g * dim, *Vc = a.v.base + (size_t)slot * a.v.slab + g * vdim;
    const int first = w0 > a.ring.keep ? (w0 - a.ring.keep) % a.ring.ring : 0;      /* ring place of the window's first key */
    uint4 kq[kSgKeys], vq[kSgKeys];
    /* keys xb, xb + 8, ...: requested without a branch or a conversion between them, so that all are in flight together (16 trips
     * one after another, 8 us a pass, where each was behind a condition); beyond the slice and for the new token: not used */
    const int dk = 4 * lane < dim ? 4 * lane : 0, dv = 4 * lane < vdim ? 4 * lane : 0;
    auto fetch = [&](int xb) {
#pragma unroll
        for (int u = 0; u < kSgKeys; u++) {
            int x = xb + u * kSgWarps;
            x = x < x1 ? x : x1 > 0 ? x1 - 1 : 0;
            int r = first + x - n_keep;
            r = x < n_keep ? x : a.ring.keep + (r < a.ring.ring ? r : r - a.ring.ring);
            kq[u] = kv_raw4<SPLIT>(Kc + (size_t)r * nk, dim, dk);
            vq[u] = kv_raw4<SPLIT>(Vc + (size_t)r * nv, vdim, dv);
        }
    };
    int xb = x0 + warp;
    fetch(xb);
    for (int i = tid; i < half; i += kSgThreads) lm_angle(pos, a.freq[i], a.freq[half + i], a.mag, &cs[i], &cs[half + i]);
    const int own0 = g * group * dim, k0 = nq + g * dim, total = (writer ? group + 1 : group) * dim;
    constexpr int kMine = (kSgHeads + 1) * kSgDim / kSgThreads + 1;
    float gain[kMine];
#pragma unroll
    for (int u = 0; u < kMine; u++) {
        const int i = tid + u * kSgThreads;
        gain[u] = i >= total ? 0.0f : i < group * dim ? __ldg(a.q_gain + own0 + i) : __ldg(a.k_gain + g * dim + i - group * dim);
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");             /* all barriers of the cluster are set up */
    pdl_wait();

    /* every CTA sums the squares of the whole q and k projection itself, up to 8 x 1024 columns requested together */
    float sq = 0.0f, sk = 0.0f;
    for (int c0 = tid * 4; c0 < nq + nk; c0 += kSgColumns * kSgThreads * 4) {
        float4 v[kSgColumns];
#pragma unroll
        for (int u = 0; u < kSgColumns; u++) v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
        for (int p = 0; p < a.qkv.n; p++) {
            const float *at = a.qkv.p + (size_t)p * a.qkv.stride;
            float4 t[kSgColumns];
#pragma unroll
            for (int u = 0; u < kSgColumns; u++) {
                const int c = c0 + u * kSgThreads * 4;
                t[u] = c < nq + nk ? vb_ldcg4(at + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < kSgColumns; u++) { v[u].x += t[u].x; v[u].y += t[u].y; v[u].z += t[u].z; v[u].w += t[u].w; }
        }
#pragma unroll
        for (int u = 0; u < kSgColumns; u++) {
            const int c = c0 + u * kSgThreads * 4;
            const float ss = v[u].x * v[u].x + v[u].y * v[u].y + v[u].z * v[u].z + v[u].w * v[u].w;
            if (c < nq) sq += ss;
            else if (c < nq + nk) sk += ss;
            if (c >= own0 && c < own0 + group * dim) *reinterpret_cast<float4 *>(raw + c - own0) = v[u];
            else if (c >= k0 && c < k0 + dim) *reinterpret_cast<float4 *>(raw + group * dim + c - k0) = v[u];
        }
    }
    const size_t new_row = (size_t)lm_ring_row(a.ring, pos);
    /* what the cache keeps of the new token is what this step attends to */
    auto kept = [](float v) {
        if constexpr (!SPLIT) return v;
        uint32_t hi, lo;
        hilo(v, hi, lo);
        return __uint_as_float(hi << 16) + __uint_as_float(lo << 16);
    };
    if (writer && tid < vdim) {
        const float v = lm_sum_batch(a.qkv, 0, nq + nk + g * vdim + tid);
        vs[tid] = kept(v);
        kv_put(Vc + new_row * nv, vdim, tid, v, SPLIT);
    }
    sq = vb_warp_sum(sq);
    sk = vb_warp_sum(sk);
    if (lane == 0) { red[0][warp] = sq; red[1][warp] = sk; }
    __syncthreads();
    sq = sk = 0.0f;
#pragma unroll
    for (int w = 0; w < kSgWarps; w++) { sq += red[0][w]; sk += red[1][w]; }
    const float rq = 1.0f / sqrtf(sq / (float)nq + a.eps), rk = 1.0f / sqrtf(sk / (float)nk + a.eps);
#pragma unroll
    for (int u = 0; u < kMine; u++) {
        const int i = tid + u * kSgThreads;
        if (i >= total) continue;
        const bool isq = i < group * dim;
        const int d = i % dim;
        const float r = isq ? rq : rk;
        float v = raw[i] * r * gain[u];
        if (d < a.rot) {
            const int j = d < half ? d : d - half, other = d < half ? half : -half;
            const float y = raw[i + other] * r * __ldg((isq ? a.q_gain + own0 + i : a.k_gain + g * dim + d) + other);
            v = d < half ? v * cs[j] - y * cs[half + j] : v * cs[j] + y * cs[half + j];
        }
        if (isq) {
            qs[i / dim][d] = v;
        } else {
            ks[d] = kept(v);
            kv_put(Kc + new_row * nk, dim, d, v, SPLIT);
        }
    }
    __syncthreads();

    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 q4[kSgHeads], o[kSgHeads];
#pragma unroll
    for (int h = 0; h < kSgHeads; h++) {
        q4[h] = h < group && 4 * lane < dim ? *reinterpret_cast<const float4 *>(&qs[h][4 * lane]) : zero;
        o[h] = zero;
    }
    float mx = -INFINITY, den = 0.0f;                      /* of head lane / 8 */
    static_assert(kSgKeys * kSgHeads == 32, "a lane per key and head");
    while (xb < x1) {
        float s[32];                                       /* [head][key] */
#pragma unroll
        for (int u = 0; u < kSgKeys; u++) {
            const int x = xb + u * kSgWarps;
            float4 k = kv_value4<SPLIT>(kq[u]);
            if (writer && x == n_keys - 1) k = *reinterpret_cast<const float4 *>(ks + dk);
            if (4 * lane >= dim) k = zero;
#pragma unroll
            for (int h = 0; h < kSgHeads; h++)
                s[h * kSgKeys + u] = q4[h].x * k.x + q4[h].y * k.y + q4[h].z * k.z + q4[h].w * k.w;
        }
        vb_warp_halve32(s, lane);
        float e = s[0] * a.scale;
        if (a.softcap > 0.0f) e = a.softcap * tanhf(e / a.softcap);
        if (xb + (lane % kSgKeys) * kSgWarps >= x1) e = -INFINITY;
        float top = e;
#pragma unroll
        for (int n = kSgKeys / 2; n > 0; n >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, n));
        const float now = fmaxf(mx, top), c = expf(mx - now), w = expf(e - now);      /* the first key of a pass is always there: finite */
        float sum = w;
#pragma unroll
        for (int n = kSgKeys / 2; n > 0; n >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, n);
        den = den * c + sum;
        mx = now;
#pragma unroll
        for (int h = 0; h < kSgHeads; h++) {
            const float ch = __shfl_sync(0xffffffffu, c, h * kSgKeys);
            o[h].x *= ch; o[h].y *= ch; o[h].z *= ch; o[h].w *= ch;
        }
#pragma unroll
        for (int u = 0; u < kSgKeys; u++) {
            const int x = xb + u * kSgWarps;
            float4 v = kv_value4<SPLIT>(vq[u]);
            if (writer && x == n_keys - 1) v = *reinterpret_cast<const float4 *>(vs + dv);
            if (x >= x1) v = zero;                         /* whatever lies there: its weight is zero, and so must it be */
#pragma unroll
            for (int h = 0; h < kSgHeads; h++) {
                const float wu = __shfl_sync(0xffffffffu, w, h * kSgKeys + u);
                o[h].x = fmaf(wu, v.x, o[h].x); o[h].y = fmaf(wu, v.y, o[h].y);
                o[h].z = fmaf(wu, v.z, o[h].z); o[h].w = fmaf(wu, v.w, o[h].w);
            }
        }
        xb += kSgKeys * kSgWarps;
        if (xb < x1) fetch(xb);
    }
#pragma unroll
    for (int h = 0; h < kSgHeads; h++) *reinterpret_cast<float4 *>(&warp_o[warp][h][4 * lane]) = o[h];
    if (lane % kSgKeys == 0) warp_ml[warp][lane / kSgKeys] = make_float2(mx, den);
    __syncthreads();

    /* the warps' results, to the CTA that merges these columns: thread = (head, pair of columns) */
    const int share = kSgThreads / S;
    {
        const int h = tid / (kSgDim / 2), d = tid % (kSgDim / 2);
        float M0 = -INFINITY, L = 0.0f;
        float2 O = make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < kSgWarps; u++) M0 = fmaxf(M0, warp_ml[u][h].x);
#pragma unroll
        for (int u = 0; u < kSgWarps; u++) {
            const float2 ml = warp_ml[u][h], v = *reinterpret_cast<const float2 *>(&warp_o[u][h][2 * d]);
            const float f = ml.x > -INFINITY ? expf(ml.x - M0) : 0.0f;
            L = fmaf(ml.y, f, L);
            O.x = fmaf(v.x, f, O.x);
            O.y = fmaf(v.y, f, O.y);
        }
        vb_cluster_send(&slices[sp * share + tid % share], &arrived, tid / share, O.x, O.y, M0, L);
    }
    if (!vb_mbar_wait_cluster(&arrived, &gave_up, a.status, 53)) return;
    const int i = sp * share + tid, h = i / (kSgDim / 2), c = 2 * (i % (kSgDim / 2));
    if (tid < share && h < group && c < vdim) {
        float2 O = make_float2(0.f, 0.f);
        float M0 = -INFINITY, L = 0.0f;
        for (int u = 0; u < S; u++) M0 = fmaxf(M0, slices[u * share + tid].z);
        for (int u = 0; u < S; u++) {
            const float4 e = slices[u * share + tid];
            const float f = e.z > -INFINITY ? expf(e.z - M0) : 0.0f;
            L = fmaf(e.w, f, L);
            O.x = fmaf(e.x, f, O.x);
            O.y = fmaf(e.y, f, O.y);
        }
        lm_put(a.out, 0, (g * group + h) * vdim + c, O.x / L);
        lm_put(a.out, 0, (g * group + h) * vdim + c + 1, O.y / L);
    }
}

/* ------------------------------------------------------------------ prompts on the tensor cores (vb_attn_tc.cuh) */
/* Rows of a value tile beyond its keys: their weights are zero, and so must they be. */
template <int BLOCKS>
VB_DEVINL void clear_keys(unsigned char *slot, int lw, int lane, int n) {
    for (int key = n > lw * 16 ? n : lw * 16; key < lw * 16 + 16; key++)
        for (int f = lane; f < 2 * BLOCKS * 8; f += 32) *reinterpret_cast<uint4 *>(slot + (f >> 3) * kAtBlock + at_off(key, f)) = make_uint4(0u, 0u, 0u, 0u);
}

/* Keys and values from a cache of split rows. */
struct AtCache {
    static constexpr bool kBoxes = false, kParts = false;
    const LmDyn *dyn;
    const float *q;
    LmState k, v;
    LmRing ring;
    LmSink out;
    int heads, kv_heads, dim, vdim;
    const float *kc, *vc;
    VB_DEVINL void start() { kc = lm_state(k, dyn); vc = lm_state(v, dyn); }
    VB_DEVINL int rows(const AtArgs &a) const { return a.M; }
    VB_DEVINL const AtCache &here() const { return *this; }
    VB_DEVINL int pos0() const { return dyn->pos; }
    VB_DEVINL float4 q4(int row, int head, int d, int) const {
        return d < dim ? vb_ldcg4(q + ((size_t)row * heads + head) * dim + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    VB_DEVINL float4 turned(int, int, int, float4 x) const { return x; }
    VB_DEVINL bool boxes(int j0, int n) const { return n == kAtKeys && lm_ring_row(ring, j0 + kAtKeys - 1) - lm_ring_row(ring, j0) == kAtKeys - 1; }
    template <int BLOCKS>
    VB_DEVINL void box(const CUtensorMap *map, int size, unsigned char *slot, int g, int j0, uint64_t *bar) const {
        const int row = lm_ring_row(ring, j0);
#pragma unroll
        for (int b = 0; b < 2 * BLOCKS; b++) at_tma(slot + b * kAtBlock, map, g * 2 * size + (b / BLOCKS) * size + (b % BLOCKS) * 64, row, dyn->slot, bar);
    }
    template <int BLOCKS>
    VB_DEVINL void tma_keys(const AtArgs &, const AtMaps &m, unsigned char *slot, int g, int j0, uint64_t *bar) const {
        box<BLOCKS>(&m.k, dim, slot, g, j0, bar);
    }
    template <int BLOCKS>
    VB_DEVINL void tma_values(const AtArgs &, const AtMaps &m, unsigned char *slot, int g, int j0, uint64_t *bar) const {
        box<BLOCKS>(&m.v, vdim, slot, g, j0, bar);
    }
    template <int BLOCKS>
    VB_DEVINL void rows(const float *cache, int size, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        const int key = lw * 16 + (lane & 15);
        const int own = lm_ring_row(ring, j0 + (key < n ? key : n - 1));
        const int ld = kv_heads * size, per = size / 8;
        int at[16];
#pragma unroll
        for (int x = 0; x < 16; x++) at[x] = __shfl_sync(0xffffffffu, own, x);
#pragma unroll 1
        for (int f = lane; f < 2 * per; f += 32) {
            const int plane = f >= per ? 1 : 0, chunk = f - plane * per;
            unsigned char *block = slot + (plane * BLOCKS + (chunk >> 3)) * kAtBlock;
            const uint16_t *col = reinterpret_cast<const uint16_t *>(cache + g * size) + f * 8;
#pragma unroll
            for (int x = 0; x < 16; x++)
                if (lw * 16 + x < n) lm_cp16(block + at_off(lw * 16 + x, chunk), col + (size_t)at[x] * ld * 2);
        }
    }
    template <int BLOCKS>
    VB_DEVINL void keys(const AtArgs &, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        rows<BLOCKS>(kc, dim, slot, g, lw, lane, j0, n);
    }
    template <int BLOCKS>
    VB_DEVINL void values(const AtArgs &, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        rows<BLOCKS>(vc, vdim, slot, g, lw, lane, j0, n);
        clear_keys<BLOCKS>(slot, lw, lane, n);
    }
    VB_DEVINL float gate(int, int) const { return 1.0f; }
    VB_DEVINL void put4(int row, int c, const float (&e)[4]) const { lm_put4(out, row, c, e); }
};

/* Every head has keys and values of its own, read out of a latent (LmWide): a head's own columns of the written-out
 * rows, then the key part that all heads share from the latent's cache row. ONE: q comes in one part, as from GEMMs of many rows (without
 * the code for several 153 -> 138 us, 2048 rows of heads of 192). */
template <bool ONE>
struct AtWide {
    static constexpr bool kBoxes = false, kParts = !ONE;
    const LmDyn *dyn;
    LmWide w;
    LmRing ring;
    LmSink out;
    int heads, dim, vdim, rot;
    VB_DEVINL void start() { w.cache += (size_t)dyn->slot * w.slab; }
    VB_DEVINL int rows(const AtArgs &a) const { return a.M; }
    VB_DEVINL const AtWide &here() const { return *this; }
    VB_DEVINL int pos0() const { return dyn->pos; }
    VB_DEVINL int parts() const { return w.q.n; }
    VB_DEVINL float4 q4(int row, int head, int d, int part) const {
        if (d >= dim) return make_float4(0.f, 0.f, 0.f, 0.f);
        return vb_ldcg4(w.q.p + (ONE ? 0 : (size_t)part * w.q.stride) + (size_t)row * w.q.ld + head * dim + d);
    }
    VB_DEVINL float4 turned(int row, int, int d, float4 x) const {
        const int half = rot / 2, i0 = (d - (dim - w.rot_dim)) / 2;
        float e[4] = {x.x, x.y, x.z, x.w};
        if (d >= dim - w.rot_dim && d < dim) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (i0 + i < half) {
                    const float c = w.cs[(size_t)row * rot + i0 + i], s = w.cs[(size_t)row * rot + half + i0 + i];
                    const float u = e[2 * i], t = e[2 * i + 1];
                    e[2 * i] = u * c - t * s;
                    e[2 * i + 1] = t * c + u * s;
                }
            }
        }
        return make_float4(e[0], e[1], e[2], e[3]);
    }
    VB_DEVINL bool boxes(int j0, int n) const { return n == kAtKeys && lm_ring_row(ring, j0 + kAtKeys - 1) - lm_ring_row(ring, j0) == kAtKeys - 1; }
    template <int BLOCKS>
    VB_DEVINL void tma_keys(const AtArgs &, const AtMaps &m, unsigned char *slot, int g, int j0, uint64_t *bar) const {
        const int own = (dim - w.rot_dim) / 64, row = w.rank + w.rot_dim;
#pragma unroll
        for (int b = 0; b < 2 * BLOCKS; b++) {
            const int plane = b / BLOCKS, c = b % BLOCKS;
            if (c < own) at_tma(slot + b * kAtBlock, &m.k, (g * own + c) * 64, j0 - w.first, plane, bar);
            else at_tma(slot + b * kAtBlock, &m.k2, plane * row + w.rank + (c - own) * 64, lm_ring_row(ring, j0), dyn->slot, bar);
        }
    }
    template <int BLOCKS>
    VB_DEVINL void tma_values(const AtArgs &, const AtMaps &m, unsigned char *slot, int g, int j0, uint64_t *bar) const {
#pragma unroll
        for (int b = 0; b < 2 * BLOCKS; b++) at_tma(slot + b * kAtBlock, &m.v, w.v0 + g * vdim + (b % BLOCKS) * 64, j0 - w.first, b / BLOCKS, bar);
    }
    template <int BLOCKS>
    VB_DEVINL void keys(const AtArgs &, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        const int own = (dim - w.rot_dim) / 8, per = dim / 8, row = w.rank + w.rot_dim;
        const int first = j0 - w.first + lw * 16;
        const int key = lw * 16 + (lane & 15);
        const int mine = lm_ring_row(ring, j0 + (key < n ? key : n - 1));
        int at[16];
#pragma unroll
        for (int x = 0; x < 16; x++) at[x] = __shfl_sync(0xffffffffu, mine, x);
#pragma unroll 1
        for (int f = lane; f < 2 * per; f += 32) {
            const int plane = f >= per ? 1 : 0, chunk = f - plane * per;
            unsigned char *block = slot + (plane * BLOCKS + (chunk >> 3)) * kAtBlock;
            const uint16_t *p = chunk < own ? w.kv + plane * w.plane + (size_t)first * w.ld + g * own * 8 + chunk * 8
                                            : reinterpret_cast<const uint16_t *>(w.cache) + plane * row + w.rank + (chunk - own) * 8;
#pragma unroll
            for (int x = 0; x < 16; x++)
                if (lw * 16 + x < n) lm_cp16(block + at_off(lw * 16 + x, chunk), p + (chunk < own ? (size_t)x * w.ld : (size_t)at[x] * row * 2));
        }
    }
    template <int BLOCKS>
    VB_DEVINL void values(const AtArgs &, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        const int per = vdim / 8, first = j0 - w.first + lw * 16;
#pragma unroll 1
        for (int f = lane; f < 2 * per; f += 32) {
            const int plane = f >= per ? 1 : 0, chunk = f - plane * per;
            unsigned char *block = slot + (plane * BLOCKS + (chunk >> 3)) * kAtBlock;
            const uint16_t *p = w.kv + plane * w.plane + (size_t)first * w.ld + w.v0 + g * vdim + chunk * 8;
#pragma unroll
            for (int x = 0; x < 16; x++)
                if (lw * 16 + x < n) lm_cp16(block + at_off(lw * 16 + x, chunk), p + (size_t)x * w.ld);
        }
        clear_keys<BLOCKS>(slot, lw, lane, n);
    }
    VB_DEVINL float gate(int row, int head) const { return w.gate[(size_t)row * heads + head]; }
    VB_DEVINL void put4(int row, int c, const float (&e)[4]) const { lm_put4(out, row, c, e); }
};

AtArgs at_args(const LmAttn &a, int M) { return {M, a.heads, a.kv_heads, a.dim, a.vdim, a.window, a.keep, a.scale, a.softcap, a.status, 0}; }

constexpr int kSplitBudget = 296;        /* two CTAs per SM */
constexpr int kStepCtas = 148;           /* one-token kernel: one CTA per SM */

} // namespace

size_t lm_attn_scratch_floats(int heads, int kv_heads, int vdim) {
    (void)heads; (void)kv_heads;
    return std::max((size_t)kSplitBudget * kGaManyPairs * ga_stride(vdim), (size_t)kSplitBudget * kLmAttnPairs * (vdim + 2));
}
int lm_attn_ticket_count(int heads, int kv_heads) {
    (void)heads; (void)kv_heads;
    return kSplitBudget;
}

int lm_attn_prepare(const LmAttn &a, int M, cudaStream_t st) {
    const size_t smem = sizeof(float) * ((size_t)(a.heads + a.kv_heads) * a.dim + a.rot);
    if (smem > 200 * 1024) return -1;
    static size_t set = 48 * 1024;
    if (smem > set) {
        if (cudaFuncSetAttribute(lm_attn_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        set = smem;
    }
    return ok(launch_pdl(lm_attn_prepare_kernel, dim3(M), dim3(kPrepThreads), smem, st, a));
}

template <int PAIRS, int KEYS, int NV, bool SPLIT>
static int launch_generic(const LmAttn &a, int M, cudaStream_t st) {
    const size_t smem = ga_smem(PAIRS, KEYS, a.dim, a.vdim);
    if (smem > 200 * 1024) return -1;
    static size_t set = 32 * 1024;      /* 48 KB without asking, static arrays included */
    if (smem > set) {
        if (cudaFuncSetAttribute(lm_attn_generic_kernel<PAIRS, KEYS, NV, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        set = smem;
    }
    const int tiles = (M * (a.heads / a.kv_heads) + PAIRS - 1) / PAIRS;
    int splits = kSplitBudget / (tiles * a.kv_heads);
    splits = splits < 1 ? 1 : splits > kLmAttnSplits ? kLmAttnSplits : splits;
    return ok(launch_pdl(lm_attn_generic_kernel<PAIRS, KEYS, NV, SPLIT>, dim3(tiles, a.kv_heads, splits), dim3(kGaThreads), smem, st, a, M));
}

template <int PAIRS, int KEYS>
static int launch_generic(const LmAttn &a, int M, cudaStream_t st) {
    if (a.vdim > 128) return a.split ? launch_generic<PAIRS, KEYS, 4, true>(a, M, st) : launch_generic<PAIRS, KEYS, 4, false>(a, M, st);
    return a.split ? launch_generic<PAIRS, KEYS, 2, true>(a, M, st) : launch_generic<PAIRS, KEYS, 2, false>(a, M, st);
}

int lm_attn_generic(const LmAttn &a, int M, cudaStream_t st) {
    if (a.dim > 256 || a.vdim > 256) return -1;
    const int pairs = M * (a.heads / a.kv_heads);
    if (pairs > kGaManyPairs / 2) return launch_generic<kGaManyPairs, kGaKeys>(a, M, st);
    /* Few pairs and few keys: tiles of 32 keys, twice the CTAs, while those of 64 leave SMs without one. Two rows of eight heads of
     * 128, a layer of an attention-only model at 220 keys: 47.8 us with 64, 39.4 with 32, 38.0 with a tile's loads in flight
     * together besides; 32 in 32 bits at 1000 keys 51.8, 64 49.4, before the latter. */
    const long long ctas = (long long)((pairs + kLmAttnPairs - 1) / kLmAttnPairs) * a.kv_heads * ((a.most + kGaKeys - 1) / kGaKeys);
    return ctas < kStepCtas ? launch_generic<kLmAttnPairs, kGaFewKeys>(a, M, st) : launch_generic<kLmAttnPairs, kGaKeys>(a, M, st);
}

bool lm_attn_mma_ok(int dim, int vdim) { return dim <= 128 && vdim <= 128 && dim % 8 == 0 && vdim % 8 == 0; }

int lm_attn_mma(const LmAttn &a, int M, cudaStream_t st) {
    AtCache c = {};
    c.dyn = a.dyn; c.q = a.q; c.k = a.k; c.v = a.v; c.ring = a.ring; c.out = a.out;
    c.heads = a.heads; c.kv_heads = a.kv_heads; c.dim = a.dim; c.vdim = a.vdim;
    AtArgs t = at_args(a, M);
    AtMaps m = {};
    if (a.dim % 64 == 0 && a.vdim % 64 == 0) {
        const uint64_t rows = (uint64_t)a.ring.keep + a.ring.ring, ck = (uint64_t)2 * a.kv_heads * a.dim, cv = (uint64_t)2 * a.kv_heads * a.vdim;
        t.tma = tc_map3(&m.k, a.k.base, a.slots, a.k.slab * 4, rows, ck * 2, ck, kAtKeys) == 0 &&
                tc_map3(&m.v, a.v.base, a.slots, a.v.slab * 4, rows, cv * 2, cv, kAtKeys) == 0;
    }
    if (a.dim <= 64) return a.vdim <= 64 ? launch_attn_tc<1, 1>(t, c, st, m) : launch_attn_tc<1, 2>(t, c, st, m);
    return a.vdim <= 64 ? launch_attn_tc<2, 1>(t, c, st, m) : launch_attn_tc<2, 2>(t, c, st, m);
}

bool lm_attn_wide_ok(int plain, int rot_dim, int vdim) {
    return plain + rot_dim <= 192 && vdim <= 128 && plain % 8 == 0 && rot_dim % 8 == 0 && vdim % 8 == 0;
}

template <bool ONE>
static int launch_wide(const LmAttn &a, const LmWide &w, int M, cudaStream_t st) {
    AtWide<ONE> c = {};
    c.dyn = a.dyn; c.w = w; c.ring = a.ring; c.out = a.out;
    c.heads = a.heads; c.dim = a.dim; c.vdim = a.vdim; c.rot = a.rot;
    AtArgs t = at_args(a, M);
    AtMaps m = {};
    if (a.dim % 64 == 0 && w.rot_dim % 64 == 0 && a.vdim % 64 == 0) {
        const uint64_t row = (uint64_t)w.rank + w.rot_dim, rows = w.plane / w.ld;
        t.tma = tc_map3(&m.k, w.kv, 2, w.plane * 2, rows, (uint64_t)w.ld * 2, w.ld, kAtKeys) == 0 &&
                (w.rot_dim == 0 || tc_map3(&m.k2, w.cache, a.slots, w.slab * 4, (uint64_t)a.ring.keep + a.ring.ring, row * 4, row * 2, kAtKeys) == 0);
        m.v = m.k;
    }
    const bool v1 = a.vdim <= 64;
    if (a.dim <= 64) return v1 ? launch_attn_tc<1, 1>(t, c, st, m) : launch_attn_tc<1, 2>(t, c, st, m);
    if (a.dim <= 128) return v1 ? launch_attn_tc<2, 1>(t, c, st, m) : launch_attn_tc<2, 2>(t, c, st, m);
    return v1 ? launch_attn_tc<3, 1>(t, c, st, m) : launch_attn_tc<3, 2>(t, c, st, m);
}

int lm_attn_wide(const LmAttn &a, const LmWide &w, int M, cudaStream_t st) {
    return w.q.n == 1 ? launch_wide<true>(a, w, M, st) : launch_wide<false>(a, w, M, st);
}

bool lm_attn_step_ok(const LmAttn &a) {
    return a.heads / a.kv_heads <= kSaWarps && a.kv_heads <= kSplitBudget && a.dim % 4 == 0 && a.vdim % 4 == 0 && a.dim <= 256 &&
           a.vdim <= 256;
}

/* Key splits of lm_attn_step_group_kernel: as long as a CTA finds an SM of its own. */
static int group_splits(int kv_heads) {
    int splits = kSgSplits;
    while (splits > 1 && splits * kv_heads > kStepCtas) splits /= 2;
    return splits;
}

/* It is for short sequences and windows: its CTAs are at most 8 a KV head, of 8 warps, where lm_attn_step_kernel has up to 32 of
 * 16. Layer of an attention-only model, both kernels, at 220, 1000, 2000, 4000 keys: 8 KV heads of 128 with 8 query heads 17.1 /
 * 21.9, 21.5 / 24.8, 26.2 / 25.4, 37.0 / 28.3 us, with 32 19.5 / 26.2, 23.5 / 30.4, 28.1 / 34.1, 38.9 / 39.8; one of 128 16.1 /
 * 20.5, 19.4 / 22.7, 23.4 / 22.6, 32.9 / 22.7; 64 of 64 24.3 / 27.8, 47.4 / 34.3, 73.9 / 42.4, 129 / 57; 96 of 32, which
 * leave one CTA each, 29.7 / 22.1 at 220 already. */
int lm_attn_step_near(int heads, int kv_heads, int dim, int vdim) {
    const int splits = group_splits(kv_heads);
    return heads / kv_heads <= kSgHeads && dim <= kSgDim && vdim <= kSgDim && splits > 1 ? kSgMost * splits : 0;
}

int lm_attn_step(const LmAttn &a, cudaStream_t st) {
    const int group = a.heads / a.kv_heads;
    if (a.most <= lm_attn_step_near(a.heads, a.kv_heads, a.dim, a.vdim)) {
        const int splits = group_splits(a.kv_heads);
        return ok(launch_pdl_cluster(a.split ? lm_attn_step_group_kernel<true> : lm_attn_step_group_kernel<false>, splits, dim3(splits, a.kv_heads),
                                     dim3(kSgThreads), 0, st, a));
    }
    int lanes_h = 1;
    while (lanes_h < group) lanes_h *= 2;
    int splits = kStepCtas / a.kv_heads;
    splits = splits < 1 ? 1 : splits > kLmAttnSplits ? kLmAttnSplits : splits;
    if (a.split) return launch_attn_step<1, 1, 8, true>(a, splits, lanes_h, st);      /* sizes up to 128 */
    if (a.dim <= 128 && a.vdim <= 128) return launch_attn_step<1, 1, 8, false>(a, splits, lanes_h, st);
    return launch_attn_step<2, 2, 4, false>(a, splits, lanes_h, st);
}

} // namespace vb
