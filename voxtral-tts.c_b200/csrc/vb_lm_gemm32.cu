/*
 * vb_lm_gemm32.cu - the GEMMs of the language models' 32-bit mode: fp32 rows times BF16 weights, no product rounded,
 * sums as exact as the fp32 pipes make them.
 *
 * Up to kLmF32FewRows rows the weights are the traffic: a warp streams whole weight rows and keeps one fp32 sum per
 * row and lane. Above, the arithmetic is the bound, and the tensor cores do it: a row is the sum of three BF16 terms (24 bits),
 * a term's products with BF16 weights are exact, and the row-block GEMM adds them up in short stretches (kManySegment).
 * 390 x 11264 x 2048: 569 us in register tiles on the fp32 pipes, 32 TFLOP/s of their 74. Experts' rows, sorted by
 * matrix, still run in such tiles. All split K over CTAs when a matrix alone does not fill the chip; the partial sums are
 * added by the kernel that reads them.
 */
#include "vb_lm_kernels.cuh"

#include "vb_tc.cuh"

#include <algorithm>

namespace vb {

namespace {

typedef unsigned long long f2;   /* two packed floats */
VB_DEVINL f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
VB_DEVINL f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
VB_DEVINL f2 f2_two(float v) {
    f2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
VB_DEVINL float2 f2_get(f2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

VB_DEVINL float act_of(float v, int act) { return act == LM_ACT_RELU2 ? fmaxf(v, 0.0f) * fmaxf(v, 0.0f) : v; }

/* ---------------------------------------------------------------- rows sorted by matrix */
/* 64 x 128 results per CTA, 8 x 8 per thread, 16 columns of K per step, double-buffered. A warp's step is 32 packed
 * multiply-adds on 6 wavefronts of shared memory, so the fp32 pipes are the bound. Three CTAs fit an SM.
 * The sum over K is taken in two levels of 32 columns, so that its rounding error grows with the step length and the
 * number of steps, not with K. 390 x 2048 x 2048: 538 us with 64 x 64 tiles of single multiply-adds, element-wise
 * loads and no pipeline. */
constexpr int kFgM = 64, kFgN = 128, kFgK = 16, kFgThreads = 128;

__global__ void __launch_bounds__(kFgThreads, 3)
lm_gemm_f32_tile_kernel(float *y, int ld_out, size_t part_stride, const float *x, int ldx, const uint16_t *W, int ldw, int M, int N,
                        int steps, int act, const int4 *table, int group_rows) {
    __shared__ __align__(16) float xs[2][kFgK][kFgM + 4], ws[2][kFgK][kFgN + 4];
    pdl_launch_dependents();
    pdl_wait();
    const int n0 = blockIdx.x * kFgN;
    int m0 = blockIdx.y * kFgM;
    if (table) {                       /* two tiles of rows per block of 128 */
        const int4 g = __ldcg(table + (blockIdx.y >> 1));
        m0 = g.y + (int)(blockIdx.y & 1) * kFgM;
        M = g.y + g.z;
        if (g.x < 0 || m0 >= M) return;
        W += (size_t)g.x * group_rows * ldw;
    }
    /* steps of 32 columns, shared out over the splits */
    const int s0 = (int)((long long)steps * blockIdx.z / gridDim.z), s1 = (int)((long long)steps * (blockIdx.z + 1) / gridDim.z);
    const int tid = threadIdx.x, tm = (tid >> 4) * 8, tn = (tid & 15) * 4;
    /* what this thread brings in: 2 x 4 columns of x, 2 x 8 columns of W */
    const int xr = tid >> 2, xk = (tid & 3) * 4, wr = tid >> 1, wk = (tid & 1) * 8;
    const float *xp[2];
    const uint16_t *wp[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int m = m0 + xr + 32 * i, n = n0 + wr + 64 * i;
        xp[i] = m < M ? x + (size_t)m * ldx + xk : nullptr;
        wp[i] = n < N ? W + (size_t)n * ldw + wk : nullptr;
    }
    float4 xv[2];
    uint4 wv[2];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            xv[i] = xp[i] ? __ldcg((const float4 *)(xp[i] + k0)) : make_float4(0.f, 0.f, 0.f, 0.f);
            wv[i] = wp[i] ? __ldg((const uint4 *)(wp[i] + k0)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float e[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
            const uint32_t w[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                xs[b][xk + j][xr + 32 * i] = e[j];
                ws[b][wk + 2 * j][wr + 64 * i] = vb_bf16_lo(w[j]);
                ws[b][wk + 2 * j + 1][wr + 64 * i] = vb_bf16_hi(w[j]);
            }
        }
    };
    f2 sum[8][4] = {}, acc[8][4] = {};
    const int t0 = 2 * s0, t1 = 2 * s1;          /* steps of 16 columns */
    if (t0 < t1) {
        fetch(t0 * kFgK);
        put(t0 & 1);
    }
    __syncthreads();
    for (int t = t0; t < t1; t++) {
        const int b = t & 1;
        if (t + 1 < t1) fetch((t + 1) * kFgK);
#pragma unroll
        for (int k = 0; k < kFgK; k++) {
            const float4 a0 = *(const float4 *)&xs[b][k][tm], a1 = *(const float4 *)&xs[b][k][tm + 4];
            const ulonglong2 b0 = *(const ulonglong2 *)&ws[b][k][tn], b1 = *(const ulonglong2 *)&ws[b][k][tn + 64];
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const f2 a = f2_two(av[i]);
                acc[i][0] = f2_fma(a, b0.x, acc[i][0]);
                acc[i][1] = f2_fma(a, b0.y, acc[i][1]);
                acc[i][2] = f2_fma(a, b1.x, acc[i][2]);
                acc[i][3] = f2_fma(a, b1.y, acc[i][3]);
            }
        }
        if (t & 1) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    sum[i][j] = f2_add(sum[i][j], acc[i][j]);
                    acc[i][j] = 0ull;
                }
        }
        if (t + 1 < t1) put(b ^ 1);
        __syncthreads();
    }
    y += (size_t)blockIdx.z * part_stride;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int m = m0 + tm + i;
        if (m >= M) break;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int n = n0 + tn + 64 * h;
            const float2 u = f2_get(sum[i][2 * h]), v = f2_get(sum[i][2 * h + 1]);
            if (act == LM_ACT_SWIGLU) {
                float *o = y + (size_t)m * ld_out + n / 2;
                if (n + 1 < N) o[0] = u.x / (1.0f + expf(-u.x)) * u.y;
                if (n + 3 < N) o[1] = v.x / (1.0f + expf(-v.x)) * v.y;
            } else {
                float *o = y + (size_t)m * ld_out + n;
                const float e[4] = {act_of(u.x, act), act_of(u.y, act), act_of(v.x, act), act_of(v.y, act)};
                if (n + 3 < N && (ld_out & 3) == 0 && ((uintptr_t)y & 15) == 0) {
                    *(float4 *)o = make_float4(e[0], e[1], e[2], e[3]);
                } else {
                    for (int j = 0; j < 4; j++)
                        if (n + j < N) o[j] = e[j];
                }
            }
        }
    }
}

/* ---------------------------------------------------------------- few rows */
/* A warp owns R weight rows and up to eight rows of x: it streams the weights 8 columns (16 bytes) per lane and row,
 * two steps of 256 columns in flight, against x staged 512 columns at a time; every lane keeps its own sums, added up
 * over the warp at the end. Bound by the weight stream (and, at eight rows, by shared memory: two 16-byte reads of
 * x serve R rows of weights). 5 x 22528 x 2048: 314 us in 64-row tiles. */
constexpr int kSkWarps = 8, kSkRows = 8, kSkCols = 512;
template <int R>
__global__ void __launch_bounds__(32 * kSkWarps)
lm_gemm_f32_rows_kernel(float *y, int ld_out, size_t part_stride, const float *x, int ldx, const uint16_t *W, int ldw, int M, int N,
                        int cols, int act) {
    __shared__ __align__(16) float xs[kSkRows][kSkCols];
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = (blockIdx.x * kSkWarps + warp) * R, m0 = blockIdx.y * kSkRows, Mb = min(M - m0, kSkRows);
    /* steps of 512 columns, shared out over the splits */
    const int steps = (cols + kSkCols - 1) / kSkCols;
    const int s0 = (int)((long long)steps * blockIdx.z / gridDim.z), s1 = (int)((long long)steps * (blockIdx.z + 1) / gridDim.z);
    uint4 w[2][R];
    auto fetch = [&](int s) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int c = s * kSkCols + h * 256 + lane * 8;
#pragma unroll
            for (int r = 0; r < R; r++)
                w[h][r] = n0 + r < N && c < cols ? __ldg((const uint4 *)(W + (size_t)(n0 + r) * ldw + c)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    if (s0 < s1) fetch(s0);          /* the weights depend on nothing that runs before */
    pdl_wait();
    float acc[R][kSkRows] = {};
    for (int s = s0; s < s1; s++) {
        __syncthreads();
        for (int i = tid; i < kSkRows * (kSkCols / 4); i += 32 * kSkWarps) {
            const int m = i / (kSkCols / 4), c = (i % (kSkCols / 4)) * 4;
            const bool in = m < Mb && s * kSkCols + c < cols;
            *(float4 *)&xs[m][c] = in ? __ldcg((const float4 *)(x + (size_t)(m0 + m) * ldx + s * kSkCols + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        float wf[2][R][8];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t u[4] = {w[h][r].x, w[h][r].y, w[h][r].z, w[h][r].w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    wf[h][r][2 * j] = vb_bf16_lo(u[j]);
                    wf[h][r][2 * j + 1] = vb_bf16_hi(u[j]);
                }
            }
        if (s + 1 < s1) fetch(s + 1);
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int m = 0; m < kSkRows; m++) {
                if (m >= Mb) break;
                const float4 a = *(const float4 *)&xs[m][h * 256 + lane * 8], b = *(const float4 *)&xs[m][h * 256 + lane * 8 + 4];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float *q = wf[h][r];
                    float t = acc[r][m];
                    t = fmaf(a.x, q[0], t); t = fmaf(a.y, q[1], t); t = fmaf(a.z, q[2], t); t = fmaf(a.w, q[3], t);
                    t = fmaf(b.x, q[4], t); t = fmaf(b.y, q[5], t); t = fmaf(b.z, q[6], t); t = fmaf(b.w, q[7], t);
                    acc[r][m] = t;
                }
            }
    }
    y += (size_t)blockIdx.z * part_stride;
#pragma unroll
    for (int m = 0; m < kSkRows; m++) {
        if (m >= Mb) break;
        float t[R];
#pragma unroll
        for (int r = 0; r < R; r++) t[r] = vb_warp_sum(acc[r][m]);
        if (lane) continue;
        float *o = y + (size_t)(m0 + m) * ld_out;
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (act == LM_ACT_SWIGLU) {
                if ((r & 1) == 0 && n0 + r + 1 < N) o[(n0 + r) / 2] = t[r] / (1.0f + expf(-t[r])) * t[r + 1];
            } else if (n0 + r < N) {
                o[n0 + r] = act_of(t[r], act);
            }
        }
    }
}

/* ---------------------------------------------------------------- rows as terms */
/* fp32 rows -> three BF16 terms [3][rows_pad][ld], whose sum is the row to 24 bits. What BF16 cannot hold stays what the
 * fp32 pipes would have multiplied: infinities and NaN are their own first term, a finite value that rounds to
 * infinity is cut off. */
__global__ void __launch_bounds__(256) lm_split_rows_kernel(uint16_t *terms, int rows_pad, int ld, const float *x, int n4) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    const float4 v = __ldcg(reinterpret_cast<const float4 *>(x) + i);
    const float e[4] = {v.x, v.y, v.z, v.w};
    uint16_t t[3][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        vb_split3(e[j], t[0][j], t[1][j], t[2][j]);
        if ((t[0][j] & 0x7f80u) == 0x7f80u) {
            const uint32_t u = __float_as_uint(e[j]);
            if ((u & 0x7f800000u) == 0x7f800000u) {
                t[1][j] = t[2][j] = 0;
            } else {
                uint16_t last;
                t[0][j] = (uint16_t)(u >> 16);
                vb_split3(e[j] - __uint_as_float(u & 0xffff0000u), t[1][j], t[2][j], last);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
        *(reinterpret_cast<uint2 *>(terms + (size_t)k * rows_pad * ld) + i) =
            make_uint2(t[k][0] | ((uint32_t)t[k][1] << 16), t[k][2] | ((uint32_t)t[k][3] << 16));
}

/* Weight rows per warp: four halve the reads of x per weight; two where four would leave SMs without a CTA. */
int skinny_rows(int N) { return N >= 148 * kSkWarps * 4 ? 4 : 2; }

} // namespace

/* K splits: enough CTAs for two per SM, no split shorter than 512 columns. Many rows: what suits the row-block GEMM. */
int lm_gemm_f32_splits(int M, int N, int K, int n_sm) {
    if (M > kLmF32FewRows) return tc_row_splits(N, (K + kTcBlockK - 1) / kTcBlockK * kTcBlockK, M, n_sm, kTcTerms);
    const int rows = kSkWarps * skinny_rows(N), ctas = ((N + rows - 1) / rows) * ((M + kSkRows - 1) / kSkRows);
    return std::max(1, std::min({2 * n_sm / ctas, K / 512, 4}));
}

int lm_gemm_f32(float *y, int ld_out, const float *x, int ldx, const uint16_t *W, int ldw, int M, int N, int K, LmAct act,
                cudaStream_t st, int splits, const int4 *table, int group_rows) {
    /* whole 16-byte reads of both operands, up to the zero columns behind K */
    if (M < 1 || N < 1 || (ldx & 3) || (ldw & 31) || (K + 31) / 32 * 32 > std::min(ldx, ldw) || splits < 1 || (splits > 1 && act != LM_ACT_NONE)) return -1;
    const size_t stride = (size_t)M * ld_out;
    cudaError_t e;
    if (!table) {
        if (M > kLmF32FewRows) return -1;
        const int r = skinny_rows(N), cols = (K + 31) / 32 * 32;
        const dim3 g((N + kSkWarps * r - 1) / (kSkWarps * r), (M + kSkRows - 1) / kSkRows, splits);
        e = launch_pdl(r == 4 ? lm_gemm_f32_rows_kernel<4> : lm_gemm_f32_rows_kernel<2>, g, dim3(32 * kSkWarps), 0, st, y, ld_out, stride, x,
                       ldx, W, ldw, M, N, cols, (int)act);
    } else {
        const dim3 g((N + kFgN - 1) / kFgN, (M + kFgM - 1) / kFgM, splits);
        e = launch_pdl(lm_gemm_f32_tile_kernel, g, dim3(kFgThreads), 0, st, y, ld_out, stride, x, ldx, W, ldw, M, N, (K + 31) / 32, (int)act,
                       table, group_rows);
    }
    return e == cudaSuccess ? 0 : -1;
}

/* k-blocks that TMEM sums before registers add them up. A 24-run model of width 2048, seven prompts of 40 to 390 rows,
 * logits off 64 bits on average: 4.2e-6 on the fp32 pipes, 3.3e-6 with one or two k-blocks, 4.2e-6 with four, 6.7e-6
 * with eight; 390 rows take 13.9, 12.1, 11.5 and 11.3 ms (37.8 on the fp32 pipes). */
constexpr int kManySegment = 2;

int lm_gemm_f32_many(float *y, int ld_out, const float *x, int ldx, const TcWeight &w, uint16_t *terms, int M, bool swiglu, cudaStream_t st,
                     int splits, int *status) {
    TcActs a;
    if (ldx != w.K || tc_acts_blocks(&a, terms, lm_gemm_f32_rows_pad(M), w.K)) return -1;
    const int n4 = (int)((size_t)M * ldx / 4);
    if (launch_pdl(lm_split_rows_kernel, dim3((n4 + 255) / 256), dim3(256), 0, st, terms, a.rows_pad, ldx, x, n4) != cudaSuccess) return -1;
    TcGemm g;
    g.M = M;
    g.terms = kTcTerms;
    g.segment = kManySegment;
    g.status = status;
    g.out = y; g.ld_out = ld_out;
    g.epi = swiglu ? TC_EPI_SWIGLU : TC_EPI_PARTIAL;
    g.splits = splits;
    return tc_gemm(w, a, g, st);
}

} // namespace vb
