/*
 * vb_tc.cu - tcgen05 / TMEM / TMA skinny GEMM (sm_100a) for up to 64 activation rows: the frame's decoder step and
 * acoustic passes, short prompts, the language models' steps. (More rows: vb_tc_rows.cu.)
 *
 *   y[M,N] = x[M,K] . W[N,K]^T, BF16 W, fp32 x and y (tts_linear_nobias_bf16 with
 *   seq_len > 1, voxtral_tts_kernels.c:187-198, which the reference runs as
 *   weight expansion + SGEMM).
 *
 * Swap-AB: a 128-row weight tile is the UMMA A operand (K-major, 128-byte swizzle, brought in by 2-D TMA), the
 * activation rows are the narrow B operand (tiles of 16, 48 or 64 rows, their three terms side by side: UMMA N = 48,
 * 144, 192), the fp32 accumulator tile [128 x N] sits in TMEM. The kernel is HBM-bound (every weight byte is read once);
 * tensor work is a few percent.
 *
 * fp32 fidelity: the reference multiplies fp32 activations by exactly expanded BF16 weights. Each activation is split
 * into three BF16 terms, x = hi + lo + lo2 (8 + 8 + 8 mantissa bits), whose products with the weights are summed apart in
 * TMEM and added up by the epilogue; BF16 x BF16 products are exact in fp32, so only the summation differs from the
 * reference.
 *
 * Warp roles: warps 0-3 epilogue (TMEM lanes 32w..32w+31 -> registers -> global), warp 4 lane 0 TMA producer, warp 5
 * lane 0 MMA issuer. The GEMMs that end a sublayer (TcJoin) run in clusters of kTcJoinSplits CTAs, the others without;
 * no multicast. All waits are bounded; on expiry a status word is set, every role falls through, and the TMEM columns
 * are released before the CTA exits.
 */
#include "vb_tc.cuh"
#include "vb_common.cuh"
#include "vb_umma.cuh"

#include <cuda_bf16.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

namespace vb {

/* ---------------------------------------------------------------- host: tensor maps */
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;

int tc_init() {
    if (g_encode) return 0;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
        cudaGetLastError();
        return -1;
    }
    g_encode = (EncodeTiledFn)fn;
    return 0;
}

/* [rows, cols] BF16 row-major; box = 64 columns x box_rows rows, 128-byte swizzle. */
int tc_map(CUtensorMap *m, const void *base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    if (tc_init()) return -1;
    if (((uintptr_t)base & 15) || (cols * 2) % 16) return -1;
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)kTcBlockK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)base, gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -1;
}

int tc_map3(CUtensorMap *m, const void *base, uint64_t planes, uint64_t plane_bytes, uint64_t rows, uint64_t row_bytes, uint64_t cols, uint32_t box_rows) {
    if (tc_init()) return -1;
    if (((uintptr_t)base & 15) || row_bytes % 16 || plane_bytes % 16 || cols < kTcBlockK) return -1;
    cuuint64_t gdim[3] = {cols, rows, planes};
    cuuint64_t gstride[2] = {row_bytes, plane_bytes};
    cuuint32_t box[3] = {(cuuint32_t)kTcBlockK, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void *)base, gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -1;
}

int tc_weight(TcWeight *w, const uint16_t *d_W, int N, int K) {
    w->ok = false;
    w->W = d_W; w->N = N; w->K = K; w->tiled = false;
    if (N <= 0 || K <= 0 || (K % kTcBlockK) != 0) return -1;
    if (tc_map(&w->map, d_W, (uint64_t)N, (uint64_t)K, kTcTileN)) return -1;
    w->ok = true;
    return 0;
}

/* Weights re-laid out so that every [128 rows x 64 columns] tile the kernel fetches is one
 * contiguous 16 KB block (tile-major, then k-block), instead of 128 pieces of 128 bytes that
 * sit a whole weight row apart: the TMA request becomes a single DRAM-friendly burst. */
__global__ void vb_tc_tile_weights_kernel(uint4 *dst, const uint4 *src, int N, int K) {
    const int kblocks = K / kTcBlockK;
    const size_t n_vec = (size_t)((N + kTcTileN - 1) / kTcTileN) * kblocks * kTcTileN * (kTcBlockK / 8);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_vec) return;
    const int v = (int)(i % (kTcBlockK / 8));                 /* 16-byte vector inside the 128-byte row */
    const int r = (int)((i / (kTcBlockK / 8)) % kTcTileN);    /* row inside the tile */
    const size_t blk = i / ((kTcBlockK / 8) * kTcTileN);
    const int kb = (int)(blk % kblocks), t = (int)(blk / kblocks);
    const int row = t * kTcTileN + r;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (row < N) val = src[((size_t)row * K + (size_t)kb * kTcBlockK) / 8 + v];
    dst[i] = val;
}

size_t tc_tiled_bytes(int N, int K) {
    return (size_t)((N + kTcTileN - 1) / kTcTileN) * kTcTileN * K * 2;
}

int tc_weight_tiled(TcWeight *w, const uint16_t *d_W, int N, int K, uint16_t *d_tiled, cudaStream_t st) {
    w->ok = false;
    w->W = d_tiled; w->N = N; w->K = K; w->tiled = true;
    if (N <= 0 || K <= 0 || (K % kTcBlockK) != 0 || ((uintptr_t)d_W & 15) || ((uintptr_t)d_tiled & 15)) return -1;
    const size_t n_vec = tc_tiled_bytes(N, K) / 16;
    vb_tc_tile_weights_kernel<<<(unsigned)((n_vec + 255) / 256), 256, 0, st>>>((uint4 *)d_tiled, (const uint4 *)d_W, N, K);
    if (cudaGetLastError() != cudaSuccess) return -1;
    const uint64_t rows = (uint64_t)((N + kTcTileN - 1) / kTcTileN) * (K / kTcBlockK) * kTcTileN;
    if (tc_map(&w->map, d_tiled, rows, (uint64_t)kTcBlockK, kTcTileN)) return -1;
    w->ok = true;
    return 0;
}

int tc_rows_pad(int M) { return M <= 16 ? 16 : M <= 64 ? 64 : M <= 256 ? 256 : 0; }

/* The tile a frame's GEMMs use for M rows: 17 .. 48 rows (the acoustic rows of 3 .. 8 utterances)
 * take the 48-row tile, whose stages are 6 KB smaller than the 64-row tile's, so that a sixth stage
 * fits and the weight stream keeps 96 KB in flight per SM. */
int tc_rows_pad_frame(int M) { return (M > 16 && M <= 48) ? 48 : tc_rows_pad(M); }

/* Any number of rows: beyond 256 the buffer is padded to whole 128-row blocks (row-block kernel). */
int tc_rows_pad_any(int M) {
    if (M <= 256) return tc_rows_pad(M);
    return M <= kTcMaxRows ? (M + 127) / 128 * 128 : 0;
}

size_t tc_acts_bytes(int rows_pad, int K) { return (size_t)kTcTerms * rows_pad * K * 2; }

int tc_acts(TcActs *a, uint16_t *d_buf, int rows_pad, int K) {
    a->ok = false;
    a->buf = d_buf; a->rows_pad = rows_pad; a->K = K;
    const bool big = rows_pad > 256 && rows_pad <= kTcMaxRows && rows_pad % 128 == 0;
    if ((rows_pad != 16 && rows_pad != 48 && rows_pad != 64 && rows_pad != 256 && !big) || (K % kTcBlockK) != 0) return -1;
    /* (a TMA box holds at most 256 rows; the row-block kernel makes a map of its own for the rows it takes at once) */
    if (((uintptr_t)d_buf & 15) != 0) return -1;
    if (!big && tc_map(&a->map, d_buf, (uint64_t)kTcTerms * rows_pad, (uint64_t)K, (uint32_t)rows_pad)) return -1;
    a->ok = true;
    return 0;
}

int tc_acts_blocks(TcActs *a, uint16_t *d_buf, int rows, int K) {
    a->ok = false;
    a->buf = d_buf; a->rows_pad = rows; a->K = K;
    if (rows <= 0 || rows % 128 || (K % kTcBlockK) != 0 || ((uintptr_t)d_buf & 15)) return -1;
    a->ok = true;
    return 0;
}

int tc_pick_splits(int N, int K, int n_sm) {
    const int tiles = (N + kTcTileN - 1) / kTcTileN;
    int s = n_sm / tiles;
    if (s < 1) s = 1;
    if (s > kTcMaxSplits) s = kTcMaxSplits;
    if (s > K / kTcBlockK) s = K / kTcBlockK;
    return s;
}

/* ---------------------------------------------------------------- the kernel */
template <int NB, int ST, int ACCS>
struct TcCfg {
    static constexpr int kStageA = kTcTileN * kTcBlockK * 2;        /* 16 KB */
    static constexpr int kTermB = NB * kTcBlockK * 2;               /* one BF16 term of the activations */
    static constexpr int kStage = kStageA + kTcTerms * kTermB;
    static constexpr int kStages = ST;   /* one CTA per SM: rings small enough for two cost more than the overlap gave (212 frames: 611 ms and more for 594) */
    /* The three BF16 terms of the activations lie one after another in a stage, so that they
     * form ONE B operand of 3*NB rows: a single MMA per 16-wide K step writes the three partial
     * products to separate TMEM column groups (summed in the epilogue) instead of three narrow
     * MMAs - the narrow ones are issue-latency bound, not throughput bound. */
    static constexpr int kAccCols = kTcTerms * NB;
    static_assert(kAccCols <= 256, "wider than an MMA");
    /* The tensor core cuts its fp32 sums off at every step, so that their error grows with the chain: a CTA's share of K
     * goes into ACCS accumulators, one after another, whose sums the epilogue adds. One utterance, 40 frames: 2.714 ms a
     * frame with one accumulator (and 16 columns read for every row count), 2.709 with two, whose hidden states are 2.0e-5
     * for 2.4e-5 off 64 bits; segments of 512 to 1024 columns that the epilogue fetches under the main loop, with a commit
     * for each, 2.74 to 2.78. A velocity call: 8.7e-6 with one, 4.4e-6 with two, 2.2e-6 with four. */
    static constexpr int kTmemCols = ACCS * kAccCols <= 128 ? 128 : ACCS * kAccCols <= 256 ? 256 : 512;
    static_assert(ACCS * kAccCols <= kTmemCols, "accumulators over TMEM");
    static constexpr int kSmemBytes = kStages * kStage + 1024 /* alignment slack */ + 256 /* barriers */ + 4 * NB;
    static_assert(kSmemBytes <= 232448, "over the 227 KB a CTA may use");
};

constexpr int kTcThreads = 192;

/* Kernel-side scalars and pointers (everything but the two tensor maps). */
struct TcKernelArgs {
    int N, K, M, rows_pad, ld_out, splits, epi;
    int a_tiled;             /* weights in the tile-contiguous layout */
    float *out;
    const float *bias;
    const float *ssq;        /* optional [M][ssq_chunks] sums of squares: deferred RMSNorm row scale */
    int ssq_chunks;
    float eps;
    uint16_t *out_terms;     /* TC_EPI_SWIGLU_TERMS: BF16 terms of the result, [3][out_rows_pad][N/2] */
    int out_rows_pad;
    int *status;
    int tile0;               /* first output tile of this launch */
    int n_tiles_launch;      /* tiles this launch covers (host side: the grid) */
};

/* Tensor parallelism is a separate instantiation of every kernel that takes part in it, with
 * its arguments in a parameter of their own: the single-GPU kernels keep their parameter block
 * and code (carrying the extra 200 bytes and branches in every launch cost 0.3 ms per frame). */
struct TcTpArgs {
    TcPush push;             /* results also go to the peers' buffers */
    TcWait wait;             /* the activation terms may be exchanged data */
};
struct TcNoTpArgs {};
/* TC_JOIN: see TcJoin. The kernel that added up the partial results of these GEMMs before ("prepare") was a launch of its
 * own, 2 of 7 in a layer: a frame had 350 launches, 264 after it; 2.86 -> 2.81 ms. */
enum TcMode { TC_PLAIN = 0, TC_TP = 1, TC_JOIN = 2 };
template <int MODE> struct TcTpSel { using type = TcNoTpArgs; };
template <> struct TcTpSel<TC_TP> { using type = TcTpArgs; };
template <> struct TcTpSel<TC_JOIN> { using type = TcJoin; };

VB_DEVINL uint32_t tc_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
VB_DEVINL void tc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
/* Four floats at the same place of CTA `rank`'s shared memory. */
VB_DEVINL float4 tc_peer4(const float *p, uint32_t rank) {
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(vb_smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

/* Rows [c0, c0 + COLS) of this lane's output column, out of TMEM to their places in shared memory: the column groups NB and
 * 2 * NB on hold the lo and lo2 products, each accumulator a part of K. */
template <int NB, int COLS, int ACCS>
VB_DEVINL void tc_stage_rows(float *to, uint32_t t, int c0, int M, int n_it, int seg, const float *rscale) {
    float v[COLS];
    t += (uint32_t)c0;
#pragma unroll
    for (int a = 0; a < ACCS; a++, t += kTcTerms * NB) {
        if (a > 0 && n_it <= a * seg) break;
        uint32_t r[3][COLS];
        tmem_ld_x3<COLS>(t, t + NB, t + 2 * NB, r);
#pragma unroll
        for (int i = 0; i < COLS; i++) {
            const float u = (__uint_as_float(r[0][i]) + __uint_as_float(r[1][i])) + __uint_as_float(r[2][i]);
            v[i] = a == 0 ? u : v[i] + u;
        }
    }
#pragma unroll
    for (int i = 0; i < COLS; i++) {
        const int m = c0 + i;
        if (m < M) to[m * kTcTileN] = rscale ? v[i] * rscale[m] : v[i];
    }
}

/* the 32-bit mode keeps infinities */
template <int ACCS> VB_DEVINL void tc_split(float v, uint16_t &t0, uint16_t &t1, uint16_t &t2) {
    if constexpr (ACCS == kTcManySums) vb_split3_inf(v, t0, t1, t2);
    else vb_split3(v, t0, t1, t2);
}

template <int NB, int ST, int MODE, int ACCS>
__global__ void __launch_bounds__(kTcThreads, 1)
vb_tc_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                  const TcKernelArgs ka, const typename TcTpSel<MODE>::type tp) {
    using Cfg = TcCfg<NB, ST, ACCS>;
    constexpr bool TP = MODE == TC_TP;
    /* the tensor maps are fetched while the first reads of the parameter block are on their way */
    if (threadIdx.x == 128) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&mapA) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&mapB) : "memory");
    }
    const int N = ka.N, K = ka.K, M = ka.M, rows_pad = ka.rows_pad, ld_out = ka.ld_out, splits = ka.splits,
              epi = ka.epi;
    float *const out = ka.out;
    const float *const bias = ka.bias;
    int *const status = ka.status;
    /* Programmatic dependent launch: the next kernel in the stream may start its own
     * prologue now; it waits (griddepcontrol.wait) before touching what this one writes. */
    pdl_launch_dependents();
    extern __shared__ unsigned char tc_smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)tc_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *stages = base;
    uint64_t *full = (uint64_t *)(base + Cfg::kStages * Cfg::kStage);
    uint64_t *empty = full + Cfg::kStages;
    uint64_t *accum = empty + Cfg::kStages;
    uint32_t *tmem_slot = (uint32_t *)(accum + 1);
    int *abort_flag = (int *)(tmem_slot + 1);
    float *rscale = (float *)(abort_flag + 1);   /* [NB] per-row scales */

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int issued = 0;   /* producer thread only: pipeline iterations whose loads were requested */
    const int tile = ka.tile0 + blockIdx.x / splits, sp = blockIdx.x % splits;
    const int kblocks = K / kTcBlockK;
    const int kb0 = (int)((long long)kblocks * sp / splits), kb1 = (int)((long long)kblocks * (sp + 1) / splits);
    const int n_it = kb1 - kb0;
    const int seg = (n_it + ACCS - 1) / ACCS;      /* k-blocks of an accumulator */

    int first = 0;   /* producer thread only: stages of the first ring-full */
    if (warp == 4 && lane == 0) {
        /* The TMA producer sets the barriers up itself and requests the first ring-full of weight
         * tiles at once - they depend on nothing, neither on the predecessor kernel nor on the
         * TMEM allocation and the CTA-wide barrier below. */
        for (int i = 0; i < Cfg::kStages; i++) { vb_mbar_init(&full[i], 1); vb_mbar_init(&empty[i], 1); }
        vb_mbar_init(accum, 1);
        *abort_flag = 0;
        vb_mbar_init_fence();
        first = n_it < Cfg::kStages ? n_it : Cfg::kStages;
        for (int it = 0; it < first; it++) {
            unsigned char *sa = stages + (size_t)it * Cfg::kStage;
            vb_mbar_arrive_expect_tx(&full[it], (uint32_t)Cfg::kStage);
            if (ka.a_tiled) tma_load_2d(sa, &mapA, 0, (tile * kblocks + kb0 + it) * kTcTileN, &full[it]);
            else tma_load_2d(sa, &mapA, (kb0 + it) * kTcBlockK, tile * kTcTileN, &full[it]);
        }
        issued = first;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(vb_smem_u32(tmem_slot)),
                     "r"((uint32_t)Cfg::kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *(volatile uint32_t *)tmem_slot;

    float4 join_x = make_float4(0.f, 0.f, 0.f, 0.f), join_gain = join_x;   /* TC_JOIN: requested under the main loop */
    if (warp == 4 && lane == 0) {
        /* ---- TMA producer ----
         * The weights of the first ring-full are already on their way (above). Now the kernel
         * waits for its predecessor (griddepcontrol.wait) and only then fetches the activation
         * terms. */
        pdl_wait();
        if constexpr (TP) {
            if (tp.wait.n > 0) {
                /* the activation terms were written by other GPUs: wait for all of them, then make
                 * those writes visible to the TMA engine's proxy */
                if (!tp_wait(tp.wait)) *(volatile int *)abort_flag = 1;
                asm volatile("fence.proxy.async;" ::: "memory");
            }
        }
        for (int it = 0; it < first; it++) {
            unsigned char *sa = stages + (size_t)it * Cfg::kStage;
#pragma unroll
            for (int j = 0; j < kTcTerms; j++)
                tma_load_2d(sa + Cfg::kStageA + j * Cfg::kTermB, &mapB, (kb0 + it) * kTcBlockK, j * rows_pad, &full[it]);
        }
        for (int it = first; it < n_it; it++) {
            const int s = it % Cfg::kStages, use = it / Cfg::kStages;
            if (!vb_mbar_wait(&empty[s], (use & 1u) ^ 1u, abort_flag)) {
                atomicCAS(status, 0, 11);
                *(volatile int *)abort_flag = 1;
                break;
            }
            unsigned char *sa = stages + (size_t)s * Cfg::kStage;
            vb_mbar_arrive_expect_tx(&full[s], (uint32_t)Cfg::kStage);
            const int kx = (kb0 + it) * kTcBlockK;
            if (ka.a_tiled) tma_load_2d(sa, &mapA, 0, (tile * kblocks + kb0 + it) * kTcTileN, &full[s]);
            else tma_load_2d(sa, &mapA, kx, tile * kTcTileN, &full[s]);
#pragma unroll
            for (int j = 0; j < kTcTerms; j++)
                tma_load_2d(sa + Cfg::kStageA + j * Cfg::kTermB, &mapB, kx, j * rows_pad, &full[s]);
            issued = it + 1;
        }
    } else if (warp == 5 && lane == 0) {
        /* ---- MMA issuer ---- */
        const uint32_t idesc = umma_idesc_bf16(Cfg::kAccCols);
        bool ok = true;
        uint32_t d = tmem, more = 0;
        int end = seg;
        for (int it = 0; it < n_it && ok; it++) {
            const int s = it % Cfg::kStages, use = it / Cfg::kStages;
            if (!vb_mbar_wait(&full[s], use & 1u, abort_flag)) {
                atomicCAS(status, 0, 12);
                *(volatile int *)abort_flag = 1;
                ok = false;
                break;
            }
            tc_fence_after();
            const unsigned char *sa = stages + (size_t)s * Cfg::kStage;
            const uint64_t adesc = umma_desc_k_sw128(sa);
            /* 16 BF16 = 32 bytes further along K inside the swizzled row: +2 in 16-byte units */
            const uint64_t bdesc = umma_desc_k_sw128(sa + Cfg::kStageA);
            if (ACCS > 1 && it == end) { d += Cfg::kAccCols; end += seg; more = 0; }
#pragma unroll
            for (int k = 0; k < kTcBlockK / 16; k++, more = 1) umma_bf16(d, adesc + 2 * k, bdesc + 2 * k, idesc, more);
            umma_commit(&empty[s]);   /* stage reusable once these MMAs have read it */
        }
        umma_commit(accum);           /* accumulator complete (arrives at once when nothing was issued) */
    } else if (warp < 4) {
        /* ---- epilogue: TMEM -> registers -> global ---- */
        /* Everything below reads or writes what earlier kernels of the stream own. While the main
         * loop runs, fetch the per-row RMSNorm scale: the activations went in as x*gain and
         * 1/sqrt(mean(x^2)+eps) is applied to the accumulators (voxtral_tts_kernels.c:333-349). */
        pdl_wait();
        if (ka.ssq) {
#pragma unroll 4
            for (int m = warp; m < M; m += 4) {
                const float t = vb_warp_sum(lane < ka.ssq_chunks ? __ldcg(ka.ssq + m * ka.ssq_chunks + lane) : 0.0f);
                if (lane == 0) rscale[m] = 1.0f / sqrtf(t / (float)K + ka.eps);
            }
            vb_named_bar(1, 128);
        }
        if constexpr (MODE == TC_JOIN) {
            const int m = (int)tc_cluster_rank() + kTcJoinSplits * warp;      /* up to 16 rows: one a warp */
            if (m < M) join_x = vb_ldcg4(tp.x + (size_t)m * N + tile * kTcTileN + lane * 4);
            if (tp.gain) join_gain = __ldg(reinterpret_cast<const float4 *>(tp.gain + tile * kTcTileN + lane * 4));
        }
        bool ok = vb_mbar_wait(accum, 0u, abort_flag);
        if (!ok) {
            atomicCAS(status, 0, 13);
            *(volatile int *)abort_flag = 1;
        }
        tc_fence_after();
        /* The results leave through shared memory (the pipeline stages are free once every MMA has
         * completed) as 16-byte stores along the output columns. Storing straight from the TMEM
         * layout - a lane owns one output column, one 4-byte store per activation row - was
         * measured at ~90 ns per store and 1.5 us per launch even with a single row. */
        float *stg = (float *)stages;                              /* [M][128 output columns] */
        if (ok && n_it > 0) {
            const uint32_t t0 = tmem + ((uint32_t)(warp * 32) << 16);
            const float *const rs = ka.ssq ? rscale : nullptr;
            if (NB <= 16 && M <= 8) {          /* half as many columns to read: 0.04 us a launch */
                tc_stage_rows<NB, 8, ACCS>(stg + warp * 32 + lane, t0, 0, M, n_it, seg, rs);
            } else {
#pragma unroll 1
                for (int c0 = 0; c0 < NB && c0 < M; c0 += 16) tc_stage_rows<NB, 16, ACCS>(stg + warp * 32 + lane, t0, c0, M, n_it, seg, rs);
            }
            if constexpr (MODE != TC_JOIN) {
                vb_named_bar(1, 128);
                const int n = tile * kTcTileN + lane * 4;             /* this lane's four output columns */
                for (int m = warp; m < M; m += 4) {
                    const float4 v = *(const float4 *)(stg + m * kTcTileN + lane * 4);
                    if (epi == TC_EPI_SWIGLU || epi == TC_EPI_SWIGLU_TERMS) {
                        /* (gate, up, gate, up) -> two results at columns n / 2 and n / 2 + 1 */
                        const float res[2] = {(v.x / (1.0f + expf(-v.x))) * v.y, (v.z / (1.0f + expf(-v.z))) * v.w};
                        const int col = n >> 1;
                        const size_t ko = (size_t)(N >> 1);
                        if (n + 3 < N && ((ko | (size_t)ld_out) & 1) == 0) {
                            if (epi == TC_EPI_SWIGLU) {
                                *(float2 *)(out + (size_t)m * ld_out + col) = make_float2(res[0], res[1]);
                            } else {
                                uint16_t q[3][2];
                                tc_split<ACCS>(res[0], q[0][0], q[1][0], q[2][0]);
                                tc_split<ACCS>(res[1], q[0][1], q[1][1], q[2][1]);
                                const size_t o = (size_t)m * ko + col;
#pragma unroll
                                for (int j = 0; j < 3; j++) {
                                    const uint32_t pk = q[j][0] | ((uint32_t)q[j][1] << 16);
                                    *(uint32_t *)(ka.out_terms + (size_t)j * ka.out_rows_pad * ko + o) = pk;
                                    if constexpr (TP) {
                                        for (int d = 1; d < tp.push.n_dst; d++)
                                            *(uint32_t *)((char *)(ka.out_terms + (size_t)j * ka.out_rows_pad * ko + o) + tp.push.dst_off[d]) = pk;
                                    }
                                }
                            }
                        } else {
                            for (int i = 0; i < 2; i++) {
                                if (n + 2 * i + 1 >= N) break;
                                if (epi == TC_EPI_SWIGLU) {
                                    out[(size_t)m * ld_out + col + i] = res[i];
                                } else {
                                    uint16_t q0, q1, q2;
                                    tc_split<ACCS>(res[i], q0, q1, q2);
                                    const size_t o = (size_t)m * ko + col + i;
                                    ka.out_terms[o] = q0;
                                    ka.out_terms[(size_t)ka.out_rows_pad * ko + o] = q1;
                                    ka.out_terms[(size_t)2 * ka.out_rows_pad * ko + o] = q2;
                                    if constexpr (TP) {
                                        for (int d = 1; d < tp.push.n_dst; d++) {
                                            uint16_t *pt = (uint16_t *)((char *)ka.out_terms + tp.push.dst_off[d]);
                                            pt[o] = q0;
                                            pt[(size_t)ka.out_rows_pad * ko + o] = q1;
                                            pt[(size_t)2 * ka.out_rows_pad * ko + o] = q2;
                                        }
                                    }
                                }
                            }
                        }
                    } else {
                        const size_t o = ((size_t)(epi == TC_EPI_STORE ? 0 : sp) * M + m) * ld_out + n;
                        if (n + 3 < N && (ld_out & 3) == 0) {
                            float4 w4 = v;
                            if (epi == TC_EPI_STORE && bias) {
                                w4.x += __ldg(bias + n); w4.y += __ldg(bias + n + 1);
                                w4.z += __ldg(bias + n + 2); w4.w += __ldg(bias + n + 3);
                            }
                            *(float4 *)(out + o) = w4;
                            if constexpr (TP) {
                                if (epi != TC_EPI_STORE)
                                    for (int d = 1; d < tp.push.n_dst; d++)
                                        *(float4 *)((char *)(out + o) + tp.push.dst_off[d]) = w4;
                            }
                        } else {
                            const float e[4] = {v.x, v.y, v.z, v.w};
                            for (int i = 0; i < 4 && n + i < N; i++) {
                                const float w1 = e[i] + (epi == TC_EPI_STORE && bias ? __ldg(bias + n + i) : 0.0f);
                                out[o + i] = w1;
                                if constexpr (TP) {
                                    if (epi != TC_EPI_STORE)
                                        for (int d = 1; d < tp.push.n_dst; d++)
                                            *(float *)((char *)(out + o + i) + tp.push.dst_off[d]) = w1;
                                }
                            }
                        }
                    }
                }
            }
        }
        if constexpr (TP) {
            if (tp.push.n_dst > 0) {
                /* once every CTA of this launch has its results in all ranks' buffers, the last one
                 * publishes the visit to every rank */
                vb_named_bar(1, 128);
                if (threadIdx.x == 0) tp_publish(tp.push, gridDim.x);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if constexpr (MODE == TC_JOIN) {
        tc_cluster_sync();                    /* all partial results are staged */
        const float *stg = (const float *)stages;
        const int rank = (int)tc_cluster_rank(), n = tile * kTcTileN + lane * 4;
        const int m = rank + kTcJoinSplits * warp;
        if (warp < 4 && m < M) {
            float4 q[kTcJoinSplits];
#pragma unroll
            for (int u = 0; u < kTcJoinSplits; u++) q[u] = tc_peer4(stg + m * kTcTileN + lane * 4, (uint32_t)u);
            float4 v = q[0];
#pragma unroll
            for (int u = 1; u < kTcJoinSplits; u++) { v.x += q[u].x; v.y += q[u].y; v.z += q[u].z; v.w += q[u].w; }
            v.x = join_x.x + v.x; v.y = join_x.y + v.y; v.z = join_x.z + v.z; v.w = join_x.w + v.w;
            *reinterpret_cast<float4 *>(tp.x_out + (size_t)m * N + n) = v;
            if (tp.tap) *reinterpret_cast<float4 *>(tp.tap + (size_t)m * N + n) = v;
            if (tp.gain) {
                const float e[4] = {v.x * join_gain.x, v.y * join_gain.y, v.z * join_gain.z, v.w * join_gain.w};
                uint16_t t[3][4];
#pragma unroll
                for (int i = 0; i < 4; i++) vb_split3(e[i], t[0][i], t[1][i], t[2][i]);
                uint16_t *o = tp.terms + (size_t)m * N + n;
#pragma unroll
                for (int j = 0; j < 3; j++)
                    *reinterpret_cast<uint2 *>(o + (size_t)j * tp.rows_pad * N) =
                        make_uint2(t[j][0] | ((uint32_t)t[j][1] << 16), t[j][2] | ((uint32_t)t[j][3] << 16));
                const float ss = vb_warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
                if (lane == 0) tp.ssq[m * (N / kTcTileN) + tile] = ss;
            }
        }
        __syncwarp();
        tc_cluster_sync();                    /* nobody reads this CTA's shared memory any more */
    }
    /* abort path: let copies already in flight land before the shared memory goes away */
    if (warp == 4 && lane == 0 && *(volatile int *)abort_flag) {
        /* the last load issued into stage s was iteration `it` with it % kStages == s: wait for
         * exactly that phase of its barrier */
        const int first_it = issued > Cfg::kStages ? issued - Cfg::kStages : 0;
        for (int it = first_it; it < issued; it++) {
            const long long t0 = clock64();
            while (!vb_mbar_try_wait(&full[it % Cfg::kStages], (uint32_t)(it / Cfg::kStages) & 1u)) {
                if (clock64() - t0 > VB_WAIT_CYCLES / 8) break;
            }
        }
    }
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)Cfg::kTmemCols)
                     : "memory");
    }
}

template <int NB, int ST, int MODE, int ACCS>
static int launch_tc_tp(const TcWeight &w, const TcActs &a, const TcKernelArgs &ka, const typename TcTpSel<MODE>::type &arg,
                        cudaStream_t st) {
    using Cfg = TcCfg<NB, ST, ACCS>;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(vb_tc_gemm_kernel<NB, ST, MODE, ACCS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 Cfg::kSmemBytes) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        attr = true;
    }
    const int tiles = ka.n_tiles_launch;
    return launch_pdl_cluster(vb_tc_gemm_kernel<NB, ST, MODE, ACCS>, MODE == TC_JOIN ? kTcJoinSplits : 0, dim3(tiles * ka.splits), dim3(kTcThreads),
                              (size_t)Cfg::kSmemBytes, st, w.map, a.map, ka, arg) == cudaSuccess
               ? 0
               : -1;
}

template <int NB, int ST, int ACCS>
static int launch_tc(const TcWeight &w, const TcActs &a, const TcKernelArgs &ka, const TcTpArgs &tpa, cudaStream_t st) {
    if (tpa.push.n_dst > 0 || tpa.wait.n > 0) return launch_tc_tp<NB, ST, TC_TP, ACCS>(w, a, ka, tpa, st);
    return launch_tc_tp<NB, ST, TC_PLAIN, ACCS>(w, a, ka, TcNoTpArgs(), st);
}

static int tc_gemm_join(const TcWeight &w, const TcActs &a, const TcGemm &g, cudaStream_t st) {
    const TcJoin &j = g.join;
    if (a.rows_pad != 16 || w.N % kTcTileN || w.K / kTcBlockK < kTcJoinSplits || !j.x_out || (j.gain && (!j.terms || !j.ssq || j.rows_pad < g.M))) return -1;
    if (g.n_tiles || g.push.n_dst || g.wait.n || g.ssq || g.bias) return -1;
    TcKernelArgs ka = {};
    ka.a_tiled = w.tiled ? 1 : 0;
    ka.N = w.N; ka.K = w.K; ka.M = g.M; ka.rows_pad = a.rows_pad; ka.splits = kTcJoinSplits; ka.status = g.status;
    ka.n_tiles_launch = w.N / kTcTileN;
    if (g.sums != 2 && g.sums != 4) return -1;
    return g.sums == 4 ? launch_tc_tp<16, 6, TC_JOIN, 4>(w, a, ka, j, st) : launch_tc_tp<16, 6, TC_JOIN, 2>(w, a, ka, j, st);
}

int tc_gemm(const TcWeight &w, const TcActs &a, const TcGemm &g, cudaStream_t st) {
    if (!w.ok || !a.ok || w.K != a.K || g.M < 1 || g.M > a.rows_pad) return -1;
    if (g.join.x) return tc_gemm_join(w, a, g, st);
    if (g.splits < 1 || g.splits > kTcMaxSplits || g.splits > w.K / kTcBlockK) return -1;
    if (g.epi != TC_EPI_PARTIAL && g.splits != 1) return -1;
    if (g.sums != 2 && (a.rows_pad == 16 ? g.push.n_dst || g.wait.n || (g.sums != 4 && g.sums != kTcManySums) : a.rows_pad < 256)) return -1;
    if ((g.epi == TC_EPI_SWIGLU || g.epi == TC_EPI_SWIGLU_TERMS) && (w.N & 1)) return -1;
    if (g.epi == TC_EPI_SWIGLU_TERMS && (!g.out_terms || g.out_rows_pad < g.M)) return -1;
    if ((g.epi == TC_EPI_TERMS || g.epi == TC_EPI_RELU2_TERMS) && a.rows_pad < 256) return -1;
    if (a.rows_pad >= 256) {
        /* sliced or exchanged launches (tensor parallelism) do not occur beyond 64 rows */
        return g.n_tiles || g.push.n_dst || g.wait.n ? -1 : tc_gemm_rows(w, a, g, st);
    }
    TcKernelArgs ka;
    ka.a_tiled = w.tiled ? 1 : 0;
    ka.N = w.N; ka.K = w.K; ka.M = g.M; ka.rows_pad = a.rows_pad; ka.ld_out = g.ld_out; ka.splits = g.splits;
    ka.epi = g.epi; ka.out = g.out; ka.bias = g.bias; ka.ssq = g.ssq; ka.ssq_chunks = g.ssq_chunks; ka.eps = g.eps;
    ka.out_terms = g.out_terms; ka.out_rows_pad = g.out_rows_pad; ka.status = g.status;
    {
        const int tiles = (w.N + kTcTileN - 1) / kTcTileN;
        ka.tile0 = g.n_tiles > 0 ? g.tile0 : 0;
        ka.n_tiles_launch = g.n_tiles > 0 ? g.n_tiles : tiles;
        if (ka.tile0 < 0 || ka.tile0 + ka.n_tiles_launch > tiles) return -1;
        if (g.push.n_dst > kTpMaxRanks || (g.push.n_dst > 0 && (!g.push.ticket || !g.push.epoch))) return -1;
    }
    TcTpArgs tpa;
    tpa.push = g.push;
    tpa.wait = g.wait;
    tpa.wait.status = g.status;
    switch (a.rows_pad) {
    case 16:
        if (g.sums == kTcManySums) return launch_tc_tp<16, 6, TC_PLAIN, kTcManySums>(w, a, ka, TcNoTpArgs(), st);
        return g.sums == 4 ? launch_tc_tp<16, 6, TC_PLAIN, 4>(w, a, ka, TcNoTpArgs(), st) : launch_tc<16, 6, 2>(w, a, ka, tpa, st);
    case 48: return launch_tc<48, 6, 1>(w, a, ka, tpa, st);   /* 8 utterances' acoustic rows: 34 KB stages, six of them */
    case 64: return launch_tc<64, 5, 1>(w, a, ka, tpa, st);
    default: return -1;
    }
}

/* ---------------------------------------------------------------- prepare */
/* Activation rows -> three BF16 terms. grid = (K / 1024, M), 256 threads x 4 columns.
 *   v = x                                   (plain)
 *   v = residual + sum_p partials[p]        (split-K reduction in fixed order + residual add)
 * optional: x_out = v (the new residual stream); with a gain, the terms hold v*gain and the
 * CTA's sum of v^2 goes to ssq[m][chunk] - the consumer GEMM applies 1/sqrt(mean+eps), so no
 * CTA has to see a whole row and the kernel is a few microseconds instead of a serial pass. */
template <bool TP>
__global__ void vb_tc_prepare_kernel(uint16_t *buf, int rows_pad, int K, const float *x, int ldx,
                                     const float *partials, int n_part, size_t part_stride,
                                     const float *residual, float *x_out, const float *gain, float *ssq,
                                     float *tap, const typename TcWaitSel<TP>::type wait) {
    __shared__ float red[8];
    pdl_launch_dependents();
    pdl_wait();
    if constexpr (TP) {   /* the partials come from every rank */
        if (threadIdx.x == 0) tp_wait(wait);
        __syncthreads();
    }
    const int m = blockIdx.y;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    float ss = 0.0f;
    if (c < K) {
        float4 v;
        if (partials) {
            /* all partial loads in flight together, then the fixed-order sum */
            float4 t[kTcMaxSplits];
#pragma unroll
            for (int p = 0; p < kTcMaxSplits; p++)
                t[p] = p < n_part ? __ldcg(reinterpret_cast<const float4 *>(partials + (size_t)p * part_stride + (size_t)m * K + c))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
            v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int p = 0; p < kTcMaxSplits; p++) {
                if (p < n_part) { v.x += t[p].x; v.y += t[p].y; v.z += t[p].z; v.w += t[p].w; }
            }
            if (residual) {
                const float4 r = *reinterpret_cast<const float4 *>(residual + (size_t)m * ldx + c);
                v.x = r.x + v.x; v.y = r.y + v.y; v.z = r.z + v.z; v.w = r.w + v.w;
            }
        } else {
            v = *reinterpret_cast<const float4 *>(x + (size_t)m * ldx + c);
        }
        if (x_out) *reinterpret_cast<float4 *>(x_out + (size_t)m * ldx + c) = v;
        if (tap) *reinterpret_cast<float4 *>(tap + (size_t)m * ldx + c) = v;     /* residual-stream tap for parity checks */
        ss = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        if (gain) {
            const float4 g = __ldg(reinterpret_cast<const float4 *>(gain + c));
            v.x *= g.x; v.y *= g.y; v.z *= g.z; v.w *= g.w;
        }
        const float e[4] = {v.x, v.y, v.z, v.w};
        uint16_t t0[4], t1[4], t2[4];
#pragma unroll
        for (int i = 0; i < 4; i++) vb_split3(e[i], t0[i], t1[i], t2[i]);
        const size_t o = (size_t)m * K + c, term = (size_t)rows_pad * K;
        *reinterpret_cast<uint2 *>(buf + o) = make_uint2(t0[0] | ((uint32_t)t0[1] << 16), t0[2] | ((uint32_t)t0[3] << 16));
        *reinterpret_cast<uint2 *>(buf + term + o) = make_uint2(t1[0] | ((uint32_t)t1[1] << 16), t1[2] | ((uint32_t)t1[3] << 16));
        *reinterpret_cast<uint2 *>(buf + 2 * term + o) = make_uint2(t2[0] | ((uint32_t)t2[1] << 16), t2[2] | ((uint32_t)t2[3] << 16));
    }
    if (ssq) {
        ss = vb_warp_sum(ss);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.0f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
            ssq[m * gridDim.x + blockIdx.x] = t;
        }
    }
}

int tc_prepare_chunks(int K) { return (K + 1023) / 1024; }

void tc_prepare(const TcActs &acts, const float *x, int ldx, int M, const float *partials, int n_part,
                size_t part_stride, const float *residual, float *x_out, const float *gain, float *ssq,
                cudaStream_t st, const TcWait &wait, float *tap, bool plain) {
    if (M <= 0) return;
    if (plain)
        vb_tc_prepare_kernel<false><<<dim3(tc_prepare_chunks(acts.K), M), 256, 0, st>>>(acts.buf, acts.rows_pad, acts.K, x, ldx, partials, n_part,
                                                                                         part_stride, residual, x_out, gain, ssq, tap, TcNoWait());
    else if (wait.n > 0)
        launch_pdl(vb_tc_prepare_kernel<true>, dim3(tc_prepare_chunks(acts.K), M), dim3(256), 0, st, acts.buf,
                   acts.rows_pad, acts.K, x, ldx, partials, n_part, part_stride, residual, x_out, gain, ssq, tap, wait);
    else
        launch_pdl(vb_tc_prepare_kernel<false>, dim3(tc_prepare_chunks(acts.K), M), dim3(256), 0, st, acts.buf,
                   acts.rows_pad, acts.K, x, ldx, partials, n_part, part_stride, residual, x_out, gain, ssq, tap,
                   TcNoWait());
}

/* y[i] = sum over the split-K partials in fixed order (+ bias[i % N]). */
__global__ void vb_tc_reduce_kernel(float *y, const float *partials, int n_part, size_t stride, size_t count,
                                    const float *bias, int N) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float v = 0.0f;
    for (int p = 0; p < n_part; p++) v += partials[(size_t)p * stride + i];
    if (bias) v += bias[i % N];
    y[i] = v;
}

void tc_reduce(float *y, const float *partials, int n_part, size_t stride, size_t count, const float *bias, int N,
               cudaStream_t st) {
    if (count == 0) return;
    launch_pdl(vb_tc_reduce_kernel, dim3((unsigned)((count + 255) / 256)), dim3(256), 0, st, y, partials, n_part, stride, count,
               bias, N);
}

/* ---------------------------------------------------------------- stand-alone probe */
__global__ void vb_tc_fill_kernel(uint16_t *p, size_t n, uint32_t seed) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    /* small BF16 values of both signs: 0x3c00 | 6 hashed mantissa bits, hashed sign */
    uint32_t h = (uint32_t)i * 2654435761u + seed;
    h ^= h >> 15;
    p[i] = (uint16_t)(0x3c00u | (h & 0x3fu) | ((h & 0x40u) << 9));
}

/* One weight matrix [N, K] of generated values, M activation rows, `reps` launches of the GEMM
 * between two events on the default stream. Needs no model: a measurement and profiling aid
 * with a small memory footprint. epi: TC_EPI_PARTIAL (split-K as the frame uses it) or
 * TC_EPI_SWIGLU_TERMS; tiled bit 0: tile-contiguous weight copy as the frame uses it; bit 1: one
 * copy only, so that a matrix smaller than L2 stays resident (how fast is a launch whose weights
 * need no HBM?). */
int tc_probe(int M, int N, int K, int epi, int tiled, int reps, int n_sm, float *ms_out, int *splits_out) {
    if (tc_init() || M < 1 || reps < 1 || (K % kTcBlockK) != 0) return -1;
    const int rp = tc_rows_pad_frame(M);
    if (!rp) return -1;
    /* enough copies of the matrix that successive launches cannot find their weights in L2 */
    const int copies = (tiled & 2) ? 1 : (int)((size_t)512 * 1024 * 1024 / ((size_t)N * K * 2)) + 1;
    tiled &= 1;
    std::vector<uint16_t *> Wc(copies, nullptr);
    std::vector<TcWeight> wc(copies);
    uint16_t *W = nullptr, *terms = nullptr, *out_terms = nullptr;
    float *out = nullptr;
    int *status = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int rc = -1;
    const size_t wn = (size_t)N * K;
    const int splits = epi == TC_EPI_PARTIAL ? tc_pick_splits(N, K, n_sm) : 1;
    do {
        if (cudaMalloc(&W, wn * 2) != cudaSuccess || cudaMalloc(&terms, tc_acts_bytes(rp, K)) != cudaSuccess ||
            cudaMalloc(&out, sizeof(float) * (size_t)kTcMaxSplits * M * N) != cudaSuccess ||
            cudaMalloc(&out_terms, tc_acts_bytes(rp, N / 2 + 64)) != cudaSuccess ||
            cudaMalloc(&status, sizeof(int)) != cudaSuccess)
            break;
        cudaMemset(status, 0, sizeof(int));
        vb_tc_fill_kernel<<<(unsigned)((wn + 255) / 256), 256>>>(W, wn, 1u);
        const size_t tn = tc_acts_bytes(rp, K) / 2;
        vb_tc_fill_kernel<<<(unsigned)((tn + 255) / 256), 256>>>(terms, tn, 2u);
        bool wok = true;
        for (int c = 0; c < copies && wok; c++) {
            const size_t bytes = tiled ? tc_tiled_bytes(N, K) : wn * 2;
            wok = cudaMalloc(&Wc[c], bytes) == cudaSuccess;
            if (wok && tiled) wok = tc_weight_tiled(&wc[c], W, N, K, Wc[c], 0) == 0;
            else if (wok) wok = cudaMemcpy(Wc[c], W, bytes, cudaMemcpyDeviceToDevice) == cudaSuccess && tc_weight(&wc[c], Wc[c], N, K) == 0;
        }
        if (!wok) break;
        TcActs a;
        if (tc_acts(&a, terms, rp, K)) break;
        TcGemm g;
        g.M = M; g.splits = splits; g.epi = epi; g.out = out; g.ld_out = epi == TC_EPI_PARTIAL ? N : N / 2;
        g.out_terms = out_terms; g.out_rows_pad = rp; g.status = status;
        if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) break;
        bool ok = true;
        for (int i = 0; i < 3 && ok; i++) ok = tc_gemm(wc[i % copies], a, g, 0) == 0;
        cudaEventRecord(e0, 0);
        for (int i = 0; i < reps && ok; i++) ok = tc_gemm(wc[(3 + i) % copies], a, g, 0) == 0;
        cudaEventRecord(e1, 0);
        if (!ok || cudaDeviceSynchronize() != cudaSuccess) break;
        int st = 0;
        cudaMemcpy(&st, status, sizeof(int), cudaMemcpyDeviceToHost);
        if (st) break;
        if (ms_out) cudaEventElapsedTime(ms_out, e0, e1);
        if (splits_out) *splits_out = splits;
        rc = 0;
    } while (0);
    cudaGetLastError();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    for (uint16_t *p : Wc) cudaFree(p);
    cudaFree(W); cudaFree(terms); cudaFree(out); cudaFree(out_terms); cudaFree(status);
    return rc;
}

} // namespace vb
