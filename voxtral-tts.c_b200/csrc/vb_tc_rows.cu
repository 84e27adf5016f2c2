/*
 * vb_tc_rows.cu - the tensor-core GEMM for many activation rows (65 and more): prompts, the codec, mixtures of experts.
 *
 *   y[M,N] = x[M,K] . W[N,K]^T, BF16 W, x as hi + lo BF16 terms (16 mantissa bits: 4e-6 relative) or, for the language
 *   models' 32-bit mode, as three (24 bits), fp32 sums
 *
 * A pair of CTAs (one cluster, tcgen05 cta_group::2) owns 256 weight rows x R activation rows: each CTA brings in its
 * own 128 weight rows and half of the activation rows, and every MMA (256 x R x 16) reads both halves. What bounds a
 * CTA is shared memory, not the tensor pipe: with one CTA per tile (256 weight rows x 128 activation rows, 128 x 128
 * MMAs) a 64-column k-block costs 128 KB of operand reads and 64 KB of TMA writes at 128 bytes per clock, 1536 clocks
 * for 1024 clocks of arithmetic - measured 0.78 us. The pair moves 64 + 48 KB per CTA for the same arithmetic, below
 * the tensor pipe's 1024 clocks.
 *
 * Persistent: every pair walks its share of the tiles, the accumulators (R <= 256 columns) sit twice in TMEM, so that
 * the epilogue of a tile runs under the main loop of the next. R is chosen per launch (pick_rows): a smaller one that
 * fills the last wave beats 256 where the tile count falls badly on the pairs.
 *
 * The tensor core's fp32 sums are cut off, not rounded, at every step, and the error grows with the chain: 1203 speech
 * rows with K in one piece were 7.1e-5 off 64 bits, in 3 to 6 splits 4.6e-5, at the price of as many partial results.
 * So TMEM sums up to 2048 columns at a time (alternating accumulators) and the epilogue warps add these up in
 * registers, 64 values a thread, under the main loop. A 4001-token prompt: 60.6 ms and 7.3e-5 in one piece, 61.9 ms and
 * 4.9e-5 so, 63.3 ms and 3.3e-5 with 1024 columns (and 66 to 69 ms where eight warps held 128 values and spilled). The
 * codec, whose K splits are fewer than before this kernel, takes 1024 (TcGemm::segment).
 *
 * Three terms: R <= 128, and the two low terms have a sum of their own, so that the high one is cut off a third as often; the
 * stages keep 40 KB (a k-block costs 512 + 3 R clocks of shared memory, 6 R of the tensor pipe). The epilogue adds a
 * segment up within the time of its main loop down to a single k-block (kF32Segment in vb_lm.cu has the figures).
 *
 * Warps: 0-15 epilogue (TMEM -> registers -> shared memory -> whole 512-byte row segments), 16 TMA producer, 17 MMA issuer (of the even
 * CTA, for both). Full barriers and the accumulator hand-back live in the even CTA; commits arrive in both. No
 * multicast loads. All waits are bounded.
 */
#include "vb_tc.cuh"
#include "vb_common.cuh"
#include "vb_umma.cuh"

#include <algorithm>

namespace vb {

namespace {

constexpr int kPrStages = 4, kPrChunk = 64, kPrAcc = 256;      /* kPrAcc: TMEM columns of an accumulator */
constexpr int kPrStageW = kTcTileN * kTcBlockK * 2;
constexpr int kPrStaging = kPrChunk * kTcTileN * 4;
constexpr int kPrEpiWarps = 16, kPrEpi = 32 * kPrEpiWarps, kPrThreads = kPrEpi + 64;
constexpr uint32_t kPrTmemCols = 512;
template <int TERMS> struct PrCfg {
    static constexpr int max_rows = TERMS == 3 ? 128 : 256;
    static constexpr int stage_x = max_rows / 2 * kTcBlockK * 2, stage = kPrStageW + TERMS * stage_x;
    static constexpr int smem = kPrStages * stage + kPrStaging + max_rows * 4 + 256 + 1024;
    static_assert(smem <= 232448, "over the 227 KB a CTA may use");
};

struct RowsArgs {
    float *out;
    uint16_t *out_terms;
    const float *bias, *ssq;
    const int4 *table;           /* grouped: {matrix or -1, first row, rows, unused} per row block */
    int *status;
    float eps;
    int N, K, M, R, rows_pad, ld_out, splits, epi, ssq_chunks, a_tiled, out_rows_pad, act_n0, out_terms_ld, out_col0;
    int row_blocks, pairs, group_tiles, segment;
};

VB_DEVINL uint32_t pr_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
VB_DEVINL void pr_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
/* the even CTA's copy of a barrier, as a cluster address */
VB_DEVINL uint32_t pr_leader(const uint64_t *bar) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(vb_smem_u32(bar)));
    return r;
}
VB_DEVINL void pr_arrive(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
VB_DEVINL void pr_load(void *dst, const CUtensorMap *map, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            vb_smem_u32(dst)),
        "l"(map), "r"(cluster_bar), "r"(x), "r"(y)
        : "memory");
}
VB_DEVINL void pr_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
/* arrives on this barrier of both CTAs when the MMAs issued so far are done */
VB_DEVINL void pr_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     vb_smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}

/* One tile of a pair: its place, and the MMA width its rows need. */
struct PrTile {
    int sp, t0, w0, m0, Mb, n_mma, kb0, n_it, seg;
    bool used;
};
template <bool GROUPED>
VB_DEVINL PrTile pr_tile(const RowsArgs &a, int i, int kblocks) {
    PrTile t;
    t.sp = i % a.splits;
    const int rb = (i / a.splits) % a.row_blocks;
    t.t0 = i / (a.splits * a.row_blocks) * 2;
    t.m0 = rb * a.R;
    t.Mb = min(a.M - t.m0, a.R);
    t.w0 = t.t0;
    t.used = true;
    if constexpr (GROUPED) {
        const int4 g = __ldcg(a.table + rb);
        t.used = g.x >= 0;
        t.m0 = g.y;
        t.Mb = g.z;
        t.w0 = g.x * a.group_tiles + t.t0;
    }
    t.n_mma = (t.Mb + 31) & ~31;
    t.kb0 = (int)((long long)kblocks * t.sp / a.splits);
    t.n_it = (int)((long long)kblocks * (t.sp + 1) / a.splits) - t.kb0;
    const int segments = (t.n_it + a.segment - 1) / a.segment;
    t.seg = (t.n_it + segments - 1) / segments;
    return t;
}

VB_DEVINL uint32_t pr_pack(uint16_t a, uint16_t b) { return a | ((uint32_t)b << 16); }

/* three terms keep infinities */
template <int TERMS> VB_DEVINL void pr_split(float v, uint16_t &t0, uint16_t &t1, uint16_t &t2) {
    if constexpr (TERMS == 3) vb_split3_inf(v, t0, t1, t2);
    else vb_split3(v, t0, t1, t2);
}

/* Rows [c0, c0 + 64) of a tile's results, staged as [row][128 columns], to where they belong; `t` is this CTA's weight tile. */
template <int TERMS>
VB_DEVINL void pr_store(const RowsArgs &a, const float *stg, const PrTile &tl, int t, int c0, int warp, int lane) {
    const int n = t * kTcTileN + lane * 4, end = min(tl.Mb, c0 + kPrChunk);
    if (a.epi == TC_EPI_SWIGLU || a.epi == TC_EPI_SWIGLU_TERMS) {
        if (n + 1 >= a.N) return;
        const int col = t * (kTcTileN / 2) + lane * 2;
        const size_t ko = (size_t)(a.N >> 1);
        const bool both = n + 3 < a.N;
        for (int mb = c0 + warp; mb < end; mb += kPrEpiWarps) {
            const float4 v = *(const float4 *)(stg + (mb - c0) * kTcTileN + lane * 4);
            const float r0 = (v.x / (1.0f + expf(-v.x))) * v.y, r1 = (v.z / (1.0f + expf(-v.z))) * v.w;
            const int m = tl.m0 + mb;
            if (a.epi == TC_EPI_SWIGLU) {
                float *o = a.out + (size_t)m * a.ld_out + col;
                o[0] = r0;
                if (both) o[1] = r1;
            } else {
                uint16_t p[3], q[3];
                pr_split<TERMS>(r0, p[0], p[1], p[2]);
                pr_split<TERMS>(r1, q[0], q[1], q[2]);
#pragma unroll
                for (int j = 0; j < TERMS; j++) {
                    uint16_t *o = a.out_terms + ((size_t)j * a.out_rows_pad + m) * ko + col;
                    if (both && (ko & 1) == 0) {
                        *(uint32_t *)o = pr_pack(p[j], q[j]);
                    } else {
                        o[0] = p[j];
                        if (both) o[1] = q[j];
                    }
                }
            }
        }
        return;
    }
    if (n >= a.N) return;
    if ((a.epi == TC_EPI_TERMS || a.epi == TC_EPI_RELU2_TERMS) && n >= a.act_n0) {
        const int col = a.out_col0 + n - a.act_n0;
        for (int mb = c0 + warp; mb < end; mb += kPrEpiWarps) {
            const float4 v = *(const float4 *)(stg + (mb - c0) * kTcTileN + lane * 4);
            float e[4] = {v.x, v.y, v.z, v.w};
            uint16_t q[3][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (a.epi == TC_EPI_RELU2_TERMS) { e[i] = fmaxf(e[i], 0.0f); e[i] *= e[i]; }
                pr_split<TERMS>(e[i], q[0][i], q[1][i], q[2][i]);
            }
#pragma unroll
            for (int j = 0; j < TERMS; j++) {
                uint16_t *o = a.out_terms + ((size_t)j * a.out_rows_pad + tl.m0 + mb) * a.out_terms_ld + col;
                if (n + 3 < a.N) {
                    *(uint2 *)o = make_uint2(pr_pack(q[j][0], q[j][1]), pr_pack(q[j][2], q[j][3]));
                } else {
                    for (int i = 0; i < 4 && n + i < a.N; i++) o[i] = q[j][i];
                }
            }
        }
        return;
    }
    const bool bias = a.epi == TC_EPI_STORE && a.bias, whole = n + 3 < a.N && (a.ld_out & 3) == 0;
    float b[4] = {};
    if (bias)
        for (int i = 0; i < 4 && n + i < a.N; i++) b[i] = __ldg(a.bias + n + i);
    for (int mb = c0 + warp; mb < end; mb += kPrEpiWarps) {
        const float4 v = *(const float4 *)(stg + (mb - c0) * kTcTileN + lane * 4);
        const float e[4] = {v.x + b[0], v.y + b[1], v.z + b[2], v.w + b[3]};
        float *o = a.out + ((size_t)(a.epi == TC_EPI_STORE ? 0 : tl.sp) * a.M + tl.m0 + mb) * a.ld_out + n;
        if (whole) {
            *(float4 *)o = make_float4(e[0], e[1], e[2], e[3]);
        } else {
            for (int i = 0; i < 4 && n + i < a.N; i++) o[i] = e[i];
        }
    }
}

template <bool GROUPED, int TERMS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPrThreads, 1)
vb_tc_pair_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const RowsArgs a) {
    pdl_launch_dependents();
    extern __shared__ unsigned char pr_smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)pr_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *stages = base;
    using C = PrCfg<TERMS>;
    float *stg = (float *)(base + kPrStages * C::stage);
    float *rscale = (float *)((unsigned char *)stg + kPrStaging);
    uint64_t *full = (uint64_t *)(rscale + C::max_rows);
    uint64_t *empty = full + kPrStages;
    uint64_t *done = empty + kPrStages;      /* accumulator finished, [2] */
    uint64_t *drained = done + 2;            /* accumulator read by both CTAs, [2] */
    uint32_t *tmem_slot = (uint32_t *)(drained + 2);
    int *abort_flag = (int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = pr_rank();
    const int kblocks = a.K / kTcBlockK, n_tiles = a.pairs * a.row_blocks * a.splits;
    const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    uint32_t issued = 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kPrStages; i++) { vb_mbar_init(&full[i], 1); vb_mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; i++) { vb_mbar_init(&done[i], 1); vb_mbar_init(&drained[i], 2 * kPrEpiWarps); }
        *abort_flag = 0;
        vb_mbar_init_fence();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(vb_smem_u32(tmem_slot)), "r"(kPrTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    pr_cluster_sync();           /* the other CTA's barriers are ready as well */
    tc_fence_after();
    const uint32_t tmem = *(volatile uint32_t *)tmem_slot;

    if (warp == kPrEpiWarps && lane == 0) {
        /* ---- TMA producer of this CTA; the bytes of both count on the even CTA's barriers ---- */
        const uint32_t x_bytes = (uint32_t)(a.R / 2) * kTcBlockK * 2, tx = 2u * (kPrStageW + TERMS * x_bytes);
        uint32_t full_bar[kPrStages];
#pragma unroll
        for (int s = 0; s < kPrStages; s++) full_bar[s] = pr_leader(&full[s]);
        auto load_w = [&](const PrTile &t, int it, uint32_t s) {
            unsigned char *sa = stages + (size_t)s * C::stage;
            const int tile = t.w0 + (int)rank;      /* beyond the last tile: zeros */
            if (a.a_tiled) pr_load(sa, &mapA, 0, (tile * kblocks + t.kb0 + it) * kTcTileN, full_bar[s]);
            else pr_load(sa, &mapA, (t.kb0 + it) * kTcBlockK, tile * kTcTileN, full_bar[s]);
        };
        auto load_x = [&](const PrTile &t, int it, uint32_t s) {
            unsigned char *sx = stages + (size_t)s * C::stage + kPrStageW;
            const int row = t.m0 + (int)rank * (t.n_mma >> 1);
#pragma unroll
            for (int j = 0; j < TERMS; j++)
                pr_load(sx + j * C::stage_x, &mapB, (t.kb0 + it) * kTcBlockK, j * a.rows_pad + row, full_bar[s]);
        };
        bool ok = true, first = true;
        if constexpr (GROUPED) pdl_wait();          /* the table is made by an earlier kernel */
        for (int i = cluster; i < n_tiles && ok; i += n_clusters) {
            const PrTile t = pr_tile<GROUPED>(a, i, kblocks);
            if (!t.used) continue;
            int it = 0;
            if (!GROUPED && first) {
                /* the weights of the first stages depend on nothing that runs before */
                const int n = min(t.n_it, kPrStages);
                for (int s = 0; s < n; s++) {
                    if (rank == 0) vb_mbar_arrive_expect_tx(&full[s], tx);
                    load_w(t, s, (uint32_t)s);
                }
                pdl_wait();
                for (int s = 0; s < n; s++) load_x(t, s, (uint32_t)s);
                issued = (uint32_t)n;
                it = n;
            }
            first = false;
            for (; it < t.n_it; it++) {
                const uint32_t s = issued % kPrStages, use = issued / kPrStages;
                if (!vb_mbar_wait(&empty[s], (use & 1u) ^ 1u, abort_flag)) {
                    atomicCAS(a.status, 0, 11);
                    *(volatile int *)abort_flag = 1;
                    ok = false;
                    break;
                }
                if (rank == 0) vb_mbar_arrive_expect_tx(&full[s], tx);
                load_w(t, it, s);
                load_x(t, it, s);
                issued++;
            }
        }
        /* every stage handed back: no commit of the even CTA is still on its way here */
        for (uint32_t k = issued > (uint32_t)kPrStages ? issued - kPrStages : 0; k < issued && ok; k++)
            if (!vb_mbar_wait(&empty[k % kPrStages], (k / kPrStages) & 1u, abort_flag)) {
                atomicCAS(a.status, 0, 14);
                *(volatile int *)abort_flag = 1;
                ok = false;
            }
    } else if (warp == kPrEpiWarps + 1 && lane == 0 && rank == 0) {
        /* ---- MMA issuer for both CTAs ---- */
        uint32_t k = 0, n = 0;
        bool ok = true;
        if constexpr (GROUPED) pdl_wait();
        for (int i = cluster; i < n_tiles && ok; i += n_clusters) {
            const PrTile t = pr_tile<GROUPED>(a, i, kblocks);
            if (!t.used) continue;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(t.n_mma >> 3) << 17) | ((uint32_t)(2 * kTcTileN >> 4) << 24);
            for (int it = 0; it < t.n_it && ok; n++) {
                const uint32_t acc = n & 1u, d = tmem + acc * kPrAcc;
                const int end = min(t.n_it, it + t.seg);
                if (!vb_mbar_wait(&drained[acc], ((n >> 1) & 1u) ^ 1u, abort_flag)) {
                    atomicCAS(a.status, 0, 15);
                    *(volatile int *)abort_flag = 1;
                    ok = false;
                    break;
                }
                tc_fence_after();
                for (bool first = true; it < end; it++, k++, first = false) {
                    const uint32_t s = k % kPrStages, use = k / kPrStages;
                    if (!vb_mbar_wait(&full[s], use & 1u, abort_flag)) {
                        atomicCAS(a.status, 0, 12);
                        *(volatile int *)abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const unsigned char *sa = stages + (size_t)s * C::stage;
                    const uint64_t adesc = umma_desc_k_sw128(sa);
#pragma unroll
                    for (int j = 0; j < TERMS; j++) {
                        const uint64_t bdesc = umma_desc_k_sw128(sa + kPrStageW + j * C::stage_x);
#pragma unroll
                        for (int q = 0; q < kTcBlockK / 16; q++) {
                            /* three terms: the second and third have sums of their own */
                            const bool low = TERMS == 3 && j > 0;
                            pr_mma(low ? d + kPrAcc / 2 : d, adesc + 2 * q, bdesc + 2 * q, idesc, (!first || q > 0 || j > (low ? 1 : 0)) ? 1u : 0u);
                        }
                    }
                    pr_commit(&empty[s]);
                }
                pr_commit(&done[acc]);
            }
        }
    } else if (warp < kPrEpiWarps) {
        /* ---- epilogue: accumulators -> shared memory -> global, 64 rows at a time ---- */
        const int lq = warp & 3, part = warp >> 2;
        const uint32_t drained_bar[2] = {pr_leader(&drained[0]), pr_leader(&drained[1])};
        uint32_t n = 0;
        pdl_wait();
        for (int i = cluster; i < n_tiles; i += n_clusters) {
            const PrTile t = pr_tile<GROUPED>(a, i, kblocks);
            if (!t.used) continue;
            if (a.ssq) {
                vb_named_bar(1, kPrEpi);             /* the last tile's scales are read */
                for (int m = threadIdx.x; m < t.Mb; m += kPrEpi) {
                    float s = 0.0f;
                    for (int c = 0; c < a.ssq_chunks; c++) s += __ldcg(a.ssq + (size_t)(t.m0 + m) * a.ssq_chunks + c);
                    rscale[m] = 1.0f / sqrtf(s / (float)a.K + a.eps);
                }
                vb_named_bar(1, kPrEpi);
            }
            /* this thread's column of the weight tile, rows part * 16 .. of every 64 */
            constexpr int kChunks = C::max_rows / kPrChunk;
            float sum[kChunks][16];
            for (int it = 0; it < t.n_it; it += t.seg, n++) {
                const uint32_t acc = n & 1u, d = tmem + acc * kPrAcc + ((uint32_t)(lq * 32) << 16) + (uint32_t)(part * 16);
                /* after a wait that ran out the others fail at once: no thread leaves the barriers alone */
                if (!vb_mbar_wait(&done[acc], (n >> 1) & 1u, abort_flag)) {
                    atomicCAS(a.status, 0, 13);
                    *(volatile int *)abort_flag = 1;
                }
                __syncwarp();
                tc_fence_after();
#pragma unroll
                for (int q = 0; q < kChunks; q++) {
                    if (q * kPrChunk + part * 16 < t.Mb) {
                        uint32_t r[16];
                        tmem_ld16(d + (uint32_t)(q * kPrChunk), r);
                        if constexpr (TERMS == 3) {
                            uint32_t low[16];
                            tmem_ld16(d + (uint32_t)(kPrAcc / 2 + q * kPrChunk), low);
#pragma unroll
                            for (int j = 0; j < 16; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(low[j]));
                        }
                        if (it == 0) {
#pragma unroll
                            for (int j = 0; j < 16; j++) sum[q][j] = __uint_as_float(r[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; j++) sum[q][j] += __uint_as_float(r[j]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) pr_arrive(drained_bar[acc]);
            }
#pragma unroll 1
            for (int q = 0; q * kPrChunk < t.Mb; q++) {
                const int c0 = q * kPrChunk, c = c0 + part * 16;
                if (c < t.Mb) {
                    float *to = stg + part * 16 * kTcTileN + lq * 32 + lane;
#pragma unroll
                    for (int u = 0; u < kChunks; u++)
                        if (u == q) {                       /* registers have no index */
#pragma unroll
                            for (int j = 0; j < 16; j++) to[j * kTcTileN] = a.ssq ? sum[u][j] * rscale[min(c + j, t.Mb - 1)] : sum[u][j];
                        }
                }
                vb_named_bar(1, kPrEpi);
                pr_store<TERMS>(a, stg, t, t.t0 + (int)rank, c0, warp, lane);
                vb_named_bar(1, kPrEpi);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kPrEpiWarps && lane == 0 && rank == 0 && *(volatile int *)abort_flag) {
        /* abort path: let copies already in flight land before the shared memory goes away */
        for (uint32_t k = issued > (uint32_t)kPrStages ? issued - kPrStages : 0; k < issued; k++) {
            const long long t0c = clock64();
            while (!vb_mbar_try_wait(&full[k % kPrStages], (k / kPrStages) & 1u)) {
                if (clock64() - t0c > VB_WAIT_CYCLES / 8) break;
            }
        }
    }
    __syncwarp();
    pr_cluster_sync();           /* nobody reads or signals the other CTA any more */
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPrTmemCols) : "memory");
    }
}

int sm_pairs() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return n / 2;
}

/* Clocks of a launch with tiles of R rows, as the note at the top counts them: a k-block costs the larger of the tensor
 * pipe's 2 R a term and shared memory's (16 + 8 R / 64 KB read and as many written per term, and 16 KB of weights); the
 * epilogue of the last tile is not hidden. */
long long launch_cost(int M, int pairs, int k_iters, int splits, int clusters, int R, int terms) {
    const long long tiles = (long long)pairs * ((M + R - 1) / R) * splits;
    return (tiles + clusters - 1) / clusters * (k_iters * (long long)(std::max(2 * terms * R, 128 * (1 + terms) + terms * R) + 24) + 200) + 24 * R;
}
int pick_rows(int M, int pairs, int k_iters, int splits, int clusters, int terms) {
    const int least = terms == 3 ? 32 : 64;
    int best = 0;
    long long cost = 0;
    for (int R = terms == 3 ? PrCfg<3>::max_rows : PrCfg<2>::max_rows; R >= least; R -= 32) {
        if (R > least && R >= M + 32) continue;
        const long long c = launch_cost(M, pairs, k_iters, splits, clusters, R, terms);
        if (!best || c < cost) { best = R; cost = c; }
    }
    return best;
}

template <bool GROUPED, int TERMS>
int launch_pair(const TcWeight &w, const TcActs &a, RowsArgs &ra, int clusters, cudaStream_t st) {
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(vb_tc_pair_kernel<GROUPED, TERMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, PrCfg<TERMS>::smem) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        attr = true;
    }
    CUtensorMap map;
    if (tc_map(&map, a.buf, (uint64_t)TERMS * a.rows_pad, (uint64_t)a.K, (uint32_t)ra.R / 2)) return -1;
    const long long tiles = (long long)ra.pairs * ra.row_blocks * ra.splits;
    return launch_pdl(vb_tc_pair_kernel<GROUPED, TERMS>, dim3(2 * (unsigned)std::min<long long>(tiles, clusters)), dim3(kPrThreads),
                      (size_t)PrCfg<TERMS>::smem, st, w.map, map, ra) == cudaSuccess
               ? 0
               : -1;
}

RowsArgs rows_args(const TcWeight &w, const TcActs &a, const TcGemm &g) {
    RowsArgs ra = {};
    ra.out = g.out; ra.out_terms = g.out_terms; ra.bias = g.bias; ra.ssq = g.ssq; ra.status = g.status; ra.eps = g.eps;
    ra.K = w.K; ra.rows_pad = a.rows_pad; ra.ld_out = g.ld_out; ra.splits = g.splits; ra.epi = g.epi; ra.ssq_chunks = g.ssq_chunks;
    ra.a_tiled = w.tiled ? 1 : 0; ra.out_rows_pad = g.out_rows_pad; ra.act_n0 = g.act_n0; ra.out_terms_ld = g.out_terms_ld;
    ra.out_col0 = g.out_col0; ra.segment = g.segment > 0 ? g.segment : 1;
    return ra;
}

bool terms_epilogue_ok(const TcGemm &g) {
    return g.out_terms && g.act_n0 % kTcTileN == 0 && g.out_terms_ld % 4 == 0 && g.out_col0 % 4 == 0;
}

} // namespace

int tc_row_splits(int N, int K, int M, int n_sm, int terms) {
    const int pairs = ((N + kTcTileN - 1) / kTcTileN + 1) / 2, clusters = n_sm / 2, kblocks = K / kTcBlockK;
    int best = 1;
    long long cost = 0;
    for (int s = 1; s <= std::min(kTcMaxSplits, kblocks); s++) {
        const int it = (kblocks + s - 1) / s;
        /* a further partial result is M rows of N written and read again: about 4 values per clock and pair */
        const long long c = launch_cost(M, pairs, it, s, clusters, pick_rows(M, pairs, it, s, clusters, terms), terms) +
                            (long long)s * M * N / (4LL * clusters);
        if (s == 1 || c < cost) { best = s; cost = c; }
    }
    return best;
}

int tc_gemm_rows(const TcWeight &w, const TcActs &a, const TcGemm &g, cudaStream_t st) {
    if ((g.epi == TC_EPI_TERMS || g.epi == TC_EPI_RELU2_TERMS) &&
        (!terms_epilogue_ok(g) || g.out_rows_pad < g.M || (g.act_n0 > 0 && !g.out)))
        return -1;
    const int clusters = sm_pairs();
    if (clusters < 1) return -1;
    RowsArgs ra = rows_args(w, a, g);
    ra.N = w.N; ra.M = g.M;
    ra.pairs = ((w.N + kTcTileN - 1) / kTcTileN + 1) / 2;
    ra.R = pick_rows(g.M, ra.pairs, (w.K / kTcBlockK + g.splits - 1) / g.splits, g.splits, clusters, g.terms);
    ra.row_blocks = (g.M + ra.R - 1) / ra.R;
    return g.terms == 3 ? launch_pair<false, 3>(w, a, ra, clusters, st) : launch_pair<false, 2>(w, a, ra, clusters, st);
}

int tc_gemm_grouped(const TcWeight &w, const TcActs &a, const TcGemm &g, int n, const int4 *table, int n_blocks, cudaStream_t st) {
    constexpr int kRows = 128;
    const int tiles = (n + kTcTileN - 1) / kTcTileN;
    if (!w.ok || !w.tiled || !a.ok || w.K != a.K || n < 1 || n_blocks < 1 || !table || g.splits != 1) return -1;
    if (w.N % (tiles * kTcTileN) || (size_t)n_blocks * kRows > (size_t)a.rows_pad || g.act_n0 != 0) return -1;
    if (g.epi == TC_EPI_TERMS || g.epi == TC_EPI_RELU2_TERMS) {
        if (!terms_epilogue_ok(g) || g.out_rows_pad < n_blocks * kRows) return -1;
    } else if (g.epi != TC_EPI_STORE || !g.out || g.ld_out < n) {
        return -1;
    }
    const int clusters = sm_pairs();
    if (clusters < 1) return -1;
    RowsArgs ra = rows_args(w, a, g);
    ra.a_tiled = 1;
    ra.bias = nullptr; ra.ssq = nullptr;
    ra.N = n; ra.M = n_blocks * kRows; ra.R = kRows;
    ra.row_blocks = n_blocks;
    ra.pairs = (tiles + 1) / 2;
    ra.table = table; ra.group_tiles = tiles;
    return g.terms == 3 ? launch_pair<true, 3>(w, a, ra, clusters, st) : launch_pair<true, 2>(w, a, ra, clusters, st);
}

} // namespace vb
