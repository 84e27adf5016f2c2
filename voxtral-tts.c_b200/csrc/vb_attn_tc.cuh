/*
 * vb_attn_tc.cuh - softmax attention of many query rows on the 5th-generation tensor cores: prompts of the speech
 * decoder (vb_prefill.cu) and of the language models (vb_lm_attn.cu).
 *
 * A CTA owns one KV head and 128 (row, query head) pairs, so that the heads of a group share every key and value that
 * is brought in, and walks the visible keys 64 at a time. Every product a.b is taken as a_hi.b_hi + a_hi.b_lo +
 * a_lo.b_hi on BF16 halves (16 mantissa bits each side), summed in fp32 in TMEM:
 *
 *   S [128 x 64]    = Q . K^T   Q high halves in TMEM (A operand), low halves too, or in shared memory for heads over 128
 *   O [128 x vdim] += P . V     P as halves in TMEM, in S's own columns; V rows [key][dim] are an MN-major B operand
 *
 * Scores, softcap, running maximum, weights and sums are fp32, a thread owns a row. Two warpgroups take alternate key
 * tiles with a maximum, sum and accumulator each (merged at the end), so that the tensor pipe works on one tile while
 * the other is in its softmax. An accumulator is rescaled only when a row's maximum has risen by more than 2^8: the
 * reference a row is taken against cancels in the quotient. (Alternating groups and conditional rescaling are a published
 * scheme, FlashAttention-4's.)
 *
 * Warps: 0-3, 4-7 softmax, 8-11 bring keys and 12-13 values into two rings, 14 issues the MMAs. All waits are bounded.
 *
 * What bounds it, by a timeline on the device: the S products, 24 MMAs of 64 columns a tile at 77 clocks (36 of 65 for
 * heads of 192), which is what MMAs of 128 columns take too, then P . V, 12 at 60; 3300 and 4000 clocks a tile. 2048 rows,
 * window 1024, 32 heads: 128 on 8 KV heads 588 us on warp-level MMAs (mma.sync, 16 rows a warp, 44 useful TFLOP/s), 201 with
 * tiles copied 16 bytes a lane, 164 by TMA; 192 + 128 each with its own 830, 282, 225 us. Short prompts see what comes before
 * and after the tiles: 58 rows of the speech decoder 17.8 us with queries and results moved a row at a time, 13.1 now, 1203
 * rows 78.6 -> 66.6, 2048 rows of a language model with window and softcap 175 -> 158.
 */
#ifndef VB_ATTN_TC_CUH
#define VB_ATTN_TC_CUH

#include "vb_lm_attn.cuh"
#include "vb_umma.cuh"

namespace vb {

constexpr int kAtRows = 128, kAtKeys = 64;
constexpr int kAtSoft = 256, kAtLoadK = 128, kAtLoadV = 64, kAtThreads = kAtSoft + kAtLoadK + kAtLoadV + 32;
constexpr int kAtMmaWarp = (kAtThreads - 32) / 32;
constexpr int kAtBlock = kAtKeys * 128;            /* 64 keys x 64 columns */
constexpr int kAtStatus = 52;
constexpr uint32_t kAtTmemCols = 512, kAtO = 128, kAtQ = 384;

/* What every use has in common. */
struct AtArgs {
    int M, heads, kv_heads, dim, vdim;
    int window, keep;
    float scale, softcap;
    int *status;
    int tma;                     /* the tensor maps are there: whole tiles of keys are brought in by TMA */
};
/* Keys (and a part that all heads share), values: 64 columns x 64 rows of a plane. */
struct AtMaps {
    CUtensorMap k, k2, v;
};

template <int DK, int DV>
struct AtCfg {
    static constexpr bool kQlTmem = DK <= 2;
    static constexpr int kSlots = DK <= 2 ? 3 : 2;
    static constexpr int kSlotK = 2 * DK * kAtBlock, kSlotV = 2 * DV * kAtBlock;
    static constexpr int kQl = kQlTmem ? 0 : DK * kAtRows * 128;
    static constexpr int kSmem = kQl + kSlots * (kSlotK + kSlotV) + 1024 + 256;
    /* 16-column steps of the queries that a warp has on their way at once (of 2 * DK): 8 or 16 loads of 16 bytes a lane */
    static constexpr int kQBatch = DK <= 2 ? 2 * DK : 2;
    static_assert(2 * DK % kQBatch == 0, "whole batches");
    static_assert(kSmem <= 232448, "over the 227 KB a CTA may use");
    static_assert(kAtQ + (kQlTmem ? 2 : 1) * DK * 32 <= kAtTmemCols, "Q does not fit TMEM");
};

/* A descriptor's low word, which holds the address and is what the steps of a product add to; the high word is the same for
 * all of an operand. By the source a sum of whole descriptors is the same number: addresses stay below 2^18, 16 bytes a unit, so
 * nothing carries. Even so, heads of 192 gave wrong scores from the third key tile on with such sums, as if low halves of the
 * queries had been read from beyond their place, after a change elsewhere in the kernel, and give right ones with these. The cause
 * is not known. The GEMMs (vb_tc.cu, vb_tc_rows.cu) add whole descriptors in one copy of a loop each. */
struct AtDesc {
    uint32_t lo, hi;
    VB_DEVINL explicit AtDesc(uint64_t d) : lo((uint32_t)d), hi((uint32_t)(d >> 32)) {}
    VB_DEVINL AtDesc at(int units) const {          /* so many 16 bytes on */
        AtDesc r = *this;
        r.lo += (uint32_t)units;
        return r;
    }
};
VB_DEVINL void at_mma_ts(uint32_t d, uint32_t a, AtDesc b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d), "r"(a), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
VB_DEVINL void at_mma_ss(uint32_t d, AtDesc a, AtDesc b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d), "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
#define VB_AT_R8(r, o) "r"((r)[o]), "r"((r)[o + 1]), "r"((r)[o + 2]), "r"((r)[o + 3]), "r"((r)[o + 4]), "r"((r)[o + 5]), "r"((r)[o + 6]), "r"((r)[o + 7])
#define VB_AT_W8(r, o) "=r"((r)[o]), "=r"((r)[o + 1]), "=r"((r)[o + 2]), "=r"((r)[o + 3]), "=r"((r)[o + 4]), "=r"((r)[o + 5]), "=r"((r)[o + 6]), "=r"((r)[o + 7])
/* 32 columns of this thread's TMEM lane; at_ld_wait before the values are used, at_st_wait before they are handed on */
VB_DEVINL void at_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : VB_AT_W8(r, 0), VB_AT_W8(r, 8), VB_AT_W8(r, 16), VB_AT_W8(r, 24)
        : "r"(taddr)
        : "memory");
}
VB_DEVINL void at_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::VB_AT_R8(r, 0), VB_AT_R8(r, 8), VB_AT_R8(r, 16), VB_AT_R8(r, 24), "r"(taddr)
        : "memory");
}
/* 8 columns of 16 TMEM lanes: lane l of the warp has columns 2 (l % 4) and on of rows l / 4 (a, b) and l / 4 + 8 (c, d) */
VB_DEVINL void at_st_16x8(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
VB_DEVINL void at_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
VB_DEVINL void at_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
VB_DEVINL float at_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
VB_DEVINL float at_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
/* cap2 * tanh(z), by way of one exponential: cap2 - 2 cap2 / (1 + e^2z). Its error is about 2^-22 of cap2 whatever z is, up to
 * kAtSoftcap no more than that of the two-term products (2^-17 of |q||k|). For larger caps scores below a quarter of the
 * cap are taken by the odd powers of Taylor's series to the ninth (2^-26 of the result): at cap 100000 the exponential left
 * 0.03. (The series for all caps: a 4001-token prompt, cap 30, 59.6 -> 60.3 ms.) */
constexpr float kAtTanhSmall = 0.25f, kAtSoftcap = 64.0f;
VB_DEVINL float at_tanh_small(float z, float cap2) {
    const float q = z * z;
    return cap2 * z * fmaf(q, fmaf(q, fmaf(q, fmaf(q, 62.0f / 2835.0f, -17.0f / 315.0f), 2.0f / 15.0f), -1.0f / 3.0f), 1.0f);
}
/* z = s * cap_in * ln 2 / 2 */
constexpr float kAtHalfLn2 = 0.34657359f;
VB_DEVINL float at_tanh_large(float s, float cap_in, float cap2) { return fmaf(-2.0f * cap2, at_rcp(1.0f + at_ex2(s * cap_in)), cap2); }
/* vb_mbar_wait with one answer for the warp: no lane leaves the others alone in a warp-wide instruction */
VB_DEVINL bool at_warp_wait(uint64_t *bar, uint32_t parity, volatile int *cta_abort) {
    return __all_sync(0xffffffffu, vb_mbar_wait(bar, parity, cta_abort));
}
VB_DEVINL void at_tma(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            vb_smem_u32(dst)),
        "l"(map), "r"(vb_smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
/* Two values as packed BF16 high halves and packed remainders. */
VB_DEVINL void at_split2(float a, float b, uint32_t &hi, uint32_t &lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
    const float ra = a - __uint_as_float(hi << 16), rb = b - __uint_as_float(hi & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(rb), "f"(ra));
}

/* Rows [key][64 dims] as the B operand of P . V, read along the dims (MN-major): groups of eight keys 1024 bytes apart,
 * blocks of 64 dims kAtBlock apart. */
VB_DEVINL uint64_t at_desc_mn(uint32_t addr) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)(kAtBlock >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
VB_DEVINL uint32_t at_idesc(int n, bool mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kAtRows >> 4) << 24);
}
/* Byte offset of 16-byte chunk `chunk` (0..7) of a 128-byte row, as the 128-byte swizzle has it */
VB_DEVINL uint32_t at_off(int row, int chunk) { return (uint32_t)(row * 128 + (((chunk ^ row) & 7) << 4)); }

/* A use (SRC) says where things come from and go:
 *   tma_keys(...) / tma_values(...)   request a tile by TMA: where AtArgs says so and boxes(j0, n) does, or always (kBoxes:
 *                                what lies beyond the last key is zeros)
 *   start()                      after the wait for the previous kernel: resolves what lies in device memory
 *   here()                       what of it this block is to use
 *   rows(a)                      how many there are: a launch may serve several prompts (blockIdx.z), a.M the most of one
 *   pos0()                       position of row 0
 *   q4(row, head, d, part)       four query values (zeros beyond the head), or with kParts one of parts() addends of theirs
 *   turned(row, head, d, v)      those values rotated, where they are not already
 *   keys(...) / values(...)      otherwise, with cp.async: a loading warp's 16 keys, into blocks of 64 columns, high halves
 *                                first
 *   gate(row, head)              factor of a result row
 *   put4(row, column, v)         four results */
template <int DK, int DV, class SRC>
__global__ void __launch_bounds__(kAtThreads, 1) vb_attn_tc_kernel(const __grid_constant__ AtMaps maps, const AtArgs a, const __grid_constant__ SRC src_arg) {
    using Cfg = AtCfg<DK, DV>;
    extern __shared__ unsigned char at_smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)at_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *ql_s = base, *k_s = ql_s + Cfg::kQl, *v_s = k_s + Cfg::kSlots * Cfg::kSlotK;
    uint64_t *bars = (uint64_t *)(v_s + Cfg::kSlots * Cfg::kSlotV);
    uint64_t *k_full = bars, *k_empty = k_full + Cfg::kSlots, *v_full = k_empty + Cfg::kSlots, *v_empty = v_full + Cfg::kSlots;
    uint64_t *s_full = v_empty + Cfg::kSlots, *p_full = s_full + 2, *o_done = p_full + 2, *q_full = o_done + 2;
    uint32_t *tmem_slot = (uint32_t *)(q_full + 1);
    int *abort_flag = (int *)(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = a.heads / a.kv_heads, g = blockIdx.x;
    auto src = src_arg.here();
    const int pairs = src.rows(a) * group;
    const int P0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kAtRows;           /* the latest rows see the most keys: they go first */
    if (P0 >= pairs) return;                                                   /* a shorter prompt beside a longer one */
    if (tid == 0) {
        for (int i = 0; i < Cfg::kSlots; i++) {
            vb_mbar_init(&k_full[i], kAtLoadK);
            vb_mbar_init(&v_full[i], kAtLoadV);
            vb_mbar_init(&k_empty[i], 1);
            vb_mbar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            vb_mbar_init(&s_full[i], 1);
            vb_mbar_init(&p_full[i], 128);
            vb_mbar_init(&o_done[i], 1);
        }
        vb_mbar_init(q_full, kAtSoft);
        *abort_flag = 0;
        vb_mbar_init_fence();
    }
    if (warp == kAtMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(vb_smem_u32(tmem_slot)), "r"(kAtTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *(volatile uint32_t *)tmem_slot;
    pdl_launch_dependents();       /* not before the allocation: a GEMM that starts early must not take columns this kernel needs */
    /* The queries of a softmax warp's 32 rows, 16 columns a step, the steps in turn by the two warpgroups. Four lanes read 64
     * bytes of a row, which is how a 16 x 8 TMEM store wants them; the loads of a batch are all on their way before the first
     * is used; rows past the end repeat the last one. (Two lanes a row, 32 columns at a time, by way of shared memory to the
     * lane that owns the row: 8000 clocks from the wait to queries in place for 128 x 128, 2200 to 3500 now.) */
    constexpr bool kEarly = DK <= 2;            /* one batch: before what start() fetches (in two places 147 us, not 138, for heads of 192) */
    const int w_q = warp >> 2, d_q = (lane & 3) * 4;
    int qrow[4], qhead[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int x = P0 + (warp & 3) * 32 + (lane >> 2) + 8 * i;
        qrow[i] = (x < pairs ? x : pairs - 1) / group;
        qhead[i] = g * group + (x < pairs ? x : pairs - 1) - qrow[i] * group;
    }
    float4 qv[Cfg::kQBatch][4];
    auto q_load = [&](int batch) {
        auto column = [&](int u) { return ((batch * Cfg::kQBatch + u) * 2 + w_q) * 16 + d_q; };
#pragma unroll
        for (int u = 0; u < Cfg::kQBatch; u++)
#pragma unroll
            for (int i = 0; i < 4; i++) qv[u][i] = src.q4(qrow[i], qhead[i], column(u), 0);
        if constexpr (SRC::kParts) {             /* a part of the whole batch at a time, two on their way */
#pragma unroll 2
            for (int p = 1; p < src.parts(); p++) {
                float4 t[Cfg::kQBatch][4];
#pragma unroll
                for (int u = 0; u < Cfg::kQBatch; u++)
#pragma unroll
                    for (int i = 0; i < 4; i++) t[u][i] = src.q4(qrow[i], qhead[i], column(u), p);
#pragma unroll
                for (int u = 0; u < Cfg::kQBatch; u++)
#pragma unroll
                    for (int i = 0; i < 4; i++) { qv[u][i].x += t[u][i].x; qv[u][i].y += t[u][i].y; qv[u][i].z += t[u][i].z; qv[u][i].w += t[u][i].w; }
            }
        }
    };
    pdl_wait();
    if (kEarly && warp < 8) q_load(0);
    src.start();
    const int pos0 = src.pos0();
    const int last = P0 + kAtRows < pairs ? P0 + kAtRows - 1 : pairs - 1;
    const int imin = pos0 + P0 / group, imax = pos0 + last / group;
    const KeyTiles kt = key_tiles<kAtKeys>(imin, imax, a.window, a.keep);
    const int n_tiles = kt.n_tiles;

    auto give_up = [&]() {
        atomicCAS(a.status, 0, kAtStatus);
        *(volatile int *)abort_flag = 1;
    };

    if (warp < 8) {
        /* ---- softmax: warpgroup w takes key tiles w, w + 2, ...; a thread owns pair P0 + r ---- */
        const int w = warp >> 2, r = tid & 127, P = P0 + r;
        const bool valid = P < pairs;
        const int row = valid ? P / group : 0, head = g * group + (valid ? P - row * group : 0), i = pos0 + row;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16, tS = tmem + lanes + (uint32_t)(w * kAtKeys), tO = tmem + lanes + kAtO + (uint32_t)(w * 128);
#pragma unroll 1
        for (int batch = 0; batch < 2 * DK / Cfg::kQBatch; batch++) {
            if (!kEarly || batch > 0) q_load(batch);
#pragma unroll
            for (int u = 0; u < Cfg::kQBatch; u++) {
                const int step = (batch * Cfg::kQBatch + u) * 2 + w;
                uint32_t hi[4][2], lo[4][2];
#pragma unroll
                for (int i2 = 0; i2 < 4; i2++) {
                    float4 e = src.turned(qrow[i2], qhead[i2], step * 16 + d_q, qv[u][i2]);
                    if (a.scale <= 0.0f) {             /* the scores are multiplied by |scale| below, or by one */
                        const float f = a.scale < 0.0f ? -1.0f : 0.0f;
                        e = make_float4(e.x * f, e.y * f, e.z * f, e.w * f);
                    }
                    at_split2(e.x, e.y, hi[i2][0], lo[i2][0]);
                    at_split2(e.z, e.w, hi[i2][1], lo[i2][1]);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t to = tmem + lanes + ((uint32_t)(16 * h) << 16) + kAtQ + (uint32_t)(step * 8);
                    at_st_16x8(to, hi[2 * h][0], hi[2 * h][1], hi[2 * h + 1][0], hi[2 * h + 1][1]);
                    if constexpr (Cfg::kQlTmem) at_st_16x8(to + DK * 32, lo[2 * h][0], lo[2 * h][1], lo[2 * h + 1][0], lo[2 * h + 1][1]);
                }
                if constexpr (!Cfg::kQlTmem) {
#pragma unroll
                    for (int i2 = 0; i2 < 4; i2++)
                        *reinterpret_cast<uint2 *>(ql_s + (step >> 2) * kAtRows * 128 +
                                                   at_off((warp & 3) * 32 + (lane >> 2) + 8 * i2, (step & 3) * 2 + ((lane & 3) >> 1)) + (lane & 1) * 8) =
                            make_uint2(lo[i2][0], lo[i2][1]);
                }
            }
        }
        at_st_wait();
        at_proxy_fence();
        tc_fence_before();
        vb_mbar_arrive(q_full);

        /* Scores as powers of two: S times mul (to twice fp32's precision), or with a softcap cap * tanh(x / cap), x = S *
         * scale, in these units. */
        const double log2e = 1.4426950408889634, dmul = a.softcap > 0.0f || a.scale == 0.0f ? 1.0 : fabs((double)a.scale) * log2e;
        float mul = __double2float_rz(dmul);
        if ((double)mul == dmul) mul = __uint_as_float(__float_as_uint(mul) - 1u);       /* mul_lo > 0: a masked -inf stays one */
        const float mul_lo = (float)(dmul - (double)mul);
        const float cap2 = (float)(a.softcap * log2e), cap_in = a.softcap > 0.0f ? (float)(2.0 * log2e * fabs((double)a.scale) / a.softcap) : 0.0f;
        float ref = -INFINITY, sum = 0.0f;      /* the row's reference (in powers of two), its sum of weights against it */
        int it = 0;
        for (int t = w; t < n_tiles; t += 2, it++) {
            int j0, n;
            key_tile<kAtKeys>(kt, t, &j0, &n);
            if (!at_warp_wait(&s_full[w], (uint32_t)it & 1u, abort_flag)) { give_up(); break; }
            tc_fence_after();
            float s[kAtKeys];
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t reg[32];
                at_ld32(tS + (uint32_t)(c * 32), reg);
#pragma unroll
                for (int k = 0; k < 32; k++) s[c * 32 + k] = __uint_as_float(reg[k]);
            }
            if (a.softcap > 0.0f) {
                if (a.softcap <= kAtSoftcap) {
#pragma unroll
                    for (int k = 0; k < kAtKeys; k++) s[k] = at_tanh_large(s[k], cap_in, cap2);
                } else {
#pragma unroll
                    for (int k = 0; k < kAtKeys; k++) {
                        const float z = s[k] * cap_in * kAtHalfLn2;
                        s[k] = fabsf(z) < kAtTanhSmall ? at_tanh_small(z, cap2) : at_tanh_large(s[k], cap_in, cap2);
                    }
                }
            }
            const bool all_seen = n == kAtKeys && j0 + kAtKeys - 1 <= imin && (a.window <= 0 || imax - j0 < a.window || j0 + kAtKeys <= a.keep);
            if (!all_seen) {
                const int k_end = n - 1 < i - j0 ? n - 1 : i - j0;               /* last one not too late */
                const int k_win = a.window > 0 ? i - a.window + 1 - j0 : 0, k_keep = a.keep - j0;
#pragma unroll
                for (int k = 0; k < kAtKeys; k++)
                    if (k > k_end || (k < k_win && k >= k_keep)) s[k] = -INFINITY;
            }
            float top4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int k = 4; k < kAtKeys; k++) top4[k & 3] = fmaxf(top4[k & 3], s[k]);
            const float top = fmaxf(fmaxf(top4[0], top4[1]), fmaxf(top4[2], top4[3])) * mul;
            const bool rise = top > ref + 8.0f;
            if (__any_sync(0xffffffffu, rise)) {
                const float now = rise ? top : ref, f = rise ? at_ex2(ref - now) : 1.0f;     /* the first time: 0 */
                if (it > 0) {
                    if (!at_warp_wait(&o_done[w], (uint32_t)(it - 1) & 1u, abort_flag)) { give_up(); break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 2 * DV; c++) {
                        uint32_t reg[32];
                        at_ld32(tO + (uint32_t)(c * 32), reg);
#pragma unroll
                        for (int k = 0; k < 32; k++) reg[k] = __float_as_uint(__uint_as_float(reg[k]) * f);
                        at_st32(tO + (uint32_t)(c * 32), reg);
                    }
                }
                sum *= f;
                ref = now;
            }
            const float m = ref > -INFINITY ? ref : 0.0f;         /* no key seen yet: every weight below is 2^-inf = 0 */
            float sum4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t reg[32];
#pragma unroll
                for (int k = 0; k < 32; k += 2) {
                    float p[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const float x = s[c * 32 + k + u];
                        p[u] = at_ex2(fmaf(x, mul_lo, fmaf(x, mul, -m)));
                        sum4[(k + u) & 3] += p[u];
                    }
                    at_split2(p[0], p[1], reg[k / 2], reg[16 + k / 2]);
                }
                at_st32(tS + (uint32_t)(c * 32), reg);            /* 16 columns of high halves, 16 of low ones */
            }
            sum += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
            at_st_wait();
            tc_fence_before();
            vb_mbar_arrive(&p_full[w]);
        }
        if (it > 0 && !at_warp_wait(&o_done[w], (uint32_t)(it - 1) & 1u, abort_flag)) give_up();
        /* Both halves of the keys, merged, each warpgroup half of the columns; by way of shared memory, so that a warp
         * writes the columns of a row side by side (from the TMEM layout, a thread per row, every store touches 32 rows). */
        vb_named_bar(1, kAtSoft);                                 /* every product is done: the rings are free */
        float2 *ml = reinterpret_cast<float2 *>(k_s);
        float *rows = reinterpret_cast<float *>(k_s + 2 * kAtRows * 8);
        constexpr int kLd = DV * 64 + 4;                          /* 16 bytes on: eight rows of a column hit all banks */
        static_assert(2 * kAtRows * 8 + kAtRows * kLd * 4 <= Cfg::kSlots * (Cfg::kSlotK + Cfg::kSlotV), "results do not fit the rings");
        ml[w * kAtRows + r] = make_float2(ref, sum);
        tc_fence_before();
        vb_named_bar(1, kAtSoft);
        tc_fence_after();
        const float2 A = ml[r], B = ml[kAtRows + r];
        const float top = fmaxf(A.x, B.x);
        const float fa = A.y > 0.0f ? at_ex2(A.x - top) : 0.0f, fb = B.y > 0.0f ? at_ex2(B.x - top) : 0.0f;
        const float inv = 1.0f / (A.y * fa + B.y * fb) * (valid ? src.gate(row, head) : 1.0f);
        const float ra = fa * inv, rb = fb * inv;
#pragma unroll 1
        for (int c = w * DV; c < w * DV + DV; c++) {
            uint32_t oa[32], ob[32];
            at_ld32(tmem + lanes + kAtO + (uint32_t)(c * 32), oa);
            if (n_tiles > 1) at_ld32(tmem + lanes + kAtO + 128u + (uint32_t)(c * 32), ob);
#pragma unroll
            for (int k = 0; k < 32; k++) {
                float v = __uint_as_float(oa[k]) * ra;
                if (n_tiles > 1) v += __uint_as_float(ob[k]) * rb;
                oa[k] = __float_as_uint(v);
            }
#pragma unroll
            for (int k = 0; k < 32; k += 4) *reinterpret_cast<uint4 *>(rows + r * kLd + c * 32 + k) = make_uint4(oa[k], oa[k + 1], oa[k + 2], oa[k + 3]);
        }
        vb_named_bar(1, kAtSoft);
        /* Two rows of a warp at a time, whose places each lane has worked out for one: a row at a time, with a division each,
         * took 8700 clocks of a tile of 128 x 128 with three terms, 5500 now, with two 3500 (four or eight rows: more code, no
         * faster; terms made above, where a thread has 32 values side by side, and copied from there: 1700 clocks more). */
        constexpr int kWarps = kAtSoft / 32, kAhead = 2;
        const int my_pair = P0 + warp + kWarps * (lane % (kAtRows / kWarps)), my_row = my_pair < pairs ? my_pair / group : -1;
        const int c = lane * 4;
#pragma unroll 1
        for (int n = 0; n < kAtRows / kWarps; n += kAhead) {
            int m[kAhead];
            float4 o[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                m[u] = __shfl_sync(0xffffffffu, my_row, n + u);
                if (c < a.vdim) o[u] = *reinterpret_cast<const float4 *>(rows + (warp + kWarps * (n + u)) * kLd + c);
            }
            if (m[0] < 0) break;
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                const float v[4] = {o[u].x, o[u].y, o[u].z, o[u].w};
                if (m[u] >= 0 && c < a.vdim) src.put4(m[u], (g * group + P0 + warp + kWarps * (n + u) - m[u] * group) * a.vdim + c, v);
            }
        }
    } else if (warp < kAtMmaWarp) {
        /* ---- four warps for the keys, two for the values: a slot of K is free after S, one of V only after the softmax,
         * and a loader that took both in turn handed keys over no sooner than the values before them ---- */
        const bool is_k = warp < 12;
        const int lw = is_k ? warp - 8 : (warp - 12) * 2;      /* 16 keys each, values 32 */
        uint64_t *full = is_k ? k_full : v_full, *empty = is_k ? k_empty : v_empty;
        if (is_k && a.dim % 16) {          /* the last 16 columns of a product reach beyond the head: zeros there, for good */
            const int chunk = a.dim / 8;
            for (int x = tid - kAtSoft; x < Cfg::kSlots * 2 * kAtKeys; x += kAtLoadK) {
                const int key = x % kAtKeys, plane = x / kAtKeys;
                *reinterpret_cast<uint4 *>(k_s + (plane * DK + (chunk >> 3)) * kAtBlock + at_off(key, chunk)) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        int told = 0;              /* tiles before this one are handed over */
        auto hand_over = [&](int upto) {
            if (told >= upto) return;
            at_proxy_fence();
            for (; told < upto; told++) vb_mbar_arrive(&full[told % Cfg::kSlots]);
        };
        /* (Copied row by row, 16 bytes a lane, a tile of 192-wide keys takes a warp 4000 clocks of address arithmetic. That
         * remains for tiles that end early, wrap around the ring, or have columns that are not whole boxes.) */
        for (int t = 0; t < n_tiles; t++) {
            const int slot = t % Cfg::kSlots;
            const uint32_t parity = ((uint32_t)(t / Cfg::kSlots) & 1u) ^ 1u;
            if (!__all_sync(0xffffffffu, vb_mbar_try_wait(&empty[slot], parity))) {
                lm_cp_wait_all();                    /* what waits for the slot may wait for what is on its way */
                hand_over(t);
                if (!at_warp_wait(&empty[slot], parity, abort_flag)) { give_up(); break; }
            }
            int j0, n;
            key_tile<kAtKeys>(kt, t, &j0, &n);
            if (SRC::kBoxes || (a.tma && src.boxes(j0, n))) {
                lm_cp_wait_all();
                hand_over(t);
                if (lw == 0 && lane == 0) {
                    vb_mbar_arrive_expect_tx(&full[slot], is_k ? Cfg::kSlotK : Cfg::kSlotV);
                    if (is_k) src.template tma_keys<DK>(a, maps, k_s + slot * Cfg::kSlotK, g, j0, &full[slot]);
                    else src.template tma_values<DV>(a, maps, v_s + slot * Cfg::kSlotV, g, j0, &full[slot]);
                } else {
                    vb_mbar_arrive(&full[slot]);
                }
                told = t + 1;
                continue;
            }
            if constexpr (!SRC::kBoxes) {
                if (is_k) {
                    src.template keys<DK>(a, k_s + slot * Cfg::kSlotK, g, lw, lane, j0, n);
                } else {
                    src.template values<DV>(a, v_s + slot * Cfg::kSlotV, g, lw, lane, j0, n);
                    src.template values<DV>(a, v_s + slot * Cfg::kSlotV, g, lw + 1, lane, j0, n);
                }
            }
            lm_cp_commit();
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            hand_over(t);
        }
        lm_cp_wait_all();
        if (!*(volatile int *)abort_flag) hand_over(n_tiles);
    } else if (lane == 0) {
        /* ---- MMA issuer ---- */
        const int k_steps = (a.dim + 15) / 16;
        const uint32_t idesc_s = at_idesc(kAtKeys, false), idesc_o = at_idesc((a.vdim + 15) & ~15, true);
        /* descriptors once: the one issuing thread has 32 to 64 clocks per MMA (addresses stay below 2^18, so sums carry
         * into nothing else) */
        const AtDesc k_desc(umma_desc_k_sw128(k_s)), q_desc(umma_desc_k_sw128(ql_s)), v_desc(at_desc_mn(vb_smem_u32(v_s)));
        bool ok = vb_mbar_wait(q_full, 0u, abort_flag);
        tc_fence_after();
        auto scores = [&](int t) {
            const int slot = t % Cfg::kSlots;
            if (!vb_mbar_wait(&k_full[slot], (uint32_t)(t / Cfg::kSlots) & 1u, abort_flag)) return false;
            tc_fence_after();
            const AtDesc kd = k_desc.at(slot * (Cfg::kSlotK >> 4));
            const uint32_t d = tmem + (uint32_t)((t & 1) * kAtKeys);
#pragma unroll
            for (int ks = 0; ks < DK * 4; ks++) {
                if (ks >= k_steps) break;
                const AtDesc hi = kd.at((ks >> 2) * (kAtBlock >> 4) + 2 * (ks & 3)), lo = hi.at(DK * (kAtBlock >> 4));
                const uint32_t qh = tmem + kAtQ + (uint32_t)(ks * 8);
                at_mma_ts(d, qh, hi, idesc_s, ks != 0 ? 1u : 0u);
                at_mma_ts(d, qh, lo, idesc_s, 1u);
                if constexpr (Cfg::kQlTmem) at_mma_ts(d, qh + DK * 32, hi, idesc_s, 1u);
                else at_mma_ss(d, q_desc.at((ks >> 2) * (kAtRows * 128 >> 4) + 2 * (ks & 3)), hi, idesc_s, 1u);
            }
            umma_commit(&k_empty[slot]);
            umma_commit(&s_full[t & 1]);
            return true;
        };
        ok = ok && n_tiles > 0 && scores(0);
        if (ok && n_tiles > 1) ok = scores(1);
        for (int t = 0; t < n_tiles && ok; t++) {
            const int w = t & 1, slot = t % Cfg::kSlots;
            ok = vb_mbar_wait(&v_full[slot], (uint32_t)(t / Cfg::kSlots) & 1u, abort_flag) &&
                 vb_mbar_wait(&p_full[w], (uint32_t)(t >> 1) & 1u, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const AtDesc vd = v_desc.at(slot * (Cfg::kSlotV >> 4));
            const uint32_t d = tmem + kAtO + (uint32_t)(w * 128);
#pragma unroll
            for (int ks = 0; ks < kAtKeys / 16; ks++) {
                const AtDesc hi = vd.at(ks * (2048 >> 4)), lo = hi.at(DV * (kAtBlock >> 4));
                const uint32_t ph = tmem + (uint32_t)(w * kAtKeys + (ks >> 1) * 32 + (ks & 1) * 8);
                at_mma_ts(d, ph, hi, idesc_o, (t >> 1 | ks) != 0 ? 1u : 0u);
                at_mma_ts(d, ph, lo, idesc_o, 1u);
                at_mma_ts(d, ph + 16, hi, idesc_o, 1u);
            }
            umma_commit(&v_empty[slot]);
            umma_commit(&o_done[w]);
            /* takes the columns of P once the products above have read them: MMAs of one thread run in order */
            if (t + 2 < n_tiles) ok = scores(t + 2);
        }
        if (!ok) give_up();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kAtMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAtTmemCols) : "memory");
    }
}

template <int DK, int DV, class SRC>
int launch_attn_tc(const AtArgs &a, const SRC &src, cudaStream_t st, const AtMaps &maps = AtMaps(), int prompts = 1) {
    using Cfg = AtCfg<DK, DV>;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(vb_attn_tc_kernel<DK, DV, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        attr = true;
    }
    const int tiles = (int)(((long long)a.M * (a.heads / a.kv_heads) + kAtRows - 1) / kAtRows);
    return launch_pdl(vb_attn_tc_kernel<DK, DV, SRC>, dim3(a.kv_heads, tiles, prompts), dim3(kAtThreads), (size_t)Cfg::kSmem, st, maps, a, src) == cudaSuccess
               ? 0
               : -1;
}

} // namespace vb

#endif
