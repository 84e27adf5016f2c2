/*
 * vb_common.cuh - sm_100a PTX wrappers shared by the kernels: mbarriers, 1-D bulk
 * (TMA) copies into shared memory, scoped atomics for the grid barrier, and
 * bounded waits. Every wait in this library has a deadline; a wait that runs out
 * records a status code and lets the kernel return instead of hanging the GPU.
 */
#ifndef VB_COMMON_CUH
#define VB_COMMON_CUH

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define VB_DEVINL __device__ __forceinline__

/* ~1 s at 1.9 GHz: far beyond any legitimate wait in a millisecond-scale kernel. */
#define VB_WAIT_CYCLES (2000000000LL)

VB_DEVINL uint32_t vb_smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

VB_DEVINL void vb_mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(vb_smem_u32(bar)), "r"(count));
}

VB_DEVINL void vb_mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

VB_DEVINL void vb_mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(vb_smem_u32(bar)) : "memory");
}

VB_DEVINL void vb_mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(vb_smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

VB_DEVINL bool vb_mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(vb_smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* Waits for the phase with the given parity to complete. Returns false when the
 * deadline passes or another thread of the CTA has already given up. */
VB_DEVINL bool vb_mbar_wait(uint64_t *bar, uint32_t parity, volatile int *cta_abort) {
    if (vb_mbar_try_wait(bar, parity)) return true;
    long long t0 = clock64();
    while (true) {
        if (vb_mbar_try_wait(bar, parity)) return true;
        if (*cta_abort) return false;
        if (clock64() - t0 > VB_WAIT_CYCLES) return false;
    }
}

/* The same for what the CTAs of a cluster send into one another's shared memory, called by all threads of a CTA after it has sent its
 * own. A CTA ends only when it has received everything. Where the wait runs out it reports that and stays for as long
 * again: a sender held up by a bounded wait of its own, begun with the cluster, is done before that, and what it sends meets
 * memory that is still there. */
VB_DEVINL bool vb_mbar_wait_cluster(uint64_t *bar, volatile int *cta_abort, int *status, int code) {
    if (vb_mbar_wait(bar, 0u, cta_abort)) return true;
    atomicCAS(status, 0, code);
    *cta_abort = 1;
    volatile int stay = 0;
    vb_mbar_wait(bar, 0u, &stay);
    return false;
}

/* Two packed floats per instruction. */
VB_DEVINL uint64_t vb_f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
VB_DEVINL float2 vb_f2_get(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
VB_DEVINL uint64_t vb_f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
VB_DEVINL uint64_t vb_f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
VB_DEVINL uint64_t vb_f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

/* 32 sums over the lanes of a warp by halving: lane i is left with sum i, in s[0]. */
VB_DEVINL void vb_warp_halve32(float (&s)[32], int lane) {
#pragma unroll
    for (int n = 16; n > 0; n >>= 1) {
        const bool up = (lane & n) != 0;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float send = up ? s[i] : s[i + n], keep = up ? s[i + n] : s[i];
            s[i] = keep + __shfl_xor_sync(0xffffffffu, send, n);
        }
    }
}

/* 16 bytes to the same place in the shared memory of the cluster's CTA `rank`, counted on its barrier. */
VB_DEVINL void vb_cluster_send(const void *place, const uint64_t *bar, int rank, float a, float b, float c, float d) {
    uint32_t to, count;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(vb_smem_u32(place)), "r"(rank));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(count) : "r"(vb_smem_u32(bar)), "r"(rank));
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
                 "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d)), "r"(count)
                 : "memory");
}

/* 1-D bulk copy global -> shared, completion counted in bytes on an mbarrier.
 * Both addresses 16-byte aligned, size a multiple of 16. No multicast. */
VB_DEVINL void vb_bulk_g2s(void *smem_dst, const void *gmem_src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            vb_smem_u32(smem_dst)),
        "l"(gmem_src), "r"(bytes), "r"(vb_smem_u32(bar))
        : "memory");
}

/* Pulls a global range into L2 without a destination (16-byte aligned, size a
 * multiple of 16). */
VB_DEVINL void vb_prefetch_l2(const void *gmem_src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(gmem_src), "r"(bytes) : "memory");
}

VB_DEVINL void vb_named_bar(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

VB_DEVINL unsigned vb_atomic_add_release_gpu(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

VB_DEVINL unsigned vb_atomic_add_acq_rel_gpu(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

VB_DEVINL unsigned vb_ld_acquire_gpu(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

/* System scope: words that another GPU writes or reads over NVLink (tensor-parallel flags). */
VB_DEVINL unsigned vb_ld_acquire_sys(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
VB_DEVINL void vb_st_release_sys(unsigned *p, unsigned v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

VB_DEVINL int vb_ld_relaxed_gpu_s32(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

/* Activations are produced by other SMs earlier in the same launch: read them
 * from L2, never through a possibly stale L1 line or the read-only path. */
VB_DEVINL float vb_ldcg(const float *p) { return __ldcg(p); }
VB_DEVINL float4 vb_ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }

VB_DEVINL float vb_bf16_lo(uint32_t packed) { return __uint_as_float(packed << 16); }
VB_DEVINL float vb_bf16_hi(uint32_t packed) { return __uint_as_float(packed & 0xffff0000u); }

VB_DEVINL float vb_warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

/* Sums V per-lane values over the 32 lanes with the halving butterfly: at each
 * step a lane keeps half of its values and hands the other half to its partner,
 * so the total is about V + 5 shuffles instead of 5 * V. On return v[0] holds the
 * complete sum of value `index` (returned); lanes whose index is >= V hold
 * nothing useful. */
template <int V>
VB_DEVINL int vb_warp_multi_sum(float (&v)[V], int lane) {
    int base = 0;
    int count = V;    /* slots per lane, padding included (same on every lane) */
    int real = V;     /* how many of this lane's slots carry actual values */
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (count > 1) {
            const int half = (count + 1) >> 1;
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < (V + 1) / 2; i++) {
                if (i < half) {
                    float hi = (i + half < count) ? v[i + half] : 0.0f;
                    float send = up ? v[i] : hi;
                    float keep = up ? hi : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            if (up) { base += half; real = real > half ? real - half : 0; }
            else real = real < half ? real : half;
            count = half;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    /* a lane that ended on a padding slot (odd counts on the way) owns no value */
    return real > 0 ? base : V;
}

/* Programmatic dependent launch: launch_dependents lets the next kernel of the stream begin
 * its prologue; wait blocks until the previous kernel has completed and its writes are visible
 * (a no-op for kernels launched without the attribute). */
VB_DEVINL void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
VB_DEVINL void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

/* v = t0 + t1 + t2 with three BF16 terms (8 + 8 + 8 mantissa bits): what the tensor-core
 * path feeds instead of an fp32 activation. */
VB_DEVINL void vb_split3(float v, uint16_t &t0, uint16_t &t1, uint16_t &t2) {
    const __nv_bfloat16 h0 = __float2bfloat16_rn(v);
    const float r1 = v - __bfloat162float(h0);
    const __nv_bfloat16 h1 = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(h1);
    const __nv_bfloat16 h2 = __float2bfloat16_rn(r2);
    t0 = __bfloat16_as_ushort(h0);
    t1 = __bfloat16_as_ushort(h1);
    t2 = __bfloat16_as_ushort(h2);
}

/* Two values at once, the first in the low halves: the same terms in half the conversions. */
VB_DEVINL void vb_split3_pair(float a, float b, uint32_t &t0, uint32_t &t1, uint32_t &t2) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t0) : "f"(b), "f"(a));
    a -= __uint_as_float(t0 << 16);
    b -= __uint_as_float(t0 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t1) : "f"(b), "f"(a));
    a -= __uint_as_float(t1 << 16);
    b -= __uint_as_float(t1 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t2) : "f"(b), "f"(a));
}
/* The same where a value may be infinite: its low terms are zeros, not NaN. */
VB_DEVINL void vb_split3_inf(float v, uint16_t &t0, uint16_t &t1, uint16_t &t2) {
    vb_split3(v, t0, t1, t2);
    if ((t0 & 0x7fffu) == 0x7f80u) t1 = t2 = 0;
}
/* From here on a value is infinite once rounded to BF16 (halfway between its largest number and 2^128). */
constexpr float kBf16Inf = 0x1.FFp127f;
VB_DEVINL void vb_split3_pair_inf(float a, float b, uint32_t &t1, uint32_t &t2) {
    const uint32_t keep = (fabsf(a) >= kBf16Inf ? 0u : 0xffffu) | (fabsf(b) >= kBf16Inf ? 0u : 0xffff0000u);
    t1 &= keep;
    t2 &= keep;
}

#endif
