/*
 * vb_prefill.cu - multi-token prefill of the decoder on the GPU
 * (tts_llm_prefill, voxtral_tts_llm.c:277-373): all prompt rows go through the
 * 26 layers, K and V of every row land in the cache, hidden states are dropped.
 *
 * The linears run on the tensor-core GEMM (vb_tc.cu; fp32 rows as three BF16 terms) in
 * blocks of up to 256 rows; RoPE, the cache write and the causal attention use the
 * stand-alone kernels. When the tensor maps cannot be made the same layer loop runs
 * on the streaming engine, eight rows at a time. Also here: the prompt assembled on
 * the device from token ids and BF16 voice rows (voxtral_tts.c:230-272).
 */
#include "vb_attn_tc.cuh"
#include "vb_common.cuh"
#include "vb_model.cuh"
#include "vb_simple.cuh"
#include "vb_tc.cuh"

#include <math.h>
#include <stdio.h>
#include <string.h>
#include <vector>

namespace vb {

static const int D = VB200_DIM, QD = VB200_Q_DIM, KVD = VB200_KV_DIM, HID = VB200_HIDDEN;
static const int QKV = QD + 2 * KVD;

/* Runs `op` once per block of up to 8 rows; blocks are independent, so a launch
 * carries up to 64 of them without grid barriers in between. */
static int run_row_blocks(VbOp proto, int M, int x_ld, int y_ld, bool res_is_y) {
    std::vector<VbOp> ops;
    const float *x0 = proto.x;
    float *y0 = proto.y;
    for (int r = 0; r < M; r += kMaxM) {
        VbOp o = proto;
        o.M = (M - r < kMaxM) ? M - r : kMaxM;
        o.x = x0 + (size_t)r * x_ld;
        o.y = y0 + (size_t)r * y_ld;
        if (res_is_y) o.res = o.y;
        o.flags |= VB_F_NOSYNC;
        ops.push_back(o);
        if (ops.size() == 64) {
            if (run_ops(ops)) return -1;
            ops.clear();
        }
    }
    if (!ops.empty() && run_ops(ops)) return -1;
    return 0;
}

/* ---- glue kernels of the tensor-core prefill ---- */

/* QKV of a row block: sums the split-K partials in fixed order, rotates the q and k heads
 * (interleaved pairs, voxtral_tts_kernels.c:616-634), leaves q in `qkv` for the attention
 * and writes k and v straight into the cache rows (voxtral_tts_llm.c:318-330). One thread per
 * pair of columns. */
__global__ void pf_qkv_finish_kernel(float *qkv, const float *part, int n_part, size_t part_stride, const float *cs,
                                     float *k_rows, float *v_rows, int rows) {
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.y;
    const int col = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (col >= QKV || m >= rows) return;
    float2 v = make_float2(0.0f, 0.0f);
    for (int p = 0; p < n_part; p++) {
        const float2 t = __ldcg(reinterpret_cast<const float2 *>(part + (size_t)p * part_stride + (size_t)m * QKV + col));
        v.x += t.x; v.y += t.y;
    }
    if (col < QD + KVD) {
        const int d = (col % VB200_HEAD_DIM) >> 1;
        const float2 t = *reinterpret_cast<const float2 *>(cs + ((size_t)m * (VB200_HEAD_DIM / 2) + d) * 2);
        const float a = v.x, b = v.y;
        v.x = a * t.x - b * t.y;
        v.y = a * t.y + b * t.x;
    }
    if (col < QD) *reinterpret_cast<float2 *>(qkv + (size_t)m * QKV + col) = v;
    else if (col < QD + KVD) *reinterpret_cast<float2 *>(k_rows + (size_t)m * KVD + (col - QD)) = v;
    else *reinterpret_cast<float2 *>(v_rows + (size_t)m * KVD + (col - QD - KVD)) = v;
}

/* Causal attention of prompt rows over the cache prefix (tts_causal_attention, voxtral_tts_kernels.c:403-465) on the
 * tensor cores (vb_attn_tc.cuh): queries, and the cache's fp32 keys and values, which the loading warps split into BF16
 * halves on the way to shared memory. */
struct AtRows {
    static constexpr bool kAsync = false;
    const float *q, *kc, *vc;
    float *out;
    int ldq, ldkv, ldo, start_pos;
    VB_DEVINL void start() {}
    VB_DEVINL int pos0() const { return start_pos; }
    VB_DEVINL void q8(int row, int head, int d, float (&e)[8]) const {
        const float4 *p = reinterpret_cast<const float4 *>(q + (size_t)row * ldq + head * VB200_HEAD_DIM + d);
        const float4 x = p[0], y = p[1];
        e[0] = x.x; e[1] = x.y; e[2] = x.z; e[3] = x.w; e[4] = y.x; e[5] = y.y; e[6] = y.z; e[7] = y.w;
    }
    /* a lane's four columns of 16 rows, eight loads in flight; rows beyond the tile's keys are zeros */
    VB_DEVINL void rows(const float *cache, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        unsigned char *block = slot + (lane >> 4) * kAtBlock;
        const float *col = cache + (size_t)(j0 + lw * 16) * ldkv + g * VB200_HEAD_DIM + lane * 4;
#pragma unroll
        for (int x0 = 0; x0 < 16; x0 += 8) {
            float4 v[8];
#pragma unroll
            for (int x = 0; x < 8; x++)
                v[x] = lw * 16 + x0 + x < n ? vb_ldcg4(col + (size_t)(x0 + x) * ldkv) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int x = 0; x < 8; x++) {
                uint2 hi, lo;
                at_split2(v[x].x, v[x].y, hi.x, lo.x);
                at_split2(v[x].z, v[x].w, hi.y, lo.y);
                unsigned char *at = block + at_off(lw * 16 + x0 + x, (lane & 15) >> 1) + (lane & 1) * 8;
                *reinterpret_cast<uint2 *>(at) = hi;
                *reinterpret_cast<uint2 *>(at + 2 * kAtBlock) = lo;
            }
        }
    }
    template <int BLOCKS>
    VB_DEVINL void keys(const AtArgs &, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        rows(kc, slot, g, lw, lane, j0, n);
    }
    template <int BLOCKS>
    VB_DEVINL void values(const AtArgs &, unsigned char *slot, int g, int lw, int lane, int j0, int n) const {
        rows(vc, slot, g, lw, lane, j0, n);
    }
    VB_DEVINL float gate(int, int) const { return 1.0f; }
    VB_DEVINL void put4(int row, int c, const float (&e)[4]) const {
        *reinterpret_cast<float4 *>(out + (size_t)row * ldo + c) = make_float4(e[0], e[1], e[2], e[3]);
    }
};
static_assert(VB200_HEAD_DIM == 128, "a lane's four columns cover a head");

/* ---- tensor-core prefill ---- */
struct PrefillTc {
    bool ready = false;
    /* the decoder's tile-contiguous matrices (shared with the frame graph), fetched per call */
    const TcWeight *wqkv = nullptr, *wo = nullptr, *w13 = nullptr, *w2 = nullptr;
    uint16_t *bD = nullptr, *bQ = nullptr, *bH = nullptr;
    float *part = nullptr, *ssq = nullptr;
    TcActs aD[3], aQ[3], aH[3];   /* for 16, 64 and 256 padded rows, over the same buffers */
    /* row buffers of a prefill call, kept between calls and only ever grown (allocating and
     * freeing them per call cost up to 10 ms of a 7.6 ms prefill) */
    float *x = nullptr, *qkv = nullptr, *attn = nullptr, *h = nullptr, *cs = nullptr;
    int cap_rows = 0;
};
static PrefillTc g_pf;

/* Called when the device context goes away: everything here pointed into it. */
void prefill_free_all() {
    PrefillTc &t = g_pf;
    cudaFree(t.x); cudaFree(t.qkv); cudaFree(t.attn); cudaFree(t.h); cudaFree(t.cs);
    t = PrefillTc();
}

static int prefill_rows(int M) {
    PrefillTc &t = g_pf;
    if (M <= t.cap_rows) return 0;
    cudaFree(t.x); cudaFree(t.qkv); cudaFree(t.attn); cudaFree(t.h); cudaFree(t.cs);
    t.x = t.qkv = t.attn = t.h = t.cs = nullptr;
    t.cap_rows = 0;
    const int cap = (M + 255) / 256 * 256;
    if (cudaMalloc((void **)&t.x, (size_t)cap * D * 4) != cudaSuccess || cudaMalloc((void **)&t.qkv, (size_t)cap * QKV * 4) != cudaSuccess ||
        cudaMalloc((void **)&t.attn, (size_t)cap * QD * 4) != cudaSuccess || cudaMalloc((void **)&t.h, (size_t)cap * HID * 4) != cudaSuccess ||
        cudaMalloc((void **)&t.cs, (size_t)cap * VB200_HEAD_DIM * 4) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(t.x); cudaFree(t.qkv); cudaFree(t.attn); cudaFree(t.h); cudaFree(t.cs);
        t.x = t.qkv = t.attn = t.h = t.cs = nullptr;
        return -1;
    }
    t.cap_rows = cap;
    return 0;
}
static const int kPfRows = 256;

static int pf_slot(int rows_pad) { return rows_pad == 16 ? 0 : rows_pad == 64 ? 1 : 2; }

/* The activation-term buffers and their tensor maps; called after the decoder upload. Failing here is not fatal: prefill() then uses the streaming kernel. */
int prefill_tc_setup() {
    Model &m = model();
    PrefillTc &t = g_pf;
    t.ready = false;
    if (getenv("VB200_NO_TC") || tc_init()) return 0;
    if (!t.bD) {
        void *p[5] = {};
        const size_t sz[5] = {tc_acts_bytes(kPfRows, D), tc_acts_bytes(kPfRows, QD), tc_acts_bytes(kPfRows, HID),
                              sizeof(float) * (size_t)kTcMaxSplits * kPfRows * QKV, sizeof(float) * kPfRows * 16};
        for (int i = 0; i < 5; i++) {
            if (cudaMalloc(&p[i], sz[i]) != cudaSuccess) return 0;
            m.allocs.push_back(p[i]);
            cudaMemset(p[i], 0, sz[i]);
        }
        t.bD = (uint16_t *)p[0]; t.bQ = (uint16_t *)p[1]; t.bH = (uint16_t *)p[2];
        t.part = (float *)p[3]; t.ssq = (float *)p[4];
    }
    const int pads[3] = {16, 64, 256};
    for (int i = 0; i < 3; i++)
        if (tc_acts(&t.aD[i], t.bD, pads[i], D) || tc_acts(&t.aQ[i], t.bQ, pads[i], QD) ||
            tc_acts(&t.aH[i], t.bH, pads[i], HID))
            return 0;
    t.ready = true;
    return 0;
}

/* Prefill with the tcgen05 GEMM (vb_tc.cu): per layer and per block of up to 256 rows
 * gain+terms -> QKV -> RoPE -> cache rows; causal attention over the whole cache prefix;
 * terms -> O -> residual+gain+terms -> gate/up with SwiGLU -> down -> residual. */
static int prefill_tc(float *x, float *qkv, float *attn, const float *cs, int M, int start_pos) {
    Model &m = model();
    PrefillTc &t = g_pf;
    cudaStream_t st = m.st;
    const float scale = 1.0f / sqrtf((float)VB200_HEAD_DIM);
    const int s_qkv = tc_pick_splits(QKV, D, m.sm_count), s_wo = tc_pick_splits(D, QD, m.sm_count),
              s_w2 = tc_pick_splits(D, HID, m.sm_count);
    const int chunksD = tc_prepare_chunks(D);
    for (int l = 0; l < VB200_DEC_LAYERS; l++) {
        const LayerDev &L = m.dec[l];
        for (int r0 = 0; r0 < M; r0 += kPfRows) {
            const int rows = M - r0 < kPfRows ? M - r0 : kPfRows;
            const int slot = pf_slot(tc_rows_pad(rows));
            float *xr = x + (size_t)r0 * D, *qr = qkv + (size_t)r0 * QKV;
            tc_prepare(t.aD[slot], xr, D, rows, nullptr, 0, 0, nullptr, nullptr, L.attn_norm, t.ssq, st);
            TcGemm g;
            g.M = rows; g.status = &m.d_out->status; g.epi = TC_EPI_PARTIAL; g.out = t.part; g.ld_out = QKV;
            g.splits = s_qkv; g.ssq = t.ssq; g.ssq_chunks = chunksD; g.eps = VB200_NORM_EPS;
            if (tc_gemm(t.wqkv[l], t.aD[slot], g, st)) return -1;
            float *ck = m.kv_k + ((size_t)l * m.kv_max + start_pos + r0) * KVD;
            float *cv = m.kv_v + ((size_t)l * m.kv_max + start_pos + r0) * KVD;
            launch_pdl(pf_qkv_finish_kernel, dim3(QKV / 2 / 256, rows), dim3(256), 0, st, qr, (const float *)t.part, s_qkv,
                       (size_t)rows * QKV, cs + (size_t)r0 * VB200_HEAD_DIM, ck, cv, rows);
        }
        const float *k0 = m.kv_k + (size_t)l * m.kv_max * KVD, *v0 = m.kv_v + (size_t)l * m.kv_max * KVD;
        const AtRows rows_of = {qkv, k0, v0, attn, QKV, KVD, QD, start_pos};
        const AtArgs at = {M, VB200_HEADS, VB200_KV_HEADS, VB200_HEAD_DIM, VB200_HEAD_DIM, 0, 0, scale, 0.0f, &m.d_out->status};
        if (launch_attn_tc<2, 2>(at, rows_of, st)) return -1;
        if (l == VB200_DEC_LAYERS - 1) break;   /* only the cache is kept (voxtral_tts_llm.c:281) */
        for (int r0 = 0; r0 < M; r0 += kPfRows) {
            const int rows = M - r0 < kPfRows ? M - r0 : kPfRows;
            const int rp = tc_rows_pad(rows), slot = pf_slot(rp);
            float *xr = x + (size_t)r0 * D;
            const size_t psD = (size_t)rows * D;
            tc_prepare(t.aQ[slot], attn + (size_t)r0 * QD, QD, rows, nullptr, 0, 0, nullptr, nullptr, nullptr, nullptr, st);
            TcGemm g;
            g.M = rows; g.status = &m.d_out->status; g.epi = TC_EPI_PARTIAL; g.out = t.part; g.ld_out = D;
            g.splits = s_wo;
            if (tc_gemm(t.wo[l], t.aQ[slot], g, st)) return -1;
            tc_prepare(t.aD[slot], nullptr, D, rows, t.part, s_wo, psD, xr, xr, L.ffn_norm, t.ssq, st);
            g.epi = TC_EPI_SWIGLU_TERMS; g.out = nullptr; g.out_terms = t.bH; g.out_rows_pad = rp; g.splits = 1;
            g.ld_out = HID; g.ssq = t.ssq; g.ssq_chunks = chunksD; g.eps = VB200_NORM_EPS;
            if (tc_gemm(t.w13[l], t.aD[slot], g, st)) return -1;
            g.epi = TC_EPI_PARTIAL; g.out = t.part; g.out_terms = nullptr; g.splits = s_w2; g.ld_out = D;
            g.ssq = nullptr; g.ssq_chunks = 0;
            if (tc_gemm(t.w2[l], t.aH[slot], g, st)) return -1;
            /* residual add (the terms it also writes are overwritten by the next layer's prepare) */
            tc_prepare(t.aD[slot], nullptr, D, rows, t.part, s_w2, psD, xr, xr, nullptr, nullptr, st);
        }
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int prefill(const float *embeds, int seq_len, int start_pos) {
    Model &m = model();
    if (!m.inited || !m.llm_ready) return -1;
    if (seq_len <= 0) return 0;
    if (start_pos < 0 || start_pos + seq_len > m.kv_max) {
        fprintf(stderr, "voxtral_b200: prefill of %d rows at %d exceeds the %d-row cache\n", seq_len, start_pos,
                m.kv_max);
        return -1;
    }
    const int M = seq_len;
    if (prefill_rows(M)) return -1;
    float *x = g_pf.x, *qkv = g_pf.qkv, *attn = g_pf.attn, *h = g_pf.h, *cs = g_pf.cs;
    int rc = 0;
    const float scale = 1.0f / sqrtf((float)VB200_HEAD_DIM);
    if (!rc && cudaMemcpyAsync(x, embeds, (size_t)M * D * 4, cudaMemcpyDefault, m.st) != cudaSuccess) rc = -1;
    if (!rc) rope_table(cs, start_pos, M, VB200_HEAD_DIM, VB200_ROPE_THETA, m.st);

    if (!rc && g_pf.ready && batch_tiled_decoder(&g_pf.wqkv, &g_pf.wo, &g_pf.w13, &g_pf.w2) == 0) {
        rc = prefill_tc(x, qkv, attn, cs, M, start_pos);
        if (cudaStreamSynchronize(m.st) != cudaSuccess) rc = -1;
        if (!rc) {
            int status = 0;
            cudaMemcpy(&status, &m.d_out->status, sizeof(int), cudaMemcpyDeviceToHost);
            m.last_status = status;
            if (status) {
                /* the word is sticky on the device (kernels only set it from 0): clear it so the
                 * next call starts clean */
                cudaMemset(&m.d_out->status, 0, sizeof(int));
                rc = -1;
            }
        }
        return rc;
    }
    for (int l = 0; l < VB200_DEC_LAYERS && !rc; l++) {
        const LayerDev &L = m.dec[l];
        float *ck = m.kv_k + ((size_t)l * m.kv_max + start_pos) * KVD;
        float *cv = m.kv_v + ((size_t)l * m.kv_max + start_pos) * KVD;

        VbOp o;
        memset(&o, 0, sizeof(o));
        o.type = VB_OP_GEMV; o.N = QKV; o.K = D; o.W = L.wqkv; o.x = x; o.ldx = D; o.y = qkv; o.ldy = QKV;
        o.epi = VB_EPI_STORE; o.norm_w = L.attn_norm; o.eps = VB200_NORM_EPS;
        rc = run_row_blocks(o, M, D, QKV, false);
        if (rc) break;

        rope_apply(qkv, cs, M, VB200_HEADS, VB200_HEAD_DIM, QKV, m.st);
        rope_apply(qkv + QD, cs, M, VB200_KV_HEADS, VB200_HEAD_DIM, QKV, m.st);
        if (cudaMemcpy2DAsync(ck, (size_t)KVD * 4, qkv + QD, (size_t)QKV * 4, (size_t)KVD * 4, M,
                              cudaMemcpyDeviceToDevice, m.st) != cudaSuccess ||
            cudaMemcpy2DAsync(cv, (size_t)KVD * 4, qkv + QD + KVD, (size_t)QKV * 4, (size_t)KVD * 4, M,
                              cudaMemcpyDeviceToDevice, m.st) != cudaSuccess) {
            rc = -1;
            break;
        }
        const float *k0 = m.kv_k + (size_t)l * m.kv_max * KVD;
        const float *v0 = m.kv_v + (size_t)l * m.kv_max * KVD;
        if (attention_rows(attn, qkv, k0, v0, M, start_pos + M, VB200_HEADS, VB200_KV_HEADS, VB200_HEAD_DIM,
                           scale, start_pos, 1, QKV, KVD, QD, m.st)) {
            rc = -1;
            break;
        }

        memset(&o, 0, sizeof(o));
        o.type = VB_OP_GEMV; o.N = D; o.K = QD; o.W = L.wo; o.x = attn; o.ldx = QD; o.y = x; o.ldy = D;
        o.epi = VB_EPI_ADD; o.eps = VB200_NORM_EPS;
        rc = run_row_blocks(o, M, QD, D, true);
        if (rc) break;

        memset(&o, 0, sizeof(o));
        o.type = VB_OP_GEMV; o.N = 2 * HID; o.K = D; o.W = L.w13; o.x = x; o.ldx = D; o.y = h; o.ldy = HID;
        o.epi = VB_EPI_SWIGLU; o.norm_w = L.ffn_norm; o.eps = VB200_NORM_EPS;
        rc = run_row_blocks(o, M, D, HID, false);
        if (rc) break;

        memset(&o, 0, sizeof(o));
        o.type = VB_OP_GEMV; o.N = D; o.K = HID; o.W = L.w2; o.x = h; o.ldx = HID; o.y = x; o.ldy = D;
        o.epi = VB_EPI_ADD; o.eps = VB200_NORM_EPS;
        rc = run_row_blocks(o, M, HID, D, true);
    }
    if (cudaStreamSynchronize(m.st) != cudaSuccess) rc = -1;
    if (!rc) {
        int status = 0;
        cudaMemcpy(&status, &m.d_out->status, sizeof(int), cudaMemcpyDeviceToHost);
        m.last_status = status;
        if (status) {
            cudaMemset(&m.d_out->status, 0, sizeof(int));
            cudaMemset(m.bar, 0, 16 * sizeof(unsigned));
            cudaMemset(m.exitc, 0, 16 * sizeof(unsigned));
            rc = -1;
        }
    }
    return rc;
}

/* ---- the prompt, assembled on the device ---- */
/* Row r of the prompt: a token-table row (ids[r] >= 0) or voice row -ids[r] - 1, BF16 -> fp32
 * (tts_embed_token_bf16, voxtral_tts_kernels.c:55-59; tts_voice_embed, voxtral_tts_voice.c:228-248). */
__global__ void prompt_rows_kernel(float *out, const uint16_t *table, const uint16_t *voice, const int *ids, int dim) {
    const int id = ids[blockIdx.y];
    const uint16_t *src = id >= 0 ? table + (size_t)id * dim : voice + (size_t)(-id - 1) * dim;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < dim) out[(size_t)blockIdx.y * dim + i] = __uint_as_float((uint32_t)src[i] << 16);
}

/* The prompt the orchestrator assembles on the host (voxtral_tts.c:230-272):
 *   [BOS=1] [BEGIN_AUDIO=25] voice rows [/INST=36] text tokens [INST=35] [BEGIN_AUDIO=25]
 * built on the device from the token table uploaded with the decoder weights and the BF16 voice
 * rows (host memory, [n_voice, 3072]), then prefilled from cache row start_pos. Only the token ids
 * and the BF16 voice rows cross PCIe (1.4 MB for 224 voice rows instead of 3 MB of fp32 rows, and
 * no BF16 -> fp32 pass on the host). Returns the number of prompt rows, or -1. */
int prefill_prompt(const int *text_ids, int n_text, const uint16_t *voice_bf16, int n_voice, int start_pos) {
    Model &m = model();
    if (!m.inited || !m.llm_ready || !m.tok_emb) {
        fprintf(stderr, "voxtral_b200: the prompt needs the decoder weights with the token table uploaded\n");
        return -1;
    }
    if (n_text < 0 || n_voice < 0 || (n_text > 0 && !text_ids) || (n_voice > 0 && !voice_bf16)) return -1;
    const int n = n_voice + n_text + 5;
    if (start_pos < 0 || start_pos + n > m.kv_max) {
        fprintf(stderr, "voxtral_b200: a prompt of %d rows at %d exceeds the %d-row cache\n", n, start_pos, m.kv_max);
        return -1;
    }
    std::vector<int> ids;
    ids.reserve(n);
    ids.push_back(1);
    ids.push_back(25);
    for (int i = 0; i < n_voice; i++) ids.push_back(-(i + 1));
    ids.push_back(36);
    for (int i = 0; i < n_text; i++) {
        if (text_ids[i] < 0 || text_ids[i] >= VB200_VOCAB) return -1;
        ids.push_back(text_ids[i]);
    }
    ids.push_back(35);
    ids.push_back(25);
    int *d_ids = nullptr;
    uint16_t *d_voice = nullptr;
    float *d_rows = nullptr;
    int rc = -1;
    do {
        if (cudaMalloc(&d_ids, sizeof(int) * n) != cudaSuccess || cudaMalloc(&d_rows, sizeof(float) * (size_t)n * D) != cudaSuccess)
            break;
        if (n_voice > 0 && cudaMalloc(&d_voice, (size_t)n_voice * D * 2) != cudaSuccess) break;
        if (cudaMemcpyAsync(d_ids, ids.data(), sizeof(int) * n, cudaMemcpyHostToDevice, m.st) != cudaSuccess) break;
        if (n_voice > 0 &&
            cudaMemcpyAsync(d_voice, voice_bf16, (size_t)n_voice * D * 2, cudaMemcpyHostToDevice, m.st) != cudaSuccess)
            break;
        prompt_rows_kernel<<<dim3((D + 255) / 256, n), 256, 0, m.st>>>(d_rows, m.tok_emb, d_voice, d_ids, D);
        if (cudaGetLastError() != cudaSuccess) break;
        rc = prefill(d_rows, n, start_pos) == 0 ? n : -1;    /* synchronises the stream */
    } while (0);
    cudaStreamSynchronize(m.st);
    cudaFree(d_ids); cudaFree(d_voice); cudaFree(d_rows);
    cudaGetLastError();
    return rc;
}

} // namespace vb

