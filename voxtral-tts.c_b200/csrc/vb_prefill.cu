/*
 * vb_prefill.cu - multi-token prefill of the decoder on the GPU
 * (tts_llm_prefill, voxtral_tts_llm.c:277-373): all prompt rows go through the
 * 26 layers, K and V of every row land in the cache, hidden states are dropped.
 *
 * The linears run on the tensor-core GEMMs (vb_tc.cu, vb_tc_rows.cu; fp32 rows as three or two BF16 terms) in
 * blocks of rows, the causal attention on the tensor cores too (vb_attn_tc.cuh). When the tensor maps cannot be made or
 * there is no memory for a block's operands, the same layer loop runs on the streaming engine, eight rows at a time. Also here: the prompt assembled on
 * the device from token ids and BF16 voice rows (voxtral_tts.c:230-272).
 */
#include "vb_attn_tc.cuh"
#include "vb_common.cuh"
#include "vb_model.cuh"
#include "vb_simple.cuh"
#include "vb_tc.cuh"

#include <algorithm>

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

/* A layer's keys and values as BF16 halves, [row][KV head][128 high, 128 low]: what the attention reads. */
struct PfSplit {
    uint16_t *k, *v;
};
VB_DEVINL void pf_split(uint16_t *rows, size_t row, int col, float2 v) {
    uint32_t hi, lo;
    at_split2(v.x, v.y, hi, lo);
    uint32_t *at = reinterpret_cast<uint32_t *>(rows + row * 2 * KVD + (col >> 7) * 256 + (col & 127));
    at[0] = hi;
    at[64] = lo;
}
/* The cache's earlier rows. One thread per pair of columns; grid = (rows, KVD / 512): a cache has more rows than a grid's
 * y axis (65535). */
__global__ void pf_split_kernel(PfSplit to, const float *kc, const float *vc) {
    pdl_launch_dependents();
    pdl_wait();
    const int col = 2 * (blockIdx.y * blockDim.x + threadIdx.x);
    const size_t row = blockIdx.x;
    pf_split(to.k, row, col, __ldcg(reinterpret_cast<const float2 *>(kc + row * KVD + col)));
    pf_split(to.v, row, col, __ldcg(reinterpret_cast<const float2 *>(vc + row * KVD + col)));
}

/* A block of rows is a stretch of one prompt, or several short prompts side by side: their GEMMs are one, each has its own
 * cache rows, positions and split keys. */
constexpr int kPfSegs = 8;
struct PfSeg {
    int row0, rows;              /* in the block */
    int pos, cs0;                /* position of its first row, and that row's place in the rotation table */
    int key0;                    /* where its position 0 lies among the split keys: a multiple of a key tile */
    int y0;                      /* first of its rows and zero rows in pf_qkv_finish's grid */
    float *k, *v;                /* its cache, layer 0 */
    size_t layer;                /* floats from one layer of it to the next */
};
struct PfSegs {
    int n = 0, rows = 0, keys = 0, grid = 0;
    PfSeg s[kPfSegs] = {};
    void add(int rows_, int pos, int cs0, float *k, float *v, int kv_max) {
        const int end = pos + rows_, tiles = (end + kAtKeys - 1) / kAtKeys * kAtKeys;
        s[n++] = {rows, rows_, pos, cs0, keys, grid, k, v, (size_t)kv_max * KVD};
        rows += rows_;
        keys += tiles;
        grid += tiles - pos;
    }
};

/* QKV of a row block: sums the split-K partials in fixed order, rotates the q and k heads
 * (interleaved pairs, voxtral_tts_kernels.c:616-634), leaves q in `qkv` for the attention
 * and writes k and v straight into the cache rows (voxtral_tts_llm.c:318-330) and, split, for the
 * attention, whose tiles of 64 keys end in rows of zeros. One thread per pair of columns. */
__global__ void pf_qkv_finish_kernel(float *qkv, const float *part, int n_part, size_t part_stride, const float *cs, PfSplit split,
                                     const __grid_constant__ PfSegs segs, int layer) {
    pdl_launch_dependents();
    pdl_wait();
    int i = 0;
    while (i + 1 < segs.n && (int)blockIdx.y >= segs.s[i + 1].y0) i++;
    const PfSeg &g = segs.s[i];
    const int r = (int)blockIdx.y - g.y0, m = g.row0 + r, at = g.key0 + g.pos + r;
    const int col = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (col >= QKV) return;
    if (r >= g.rows) {
        if (col >= QD) pf_split(col < QD + KVD ? split.k : split.v, at, col < QD + KVD ? col - QD : col - QD - KVD, make_float2(0.0f, 0.0f));
        return;
    }
    float2 v = make_float2(0.0f, 0.0f);
    for (int p = 0; p < n_part; p++) {
        const float2 t = __ldcg(reinterpret_cast<const float2 *>(part + (size_t)p * part_stride + (size_t)m * QKV + col));
        v.x += t.x; v.y += t.y;
    }
    if (col < QD + KVD) {
        const int d = (col % VB200_HEAD_DIM) >> 1;
        const float2 t = *reinterpret_cast<const float2 *>(cs + ((size_t)(g.cs0 + r) * (VB200_HEAD_DIM / 2) + d) * 2);
        const float a = v.x, b = v.y;
        v.x = a * t.x - b * t.y;
        v.y = a * t.y + b * t.x;
    }
    const size_t row = (size_t)layer * g.layer + (size_t)(g.pos + r) * KVD;
    if (col < QD) *reinterpret_cast<float2 *>(qkv + (size_t)m * QKV + col) = v;
    else if (col < QD + KVD) {
        *reinterpret_cast<float2 *>(g.k + row + (col - QD)) = v;
        pf_split(split.k, at, col - QD, v);
    } else {
        *reinterpret_cast<float2 *>(g.v + row + (col - QD - KVD)) = v;
        pf_split(split.v, at, col - QD - KVD, v);
    }
}

/* Causal attention of prompt rows over the cache prefix (tts_causal_attention, voxtral_tts_kernels.c:403-465) on the
 * tensor cores (vb_attn_tc.cuh). */
struct AtPrompt {
    static constexpr bool kBoxes = true, kParts = false;
    const float *q;
    LmSink out;                  /* the terms that the O projection reads */
    int ldq;
    struct Seg { int row0, rows, pos, key0; } at;          /* PfSeg */
    VB_DEVINL void start() {}
    VB_DEVINL int rows(const AtArgs &) const { return at.rows; }
    VB_DEVINL int pos0() const { return at.pos; }
    VB_DEVINL float4 q4(int row, int head, int d, int) const { return vb_ldcg4(q + (size_t)(at.row0 + row) * ldq + head * VB200_HEAD_DIM + d); }
    VB_DEVINL float4 turned(int, int, int, float4 v) const { return v; }
    VB_DEVINL bool boxes(int, int) const { return true; }
    template <int BLOCKS>
    VB_DEVINL void box(const CUtensorMap *map, unsigned char *slot, int g, int j0, uint64_t *bar) const {
#pragma unroll
        for (int b = 0; b < 2 * BLOCKS; b++) at_tma(slot + b * kAtBlock, map, (g * 2 * BLOCKS + b) * 64, at.key0 + j0, 0, bar);
    }
    template <int BLOCKS>
    VB_DEVINL void tma_keys(const AtArgs &, const AtMaps &m, unsigned char *slot, int g, int j0, uint64_t *bar) const {
        box<BLOCKS>(&m.k, slot, g, j0, bar);
    }
    template <int BLOCKS>
    VB_DEVINL void tma_values(const AtArgs &, const AtMaps &m, unsigned char *slot, int g, int j0, uint64_t *bar) const {
        box<BLOCKS>(&m.v, slot, g, j0, bar);
    }
    VB_DEVINL float gate(int, int) const { return 1.0f; }
    VB_DEVINL void put4(int row, int c, const float (&e)[4]) const { lm_put4(out, at.row0 + row, c, e); }
};
/* Several prompts: blockIdx.z chooses. */
struct AtRows : AtPrompt {
    Seg s[kPfSegs];
    VB_DEVINL AtPrompt here() const {
        AtPrompt r = *this;
        r.at = s[blockIdx.z];
        return r;
    }
};
static_assert(VB200_HEAD_DIM == 128, "two blocks of 64 columns");

/* ---- tensor-core prefill ---- */
/* Rows of a prompt that go through a layer at once: 1203 rows took 33.4 ms in blocks of 256, 23.9 ms in one. */
constexpr int kPfRows = 2048;

struct PrefillTc {
    bool ready = false;
    /* the decoder's tile-contiguous matrices (shared with the frame graph), fetched per call */
    const TcWeight *wqkv = nullptr, *wo = nullptr, *w13 = nullptr, *w2 = nullptr;
    /* buffers of a call, kept between calls and only ever grown (allocating and freeing them per call cost up to
     * 10 ms of a 7.6 ms prefill): rows of the whole prompt, then of a block of it */
    float *x = nullptr, *cs = nullptr;
    float *qkv = nullptr, *part = nullptr, *ssq = nullptr;
    uint16_t *bD = nullptr, *bQ = nullptr, *bH = nullptr;
    /* without tensor maps: all rows */
    float *attn = nullptr, *h = nullptr;
    /* a prompt given as ids and voice rows */
    int *ids = nullptr;
    uint16_t *voice = nullptr;
    PfSplit split = {};          /* of one layer, whole tiles of 64 rows */
    size_t cap[14] = {};
};
static PrefillTc g_pf;

/* Called when the device context goes away: everything here pointed into it. */
void prefill_free_all() {
    PrefillTc &t = g_pf;
    for (void *p : {(void *)t.x, (void *)t.cs, (void *)t.qkv, (void *)t.part, (void *)t.ssq, (void *)t.bD, (void *)t.bQ, (void *)t.bH,
                    (void *)t.attn, (void *)t.h, (void *)t.ids, (void *)t.voice, (void *)t.split.k, (void *)t.split.v})
        cudaFree(p);
    t = PrefillTc();
}

/* Buffer i of g_pf at least that large; what it held is lost when it grows. New memory is zero: rows of the padding are
 * multiplied like any other, and have to be finite. */
template <class T>
static int pf_grow(int i, T **p, size_t bytes) {
    PrefillTc &t = g_pf;
    if (bytes <= t.cap[i]) return 0;
    cudaFree(*p);
    *p = nullptr;
    t.cap[i] = 0;
    if (cudaMalloc((void **)p, bytes) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return -1;
    }
    t.cap[i] = bytes;
    return cudaMemsetAsync(*p, 0, bytes, model().st) == cudaSuccess ? 0 : -1;
}

/* What a block of rows needs beside the rows themselves goes back. */
static void pf_release_block() {
    PrefillTc &t = g_pf;
    cudaFree(t.qkv); cudaFree(t.part); cudaFree(t.ssq); cudaFree(t.bD); cudaFree(t.bQ); cudaFree(t.bH); cudaFree(t.split.k); cudaFree(t.split.v);
    t.qkv = t.part = t.ssq = nullptr;
    t.bD = t.bQ = t.bH = nullptr;
    t.split = PfSplit();
    for (int i : {2, 3, 4, 5, 6, 7, 12, 13}) t.cap[i] = 0;
}

/* Padded rows of a block, and the K splits of its GEMMs. */
struct PfBlock {
    int rows, rp, s_qkv, s_wo, s_w2;
};
static PfBlock pf_block(int rows) {
    const int n = model().sm_count;
    PfBlock b = {rows, tc_rows_pad_any(rows), 0, 0, 0};
    if (b.rp <= 256) {           /* short sums, as in a frame's GEMMs; a GEMM of 256 rows has tiles for a sixth of the SMs */
        b.s_qkv = tc_pick_splits(QKV, D, n); b.s_wo = tc_pick_splits(D, QD, n); b.s_w2 = tc_pick_splits(D, HID, n);
    } else {
        b.s_qkv = tc_row_splits(QKV, D, rows, n); b.s_wo = tc_row_splits(D, QD, rows, n); b.s_w2 = tc_row_splits(D, HID, rows, n);
    }
    return b;
}

/* Rows of the next block when so many are left: all of them, but 1 to 64 behind a multiple of 256 go alone, for up to 64 rows
 * are multiplied as three terms (24 bits) and more as two (16). 300 rows take 6.7 ms for it, 5.0 as one block of two
 * terms; 1300 rows 18.3 and 16.4. */
static int pf_next_rows(int left, int block) {
    if (left > block) return block;
    const int tail = left % 256;
    return left > 256 && tail >= 1 && tail <= 64 ? left - tail : left;
}

static int pf_block_buffers(size_t rows, size_t pad, size_t part, size_t keys) {
    PrefillTc &t = g_pf;
    return pf_grow(12, &t.split.k, keys * 4 * KVD) || pf_grow(13, &t.split.v, keys * 4 * KVD) || pf_grow(2, &t.qkv, rows * QKV * 4) ||
                   pf_grow(3, &t.part, part * 4) || pf_grow(4, &t.ssq, rows * tc_prepare_chunks(D) * 4) ||
                   pf_grow(5, &t.bD, tc_acts_bytes((int)pad, D)) || pf_grow(6, &t.bQ, tc_acts_bytes((int)pad, QD)) ||
                   pf_grow(7, &t.bH, tc_acts_bytes((int)pad, HID))
               ? -1
               : 0;
}

static int pf_tc_buffers(int M, int start_pos, int block) {
    /* a last block may be split more ways than a full one */
    size_t part = 0, pad = 0, rows = 0;
    for (int left = M, r; left > 0; left -= r) {
        r = pf_next_rows(left, block);
        const PfBlock b = pf_block(r);
        for (size_t n : {(size_t)b.s_qkv * r * QKV, (size_t)b.s_wo * r * D, (size_t)b.s_w2 * r * D}) part = n > part ? n : part;
        pad = (size_t)b.rp > pad ? b.rp : pad;
        rows = (size_t)r > rows ? r : rows;
    }
    return pf_block_buffers(rows, pad, part, (size_t)(start_pos + M + kAtKeys - 1) / kAtKeys * kAtKeys);
}

/* Rows that go through a layer at once, with buffers for them: fewer where little memory is left; 0: the streaming
 * kernel, which takes a third of what a block of 256 rows takes here. */
static int pf_fit(int M, int start_pos) {
    for (int block = kPfRows; block >= 256; block /= 2) {
        if (pf_tc_buffers(M, start_pos, block) == 0) return block;
        pf_release_block();
    }
    return 0;
}

/* Failing here is not fatal: prefill() then uses the streaming kernel. */
int prefill_tc_setup() {
    g_pf.ready = !getenv("VB200_NO_TC") && !tc_init();
    return 0;
}

/* Prefill with the tcgen05 GEMM (vb_tc.cu, vb_tc_rows.cu), a block of rows through all layers:
 * gain+terms -> QKV -> RoPE -> cache rows -> causal attention over the cache so far, which leaves terms -> O ->
 * residual+gain+terms -> gate/up with SwiGLU -> down -> residual+gain+terms. */
static int prefill_block(float *xr, const float *cs, const PfSegs &segs, const PfBlock &b, int segment) {
    Model &m = model();
    PrefillTc &t = g_pf;
    cudaStream_t st = m.st;
    const float scale = 1.0f / sqrtf((float)VB200_HEAD_DIM);
    const int chunksD = tc_prepare_chunks(D), rows = segs.rows;
    TcActs aD, aQ, aH;
    if (tc_acts(&aD, t.bD, b.rp, D) || tc_acts(&aQ, t.bQ, b.rp, QD) || tc_acts(&aH, t.bH, b.rp, HID)) return -1;
    const uint64_t keys = (uint64_t)segs.keys;
    AtMaps maps = {};
    if (tc_map3(&maps.k, t.split.k, 1, keys * 4 * KVD, keys, 4 * KVD, 2 * KVD, kAtKeys) ||
        tc_map3(&maps.v, t.split.v, 1, keys * 4 * KVD, keys, 4 * KVD, 2 * KVD, kAtKeys))
        return -1;
    AtRows rows_of = {{t.qkv, {t.bQ, b.rp, QD, b.rp < 256 ? kTcTerms : 2}, QKV, {}}, {}};
    int most = 0;
    for (int i = 0; i < segs.n; i++) {
        rows_of.s[i] = {segs.s[i].row0, segs.s[i].rows, segs.s[i].pos, segs.s[i].key0};
        most = std::max(most, segs.s[i].rows);
    }
    const AtArgs args = {most, VB200_HEADS, VB200_KV_HEADS, VB200_HEAD_DIM, VB200_HEAD_DIM, 0, 0, scale, 0.0f, &m.d_out->status, 1};
    const size_t psD = (size_t)rows * D;
    for (int l = 0; l < VB200_DEC_LAYERS; l++) {
        const LayerDev &L = m.dec[l];
        if (l == 0) tc_prepare(aD, xr, D, rows, nullptr, 0, 0, nullptr, nullptr, L.attn_norm, t.ssq, st);
        TcGemm g;
        g.M = rows; g.status = &m.d_out->status; g.epi = TC_EPI_PARTIAL; g.out = t.part; g.ld_out = QKV; g.segment = segment;
        g.splits = b.s_qkv; g.ssq = t.ssq; g.ssq_chunks = chunksD; g.eps = VB200_NORM_EPS;
        if (tc_gemm(t.wqkv[l], aD, g, st)) return -1;
        for (int i = 0; i < segs.n; i++) {       /* earlier rows of a prompt: those of a block of its own alone */
            const PfSeg &e = segs.s[i];
            const PfSplit to = {t.split.k + (size_t)e.key0 * 2 * KVD, t.split.v + (size_t)e.key0 * 2 * KVD};
            if (e.pos > 0 && launch_pdl(pf_split_kernel, dim3(e.pos, KVD / 512), dim3(256), 0, st, to, (const float *)(e.k + l * e.layer),
                                        (const float *)(e.v + l * e.layer)) != cudaSuccess)
                return -1;
        }
        if (launch_pdl(pf_qkv_finish_kernel, dim3(QKV / 2 / 256, segs.grid), dim3(256), 0, st, t.qkv, (const float *)t.part, b.s_qkv,
                       (size_t)rows * QKV, cs, t.split, segs, l) != cudaSuccess)
            return -1;
        if (l == VB200_DEC_LAYERS - 1) break;   /* only the cache is kept (voxtral_tts_llm.c:281) */
        if (launch_attn_tc<2, 2>(args, rows_of, st, maps, segs.n)) return -1;
        g.splits = b.s_wo; g.ld_out = D; g.ssq = nullptr; g.ssq_chunks = 0;
        if (tc_gemm(t.wo[l], aQ, g, st)) return -1;
        tc_prepare(aD, nullptr, D, rows, t.part, b.s_wo, psD, xr, xr, L.ffn_norm, t.ssq, st);
        g.epi = TC_EPI_SWIGLU_TERMS; g.out = nullptr; g.out_terms = t.bH; g.out_rows_pad = b.rp; g.splits = 1;
        g.ld_out = HID; g.ssq = t.ssq; g.ssq_chunks = chunksD;
        if (tc_gemm(t.w13[l], aD, g, st)) return -1;
        g.epi = TC_EPI_PARTIAL; g.out = t.part; g.out_terms = nullptr; g.splits = b.s_w2; g.ld_out = D;
        g.ssq = nullptr; g.ssq_chunks = 0;
        if (tc_gemm(t.w2[l], aH, g, st)) return -1;
        /* residual add and the next layer's rows */
        tc_prepare(aD, nullptr, D, rows, t.part, b.s_w2, psD, xr, xr, m.dec[l + 1].attn_norm, t.ssq, st);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

/* The row blocks of a prompt follow one another through all layers: a row sees nothing of later rows. */
static int prefill_tc(float *x, const float *cs, int M, int start_pos, int block) {
    Model &m = model();
    for (int r0 = 0, rows; r0 < M; r0 += rows) {
        rows = pf_next_rows(M - r0, block);
        PfSegs segs;
        segs.add(rows, start_pos + r0, r0, m.kv_k, m.kv_v, m.kv_max);
        if (prefill_block(x + (size_t)r0 * D, cs, segs, pf_block(rows), TcGemm().segment)) return -1;
    }
    return 0;
}

/* Checks, and the buffers of all rows: g_pf.x for the embeddings, the rotation table. */
static int prefill_begin(int M, int start_pos) {
    Model &m = model();
    if (start_pos < 0 || start_pos + M > m.kv_max) {
        fprintf(stderr, "voxtral_b200: prefill of %d rows at %d exceeds the %d-row cache\n", M, start_pos, m.kv_max);
        return -1;
    }
    PrefillTc &t = g_pf;
    if (pf_grow(0, &t.x, (size_t)M * D * 4) || pf_grow(1, &t.cs, (size_t)M * VB200_HEAD_DIM * 4)) return -1;
    rope_table(t.cs, start_pos, M, VB200_HEAD_DIM, VB200_ROPE_THETA, m.st);
    return 0;
}

static int prefill_run(int M, int start_pos);

/* Waits for what was enqueued; its status, or rc. */
static int pf_finish(int rc) {
    Model &m = model();
    int status = 0;
    if (cudaMemcpyAsync(&status, &m.d_out->status, sizeof(int), cudaMemcpyDeviceToHost, m.st) != cudaSuccess ||
        cudaStreamSynchronize(m.st) != cudaSuccess)
        return -1;
    if (rc) return rc;
    m.last_status = status;
    if (!status) return 0;
    /* the word is sticky on the device (kernels only set it from 0): clear it so the next call starts clean */
    cudaMemset(&m.d_out->status, 0, sizeof(int));
    return -1;
}

/* Several prompts from position 0 on, each into a cache of its own (kv_max rows a layer): side by side through the layers as
 * long as a block has room, so that the weights are read once and the GEMMs are wide. Eight prompts of 100 to 187 rows took
 * 27 ms one after another. Only those that alone would be one block of two-term products; the others, and all where memory
 * is short, are left for prefill(): done[i] says which are in their caches. K is summed in pieces of 1024 columns: alone,
 * those of up to 256 rows have the frame's K splits, sums of 704 to 1536 columns (2048 for gate/up). */
constexpr int kPfJointSegment = 16;
int prefill_joint(const PfPrompt *prompts, int n, int kv_max, bool *done) {
    Model &m = model();
    PrefillTc &t = g_pf;
    if (!m.inited || !m.llm_ready) return -1;
    std::vector<int> fit;
    for (int i = 0; i < n; i++) {
        done[i] = false;
        const int r = prompts[i].rows;
        if (r > 64 && r <= kv_max && r <= kPfRows && pf_next_rows(r, kPfRows) == r) fit.push_back(i);
    }
    if (!t.ready || fit.size() < 2 || batch_tiled_decoder(&t.wqkv, &t.wo, &t.w13, &t.w2)) return 0;
    for (size_t i = 0; i < fit.size();) {
        PfSegs segs;
        int most = 0;
        size_t j = i;
        for (; j < fit.size() && segs.n < kPfSegs && segs.rows + prompts[fit[j]].rows <= kPfRows; j++) {
            const PfPrompt &p = prompts[fit[j]];
            segs.add(p.rows, 0, 0, p.kv_k, p.kv_v, kv_max);
            most = std::max(most, p.rows);
        }
        if (segs.n < 2) { i = j; continue; }
        const PfBlock b = pf_block(segs.rows);
        const size_t part = std::max({(size_t)b.s_qkv * QKV, (size_t)b.s_wo * D, (size_t)b.s_w2 * D}) * segs.rows;
        if (pf_grow(0, &t.x, (size_t)segs.rows * D * 4) || pf_grow(1, &t.cs, (size_t)most * VB200_HEAD_DIM * 4) ||
            pf_block_buffers(segs.rows, b.rp, part, segs.keys)) {
            pf_release_block();
            return 0;
        }
        rope_table(t.cs, 0, most, VB200_HEAD_DIM, VB200_ROPE_THETA, m.st);
        for (size_t k = i; k < j; k++)
            if (cudaMemcpyAsync(t.x + (size_t)segs.s[k - i].row0 * D, prompts[fit[k]].embeds, (size_t)prompts[fit[k]].rows * D * 4, cudaMemcpyDefault,
                                m.st) != cudaSuccess)
                return -1;
        if (pf_finish(prefill_block(t.x, t.cs, segs, b, kPfJointSegment))) return -1;
        for (size_t k = i; k < j; k++) done[fit[k]] = true;
        i = j;
    }
    return 0;
}

int prefill(const float *embeds, int seq_len, int start_pos) {
    Model &m = model();
    if (!m.inited || !m.llm_ready) return -1;
    if (seq_len <= 0) return 0;
    if (prefill_begin(seq_len, start_pos)) return -1;
    if (cudaMemcpyAsync(g_pf.x, embeds, (size_t)seq_len * D * 4, cudaMemcpyDefault, m.st) != cudaSuccess) return -1;
    return prefill_run(seq_len, start_pos);
}

/* The rows are in g_pf.x. */
static int prefill_run(int M, int start_pos) {
    Model &m = model();
    PrefillTc &t = g_pf;
    float *x = t.x, *cs = t.cs;
    int rc = 0;
    const float scale = 1.0f / sqrtf((float)VB200_HEAD_DIM);

    const int block = t.ready && batch_tiled_decoder(&t.wqkv, &t.wo, &t.w13, &t.w2) == 0 ? pf_fit(M, start_pos) : 0;
    if (block > 0) return pf_finish(prefill_tc(x, cs, M, start_pos, block));
    if (pf_grow(2, &t.qkv, (size_t)M * QKV * 4) || pf_grow(8, &t.attn, (size_t)M * QD * 4) || pf_grow(9, &t.h, (size_t)M * HID * 4)) return -1;
    float *qkv = t.qkv, *attn = t.attn, *h = t.h;
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
    if (prefill_begin(n, start_pos)) return -1;
    PrefillTc &t = g_pf;
    if (pf_grow(10, &t.ids, sizeof(int) * n) || pf_grow(11, &t.voice, (size_t)n_voice * D * 2)) return -1;
    if (cudaMemcpyAsync(t.ids, ids.data(), sizeof(int) * n, cudaMemcpyHostToDevice, m.st) != cudaSuccess) return -1;
    if (n_voice > 0 && cudaMemcpyAsync(t.voice, voice_bf16, (size_t)n_voice * D * 2, cudaMemcpyHostToDevice, m.st) != cudaSuccess) {
        cudaStreamSynchronize(m.st);
        return -1;
    }
    prompt_rows_kernel<<<dim3((D + 255) / 256, n), 256, 0, m.st>>>(t.x, m.tok_emb, t.voice, t.ids, D);
    if (cudaGetLastError() != cudaSuccess) return -1;
    return prefill_run(n, start_pos) == 0 ? n : -1;      /* synchronises the stream */
}

} // namespace vb
