// Prompts of the 0.8B model, all positions at once (declarations: include/mk_b200.h).
//
// The kernels are those of mk_prefill.cuh with fp32-exact operands: token rows enter the tensor cores as three bf16
// pieces (24 bits), weights are exact in bf16 (int8 values need eight bits), sums are fp32 and the row scales of int8
// weights are applied to them, so a prompt's state agrees with stepping to fp32 rounding.  The decode kernels' weight
// layouts depend on the grid and are not operand tiles, so an engine that takes prompts in keeps a second copy of its
// matrices as bf16 slabs (mk_prefill_weights, 1 GB; rewriting them in every pass cost a tenth of a 512-token prompt).
#include "mk_prefill_host.h"

using namespace mkp;
typedef mk::Qwen35_08B S;

// mk_api.cu: the engine's description and parameter block
int mk_engine_view(mk_engine* e, const mk_model_desc** desc, const mk::Params** params, bool* static_only);

namespace {

constexpr int PX = 3;
// Most tokens per tile: what rows_gemm adds up in registers (bf16 weights), or what leaves two accumulators for the first piece.
int tile_tokens(int quant) { return quant == MK_QUANT_INT8 ? 160 : 32 * DRAIN_GROUPS; }

// Weight rows in the decode layout (groups of up to eight rows, 64-byte k-blocks; pack.py: pack_rows) -> slabs.
// A lane takes 16 bytes of a row; `glu` moves alternating gate / up rows into tiles of eight gates and their eight ups.
template <bool Q8>
__global__ void __launch_bounds__(256) slabs_from_rows(const uint8_t* w, int N, int rb, int unit, int grid, bool glu, uint8_t* out, int out_rows) {
    const int nkb = rb >> 6;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int q = (int)(i & 3), lr = (int)((i >> 2) & 7);
    const int kb = (int)((i >> 5) % nkb), r = (int)((i >> 5) / nkb) * 8 + lr;
    if (r >= N) return;
    const long long units = N / unit;
    const int cta = (int)((((long long)(r / unit) + 1) * grid - 1) / units);
    int r0, r1;
    mk::cta_rows(N, unit, cta, grid, r0, r1);
    const int rpc = mk::SLOT_BYTES / rb, base = r0 + (r - r0) / rpc * rpc, in = r - base, gs = in & ~7;
    const int nr = min(rpc, r1 - base), ng = min(8, nr - gs);
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(w + (size_t)(base + gs) * rb + (size_t)kb * ng * 64 + (in - gs) * 64) + q);
    const int row = glu ? ((r >> 1) >> 3) * 16 + (r & 1) * 8 + ((r >> 1) & 7) : r;
    if (Q8) {
        const uint32_t s[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t x = s[2 * h + (j >> 1)] >> (16 * (j & 1));
                o[j] = pack_bf16((float)(int)(signed char)(x & 0xff), (float)(int)(signed char)((x >> 8) & 0xff));
            }
            *reinterpret_cast<uint4*>(out + slab_offset(out_rows, row, kb * 64 + q * 16 + h * 8)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    } else {
        *reinterpret_cast<uint4*>(out + slab_offset(out_rows, row, kb * 32 + q * 8)) = v;
    }
}

// Column slices of a bf16 matrix in fragment order (pack.py: pack_col_slices): slice s holds columns [k0, k1) of all S::HID
// rows, KM 16-column products per 16-row tile.  `inter` > 0: the slices are those of CTA s's SwiGLU outputs, else 16 each.
template <int KM>
__global__ void __launch_bounds__(256) slabs_from_cols(const uint8_t* w, int slices, int inter, uint8_t* out, int out_rows) {
    constexpr int TILES = S::HID / 16;
    const int i = blockIdx.x * 256 + threadIdx.x, lane = i & 31, tile = (i >> 5) % TILES, s = (i >> 5) / TILES;
    if (s >= slices) return;
    int k0 = s * 16, k1 = k0 + 16;
    if (inter) {
        mk::cta_rows(2 * inter, 2, s, slices, k0, k1);
        k0 >>= 1;
        k1 >>= 1;
    }
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int m = 0; m < KM; m++) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(w) + ((size_t)(s * TILES + tile) * 32 + lane) * KM + m);
        const uint32_t x[4] = {v.x, v.y, v.z, v.w};                       // (low columns: row g, g + 8), (high columns: row g, g + 8)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int k = k0 + 16 * m + 8 * (j >> 1) + 2 * t + e, row = tile * 16 + g + 8 * (j & 1);
                if (k < k1) *reinterpret_cast<uint16_t*>(out + slab_offset(out_rows, row, k)) = (uint16_t)(x[j] >> (16 * e));
            }
    }
}

template <bool Q8>
__global__ void __launch_bounds__(256) embed_rows_08b(const uint8_t* table, const float* scale, const int* tokens, int vocab, float* h) {
    chain_wait();
    const int tok = max(0, min(vocab - 1, tokens[blockIdx.x])), c = threadIdx.x * 4;
    float4 v;
    if (Q8) {
        const char4 b = *reinterpret_cast<const char4*>(table + (size_t)tok * S::HID + c);
        const float s = scale[tok];
        v = make_float4(b.x * s, b.y * s, b.z * s, b.w * s);
    } else {
        const uint2 b = *reinterpret_cast<const uint2*>(table + ((size_t)tok * S::HID + c) * 2);
        v = make_float4(bf_lo(b.x), bf_hi(b.x), bf_lo(b.y), bf_hi(b.y));
    }
    *reinterpret_cast<float4*>(h + (size_t)blockIdx.x * S::HID + c) = v;
}

__global__ void put_pos(int* p, int v) {
    chain_wait();
    *p = v;
}

// Where a layer's four matrices lie among the slabs (rows rounded up to whole 128-row blocks).
struct LayerSlabs {
    const uint8_t *in, *out, *gu, *down, *end;
    static size_t bytes(int rows, int k) { return (size_t)((rows + 127) / 128 * 128) * k * 2; }
    LayerSlabs(const uint8_t* base, const mk::Params* P, int layer) {
        for (int l = 0; l <= layer; l++) {
            in = l ? end : base;
            out = in + bytes(P->layer[l].kind ? S::ATT_IN : S::GDN_IN, S::HID);
            gu = out + bytes(S::HID, S::MIX);
            down = gu + bytes(2 * S::INTER, S::HID);
            end = down + bytes(S::HID, S::INTER);
        }
    }
};

int to_slabs(const mk_model_desc* desc, const uint8_t* src, int N, int K, int unit, bool glu, const uint8_t* dst, cudaStream_t st) {
    const bool q8 = desc->quant == MK_QUANT_INT8;
    const int rb = q8 ? K : 2 * K, n = (int)(((long long)((N + 7) / 8) * (rb / 64) * 32 + 255) / 256);
    auto fn = q8 ? slabs_from_rows<true> : slabs_from_rows<false>;
    fn<<<n, 256, 0, st>>>(src, N, rb, unit, desc->grid, glu, const_cast<uint8_t*>(dst), (N + 127) / 128 * 128);
    MKP_CUDA(cudaGetLastError());
    return MK_OK;
}

struct Run {
    const mk_model_desc* desc;
    const mk::Params* P;
    int rows, nt, ntiles, xrows, sms, start, seq, batched, tile_most;
    const int* tokens;
    long long spin;
    cudaStream_t st;
    Arena arena;
    float *h, *y, *part, *qkv, *o, *q, *gram;
    float4* scal;
    uint8_t *x, *mix, *act;
    const uint8_t* slabs;
    size_t x_piece, mix_piece, act_piece;
    int* pos;

    void layout(float* resid) {
        token_tiles(rows, tile_most, &ntiles, &nt);
        xrows = ntiles * nt;
        h = resid ? resid : arena.take<float>((size_t)rows * S::HID);
        y = arena.take<float>((size_t)rows * S::PROJ_MAX);
        x_piece = (size_t)S::HID / 64 * xrows * 128;
        mix_piece = (size_t)S::MIX / 64 * xrows * 128;
        act_piece = (size_t)S::INTER / 64 * xrows * 128;
        x = arena.take<uint8_t>(PX * x_piece);
        mix = arena.take<uint8_t>(PX * mix_piece);
        act = arena.take<uint8_t>(PX * act_piece);
        qkv = arena.take<float>((size_t)rows * S::CONV_DIM);
        scal = arena.take<float4>((size_t)rows * S::LIN_H);
        o = arena.take<float>((size_t)rows * S::LIN_V);
        q = arena.take<float>((size_t)rows * S::MIX);
        gram = arena.take<float>((size_t)((rows + SCAN - 1) / SCAN) * S::LIN_H * GRAM);
        part = arena.take<float>((size_t)8 * rows * S::HID);
        pos = arena.take<int>(1);
    }

    int left = 0;                // K splits of a product whose partials wait in `part` to be added to the residual

    // The normed residual as operand slabs; adds what the product before left.
    int norm(const float* w) {
        const RowsIn R = {h, S::HID, S::HID, left, rows, part, w, 1.f, S::EPS, 1.f, x, x_piece, xrows};
        MKP_CUDA(launch(left ? rows_in<PX, true> : rows_in<PX, false>, dim3(rows), 256, 0, st, R));
        left = 0;
        return MK_OK;
    }

    // `leave`: the residual's next reader is norm(), which adds the K splits' partials.
    int product(const uint8_t* w, int N, int K, const uint8_t* xs, size_t piece, const float* scale, int out, float* dst, int dst_stride, bool leave = false) {
        GemmArgs A;
        memset(&A, 0, sizeof A);
        A.w = w;
        A.w_rows = (N + 127) / 128 * 128;
        A.tiles = (N + 15) / 16;
        A.row_scale = scale;
        A.rs_pairs = out == OUT_GLU;
        A.x = xs;
        A.x_piece = piece;
        A.x_rows = xrows;
        A.out = dst;
        A.out_stride = dst_stride;
        A.act = act;
        A.act_piece = act_piece;
        A.act_rows = xrows;
        A.act_cols = S::INTER;
        A.n_valid = N;
        A.rows = rows;
        A.nt = nt;
        A.kbs = K / 64;
        const int blocks = (N + 127) / 128;
        A.ksplit = N == S::HID ? pick_ksplit(blocks * ntiles, A.kbs, sms) : 1;     // `part` holds the narrow products only
        A.part = part;
        A.part_rows = rows;
        A.leave = leave;
        if (leave && A.ksplit > 1) left = A.ksplit;
        A.status = P->status;
        A.spin_limit_ns = spin;
        return launch_gemm<W_SLAB, PX>(A, out, blocks, ntiles, 0, st);
    }

    int run() {
        const bool q8 = desc->quant == MK_QUANT_INT8, kv32 = desc->kv_dtype == MK_KV_F32;
        int rc;
        MKP_CUDA(launch(put_pos, dim3(1), 1, 0, st, pos, start));
        if (q8) MKP_CUDA(launch(embed_rows_08b<true>, dim3(rows), 256, 0, st, P->embed, P->embed_scale, tokens, P->vocab, h));
        else MKP_CUDA(launch(embed_rows_08b<false>, dim3(rows), 256, 0, st, P->embed, nullptr, tokens, P->vocab, h));
        MKP_CUDA(cudaGetLastError());
        for (int l = 0; l < P->n_layers; l++) {
            const mk::LayerP& L = P->layer[l];
            const bool attn = L.kind != 0;
            const int in_rows = attn ? S::ATT_IN : S::GDN_IN;
            if ((rc = norm(L.in_norm)) != MK_OK) return rc;
            const LayerSlabs W(slabs, P, l);
            if ((rc = product(W.in, in_rows, S::HID, x, x_piece, L.s_in, OUT_STORE, y, S::PROJ_MAX)) != MK_OK) return rc;
            if (attn) {
                AttnArgs T;
                memset(&T, 0, sizeof T);
                T.y = y; T.y_stride = S::PROJ_MAX;
                T.M = 1; T.L = rows; T.nq = S::NQ; T.nkv = S::NKV;
                T.q_hs = 2 * S::HD; T.gate_off = S::HD; T.k_off = S::ATT_K_OFF; T.v_off = S::ATT_V_OFF;
                T.rot = S::ROT; T.pairs = S::ROT / 2;
                T.eps = S::EPS; T.scale = 1.f; T.q_scale = 0.0625f;
                T.q_norm = L.q_norm; T.k_norm = L.k_norm; T.cos = P->rope_cos; T.sin = P->rope_sin;
                T.k_cache = L.k_cache; T.v_cache = L.v_cache;
                T.bt = P->block_table + (size_t)seq * (P->max_seq / mk::KV_BLOCK);
                T.max_pages = P->max_seq / mk::KV_BLOCK; T.kv_shift = 6;
                T.s_page = S::NKV * mk::KV_BLOCK * S::HD; T.s_head = mk::KV_BLOCK * S::HD; T.s_pos = S::HD;
                T.pos = pos; T.q = q; T.out = mix; T.out_piece = mix_piece; T.out_rows = xrows;
                const dim3 pg((S::NQ + 2 * S::NKV + 7) / 8, rows), blocks((rows + AF_ROWS / S::QPK - 1) / (AF_ROWS / S::QPK), S::NKV, 1);
                const int splits = attn_splits(blocks.x * blocks.y, start + rows, sms);
                const dim3 ag(blocks.x * splits, blocks.y, 1);
                if (kv32) {
                    MKP_CUDA(launch((attn_prepare<256, true, true>), pg, 256, 0, st, T));
                    MKP_CUDA(cudaFuncSetAttribute(attn_rows_f32<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_f32_smem<true>()));
                    MKP_CUDA(launch_cluster(attn_rows_f32<true>, ag, 256, attn_f32_smem<true>(), splits, st, T));
                } else {
                    MKP_CUDA(launch((attn_prepare<256, true, false>), pg, 256, 0, st, T));
                    MKP_CUDA(cudaFuncSetAttribute(attn_rows_f32<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_f32_smem<false>()));
                    MKP_CUDA(launch_cluster(attn_rows_f32<false>, ag, 256, attn_f32_smem<false>(), splits, st, T));
                }
            } else {
                GdnArgs G;
                memset(&G, 0, sizeof G);
                G.y = y; G.y_stride = S::PROJ_MAX;
                G.M = 1; G.L = rows; G.nkh = G.nvh = S::LIN_H; G.conv_dim = S::CONV_DIM;
                G.k_off = S::LIN_QK; G.v_off = 2 * S::LIN_QK; G.z_off = S::Z_OFF; G.b_off = S::B_OFF; G.a_off = S::A_OFF;
                G.conv_w = L.conv_w; G.A_log = L.A_log; G.dt_bias = L.dt_bias; G.norm_w = L.gdn_norm;
                G.conv_state = batched ? L.conv_hist_b + (size_t)seq * S::CONV_DIM * mk::CONV_RING : L.conv_hist;
                G.ring = mk::CONV_RING; G.layout = batched ? 2 : 1;
                G.ssm = L.state + (size_t)seq * S::LIN_H * S::LIN_DV * S::LIN_DK;
                G.pos = pos; G.l2_clamp = 1; G.eps = 1e-6f; G.norm_eps = S::EPS;
                G.qkv = qkv; G.scal = scal; G.gram = gram; G.o = o; G.out = mix; G.out_piece = mix_piece; G.out_rows = xrows;
                if ((rc = launch_gdn(G, gdn_gate<PX>, sms, st)) != MK_OK) return rc;
            }
            MKP_CUDA(cudaGetLastError());
            if ((rc = product(W.out, S::HID, S::MIX, mix, mix_piece, L.s_out, OUT_ADD, h, S::HID, true)) != MK_OK) return rc;
            if ((rc = norm(L.post_norm)) != MK_OK) return rc;
            if ((rc = product(W.gu, 2 * S::INTER, S::HID, x, x_piece, L.s_gu, OUT_GLU, nullptr, 0)) != MK_OK) return rc;
            if ((rc = product(W.down, S::HID, S::INTER, act, act_piece, L.s_down, OUT_ADD, h, S::HID, l + 1 < P->n_layers)) != MK_OK) return rc;
        }
        return MK_OK;
    }
};

}  // namespace

extern "C" int64_t mk_prefill_weight_bytes(mk_engine* e) {
    const mk_model_desc* desc;
    const mk::Params* P;
    bool bare;
    if (!e || mk_engine_view(e, &desc, &P, &bare) != MK_OK) return pfail(MK_ERR_BADARG, "mk_prefill_weight_bytes: mk_set_params has not succeeded on this engine");
    return (int64_t)(LayerSlabs(nullptr, P, P->n_layers - 1).end - static_cast<const uint8_t*>(nullptr)) + 1024;
}

extern "C" int mk_prefill_weights(mk_engine* e, uint64_t weights, int64_t bytes, void* stream) {
    const mk_model_desc* desc;
    const mk::Params* P;
    bool bare;
    if (!e || !weights || mk_engine_view(e, &desc, &P, &bare) != MK_OK) return pfail(MK_ERR_BADARG, "mk_prefill_weights: null argument or no parameters");
    if (bytes < mk_prefill_weight_bytes(e)) return pfail(MK_ERR_BADARG, "mk_prefill_weights: %lld bytes, %lld needed", (long long)bytes, (long long)mk_prefill_weight_bytes(e));
    const uint8_t* base = reinterpret_cast<const uint8_t*>((weights + 1023) & ~(uint64_t)1023);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    MKP_CUDA(cudaSetDevice(desc->device));
    for (int l = 0; l < P->n_layers; l++) {
        const mk::LayerP& L = P->layer[l];
        const LayerSlabs W(base, P, l);
        int rc = to_slabs(desc, L.w_in, L.kind ? S::ATT_IN : S::GDN_IN, S::HID, 1, false, W.in, st);
        // the out- and down-projection: rows where the engine keeps them, else the column slices of the tasks / CTAs
        const uint8_t* w_out = L.kind ? L.w_out : L.w_out_rows;
        if (rc == MK_OK && w_out) rc = to_slabs(desc, w_out, S::HID, S::MIX, 1, false, W.out, st);
        else if (rc == MK_OK) slabs_from_cols<1><<<S::GDN_TASKS * (S::HID / 16) * 32 / 256, 256, 0, st>>>(L.w_out, S::GDN_TASKS, 0, const_cast<uint8_t*>(W.out), S::HID);
        if (rc == MK_OK) rc = to_slabs(desc, L.w_gu, 2 * S::INTER, S::HID, 2, true, W.gu, st);
        if (rc == MK_OK && L.w_down_rows) rc = to_slabs(desc, L.w_down_rows, S::HID, S::INTER, 1, false, W.down, st);
        else if (rc == MK_OK)
            slabs_from_cols<2><<<(desc->grid * (S::HID / 16) * 32 + 255) / 256, 256, 0, st>>>(L.w_down, desc->grid, S::INTER, const_cast<uint8_t*>(W.down), S::HID);
        if (rc != MK_OK) return rc;
        MKP_CUDA(cudaGetLastError());
    }
    return MK_OK;
}

extern "C" int64_t mk_prefill_bytes(int positions) {
    if (positions < 1 || positions > MAX_ROWS) return pfail(MK_ERR_BADARG, "mk_prefill_bytes: %d positions", positions);
    Run R;
    memset(&R, 0, sizeof R);
    R.rows = positions;
    size_t most = 0;
    for (int quant : {MK_QUANT_BF16, MK_QUANT_INT8}) {
        R.arena.off = 0;
        R.tile_most = tile_tokens(quant);
        R.layout(nullptr);
        most = R.arena.off > most ? R.arena.off : most;
    }
    return (int64_t)most + 1024;
}

extern "C" int mk_prefill(mk_engine* e, const mk_prefill_args* a, void* stream) {
    if (!e || !a) return pfail(MK_ERR_BADARG, "mk_prefill: null argument");
    Run R;
    memset(&R, 0, sizeof R);
    bool bare;
    if (mk_engine_view(e, &R.desc, &R.P, &bare) != MK_OK) return pfail(MK_ERR_BADARG, "mk_prefill: mk_set_params has not succeeded on this engine");
    if (a->positions < 1 || a->positions > MAX_ROWS || !a->tokens || !a->workspace || !a->weights) return pfail(MK_ERR_BADARG, "mk_prefill: positions %d, tokens / weights / workspace missing", a->positions);
    if (a->start_pos < 0 || (int64_t)a->start_pos + a->positions > R.desc->max_seq) return pfail(MK_ERR_BADARG, "mk_prefill: sequence would exceed max_seq=%d", R.desc->max_seq);
    if (a->sequence < 0 || a->sequence >= (R.desc->max_batch > 1 ? R.desc->max_batch : 1)) return pfail(MK_ERR_BADARG, "mk_prefill: sequence %d", a->sequence);
    // what the launches behind a prompt refuse
    if (bare) return pfail(MK_ERR_BADARG, "mk_prefill: this engine was given no hand-off buffers; only mk_launch_static can run it");
    if (a->batched && R.desc->quant != MK_QUANT_INT8) return pfail(MK_ERR_UNSUPPORTED, "mk_prefill: batched decoding is built for int8 weights only");
    if (a->batched && !R.P->actl) return pfail(MK_ERR_BADARG, "mk_prefill: the engine was given no MLP activation words (MK_G_ACTL)");
    for (int l = 0; l < R.P->n_layers; l++)
        if (a->batched && ((R.P->layer[l].kind == 0 && (!R.P->layer[l].conv_hist_b || !R.P->layer[l].w_out_rows)) || !R.P->layer[l].w_down_rows))
            return pfail(MK_ERR_BADARG, "mk_prefill: layer %d lacks the batched kernel's buffers (MK_L_CONV_HIST_B, MK_L_W_OUT_ROWS, MK_L_W_DOWN_ROWS)", l);
    MKP_CUDA(cudaSetDevice(R.desc->device));
    MKP_CUDA(cudaDeviceGetAttribute(&R.sms, cudaDevAttrMultiProcessorCount, R.desc->device));
    R.rows = a->positions;
    R.tile_most = tile_tokens(R.desc->quant);
    R.start = a->start_pos;
    R.seq = a->sequence;
    R.batched = a->batched;
    R.tokens = reinterpret_cast<const int*>(a->tokens);
    R.slabs = reinterpret_cast<const uint8_t*>((a->weights + 1023) & ~(uint64_t)1023);
    R.spin = a->spin_limit_ns > 0 ? a->spin_limit_ns : 2000000000ll;
    R.st = static_cast<cudaStream_t>(stream);
    R.arena.base = reinterpret_cast<uint8_t*>((a->workspace + 1023) & ~(uint64_t)1023);
    R.layout(reinterpret_cast<float*>(a->resid_out));
    if ((int64_t)R.arena.off + 1024 > a->workspace_bytes) return pfail(MK_ERR_BADARG, "mk_prefill: workspace of %lld bytes, %lld needed", (long long)a->workspace_bytes, (long long)R.arena.off + 1024);
    return R.run();
}
