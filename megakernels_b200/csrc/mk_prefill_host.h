// Host helpers shared by the two prompt paths (mk_prefill.cu: stage programs, mk_prefill_08b.cu: the 0.8B model).
#pragma once
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "../../include/mk_b200.h"
#include "mk_prefill.cuh"

int mk_set_error(int code, const char* text);       // mk_api.cu: the text behind mk_last_error()

namespace mkp {

inline int pfail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    return mk_set_error(code, buf);
}
#define MKP_CUDA(call)                                                                      \
    do {                                                                                    \
        cudaError_t err__ = (call);                                                         \
        if (err__ != cudaSuccess)                                                           \
            return pfail(MK_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(err__));   \
    } while (0)

// Launches a kernel of the chain (see chain_wait).
template <class Kernel, class... Args>
inline cudaError_t launch(Kernel fn, dim3 grid, int threads, size_t smem, cudaStream_t st, const Args&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

// The same in clusters of `ranks` CTAs along x.
template <class Kernel, class... Args>
inline cudaError_t launch_cluster(Kernel fn, dim3 grid, int threads, size_t smem, int ranks, cudaStream_t st, const Args&... args) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ranks;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

constexpr int SMEM_MAX = 232448;
constexpr int DRAIN_GROUPS = 4;                     // rows_gemm: three-piece products in tiles of up to 32 x 4 tokens
constexpr int MAX_ROWS = 65535;                     // token rows of a call: one grid coordinate of several kernels

// Hands out the workspace; with base == nullptr it only counts.
struct Arena {
    uint8_t* base;
    size_t off = 0;
    template <class T>
    T* take(size_t n) {
        off = (off + 1023) & ~(size_t)1023;
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += n * sizeof(T);
        return p;
    }
};

template <int FMT, int PX, int CG, int DG, bool WIDE = false>
int launch_gemm_cg(GemmArgs& A, int out, dim3 grid, int smem, cudaStream_t st) {
    auto fn = out == OUT_STORE ? rows_gemm<FMT, PX, OUT_STORE, CG, DG, WIDE> : (out == OUT_ADD ? rows_gemm<FMT, PX, OUT_ADD, CG, DG, WIDE> : rows_gemm<FMT, PX, OUT_GLU, CG, DG, WIDE>);
    MKP_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    MKP_CUDA(launch(fn, grid, (8 * CG + 2) * 32, smem, st, A));
    MKP_CUDA(cudaGetLastError());
    return MK_OK;
}

template <int FMT, int PX>
int launch_gemm(GemmArgs& A, int out, int blocks, int tiles_x, int items, cudaStream_t st) {
    constexpr int PW = weight_pieces<FMT>;
    const int stage = PW * A_BYTES + PX * A.nt * 128, fixed = (int)sizeof(GemmBars) + 1024;
    // Narrow tiles leave room for two CTAs per SM with three stages each: one's start and end hide behind the other.  Wide
    // ones have the SM to themselves, with sixteen warps to convert weights (eight cannot keep up with the MMAs).
    int stages = (SMEM_MAX / 2 - 1024 - fixed) / stage;
    const bool two = stages >= 3;
    if (!two) stages = (SMEM_MAX - fixed) / stage;
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    if (stages < 2) return pfail(MK_ERR_BADARG, "prefill: %d tokens per tile leave no room for two stages", A.nt);
    A.stages = stages;
    const int smem = stages * stage + fixed;
    const dim3 grid = items ? dim3(blocks, items, 1) : dim3(tiles_x, blocks, A.ksplit);
    int rc;
    if constexpr (FMT == W_SLAB) {
        // Adding up in registers costs 3 % of a 512-token prompt and is what bf16 weights need.  Those of an int8 matrix (the ones
        // with row scales) are integers of seven bits, whose products leave less to round away: with two accumulators for the
        // first piece such a prompt is as close to 64 bits as stepping (logits 3.8e-6 of their norm against 3.7e-6 at 300
        // tokens and 24 layers; with one 4.8e-6).
        const bool drain = A.nt > 64 && !A.row_scale;
        if (A.nt > (drain ? 32 * DRAIN_GROUPS : 160)) return pfail(MK_ERR_BADARG, "prefill: %d tokens per tile", A.nt);
        rc = drain ? launch_gemm_cg<FMT, PX, 1, DRAIN_GROUPS>(A, out, grid, smem, st) : launch_gemm_cg<FMT, PX, 1, 0>(A, out, grid, smem, st);
    } else {
        if (A.nt > 256) {
            if constexpr (PW == 1 && FMT != W_FP8_BLOCK) rc = launch_gemm_cg<FMT, PX, 2, 0, true>(A, out, grid, smem, st);
            else return pfail(MK_ERR_BADARG, "prefill: %d tokens per tile", A.nt);
        } else {
            rc = two ? launch_gemm_cg<FMT, PX, 1, 0>(A, out, grid, smem, st) : launch_gemm_cg<FMT, PX, 2, 0>(A, out, grid, smem, st);
        }
    }
    if (rc != MK_OK) return rc;
    if (A.ksplit > 1 && !A.leave) {
        const dim3 fgrid(out == OUT_GLU ? (A.act_cols + 255) / 256 : (A.n_valid + 1023) / 1024, A.rows);
        if (out == OUT_STORE) MKP_CUDA(launch((rows_finish<PX, OUT_STORE>), fgrid, 256, 0, st, A));
        else if (out == OUT_ADD) MKP_CUDA(launch((rows_finish<PX, OUT_ADD>), fgrid, 256, 0, st, A));
        else MKP_CUDA(launch((rows_finish<PX, OUT_GLU>), fgrid, 256, 0, st, A));
        MKP_CUDA(cudaGetLastError());
    }
    return MK_OK;
}

// CTAs that share a row block's keys in attn_rows_f32: `ctas` row blocks, the longest sees `keys` keys.  While the SMs have room
// for all of them, two blocks of keys each are enough; up to two CTAs per SM, one after the other, pay where the longest share is four
// blocks (they even out the causal triangle).  Passes of the int8 model without and with, ms: 120 rows (2 each) 2.82 / 2.78, 250 (2)
// 3.32 / 3.22 (with 4 3.27), 400 (2) 4.64 / 4.50, 511 (2) 5.06 / 4.91; no room: 600 with 2 all the same 5.82 / 5.75, 1000 8.28 / 8.43.
inline int attn_splits(int ctas, int keys, int sms) {
    const int blocks = (keys + AF_KEYS - 1) / AF_KEYS;
    int s = 1;
    while (s < 8 && ((2 * s * ctas <= sms && blocks >= 4 * s) || (2 * s * ctas <= 2 * sms && blocks >= 8 * s))) s *= 2;
    return s;
}

// FP8 products of routed groups with at most 8 NT8 rows per work item; `items` bounds the number of items.
template <bool BLOCKS, int NT8>
int launch_experts(GemmArgs& A, int out, int items, int sms, cudaStream_t st) {
    const int smem = experts_smem(NT8);
    const long long units = (long long)items * A.blocks;
    auto fn = out == OUT_GLU ? experts_gemm<BLOCKS, OUT_GLU, NT8> : experts_gemm<BLOCKS, OUT_STORE, NT8>;
    MKP_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    MKP_CUDA(launch(fn, dim3((int)(units < 2 * sms ? units : 2 * sms)), 256, smem, st, A));
    MKP_CUDA(cudaGetLastError());
    return MK_OK;
}

// The DeltaNet mixer of M sequences of L rows; `gate` is gdn_gate of the wanted number of pieces.
inline int launch_gdn(const GdnArgs& G, void (*gate)(GdnArgs), int sms, cudaStream_t st) {
    const int rows = G.M * G.L, chunks = (G.L + SCAN - 1) / SCAN;
    MKP_CUDA(launch(gdn_conv, dim3((G.conv_dim / 128 + 7) / 8, G.M * ((G.L + CONV_ROWS - 1) / CONV_ROWS)), 256, 0, st, G));
    MKP_CUDA(launch(gdn_gram, dim3((G.M * chunks * G.nkh + 3) / 4 + G.M * G.ring * ((G.conv_dim + 127) / 128)), 128, 0, st, G));
    // One CTA per SM or less: not with the chain's attribute.  Brought up while gdn_gram's many small CTAs drain, several of them
    // land on one SM and share its shared memory, which is what they are bound by (16 heads x 511 positions: the pass takes 6.41 instead
    // of 5.27 ms).  With more CTAs than SMs they share anyway.
    const dim3 scan(8, G.nvh, G.M);
    // (More than three CTAs per SM: fewer registers each instead of a second round.)
    if (8 * G.nvh * G.M <= sms) gdn_scan<false><<<scan, 128, 0, st>>>(G);
    else MKP_CUDA(launch(8 * G.nvh * G.M <= 3 * sms ? gdn_scan<false> : gdn_scan<true>, scan, 128, 0, st, G));
    MKP_CUDA(cudaGetLastError());
    MKP_CUDA(launch(gate, dim3((G.nvh + 15) / 16, rows), 256, 0, st, G));
    MKP_CUDA(cudaGetLastError());
    return MK_OK;
}

// Token tiles of `rows` rows: equal tiles of at most `most`, multiples of 16.
inline void token_tiles(int rows, int most, int* n, int* nt) {
    *n = (rows + most - 1) / most;
    *nt = ((rows + *n - 1) / *n + 15) / 16 * 16;
}

// CTAs that share the K range of one tile: the count with the shortest schedule (rounds of one CTA per SM, each 64-column
// block counted once, the start and end of a CTA as six and the pass that adds the partials as 4 + z: estimates), at least
// eight blocks each.
inline int pick_ksplit(int ctas, int kbs, int sms) {
    int best = 1;
    double cost = 1e30;
    for (int z = 1; z <= 8 && (z == 1 || kbs / z >= 8); z++) {
        const double c = (double)((ctas * z + sms - 1) / sms) * ((kbs + z - 1) / z + 6) + (z > 1 ? 4 + z : 0);
        if (c < cost) {
            cost = c;
            best = z;
        }
    }
    return best;
}

}  // namespace mkp
