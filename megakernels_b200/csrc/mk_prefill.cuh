// Token-parallel kernels of the prompt path (mk_prefill.cu): what a decode program does for the eight columns of
// one step, done for all positions of a prompt at once.
//
// The contractions are matrix products here, so they run on the 5th-generation tensor cores: `rows_gemm` keeps 128
// weight rows as the A operand of tcgen05.mma and up to 384 token rows as its N columns, accumulators in tensor
// memory.  (FP8 experts with few rows each: `experts_gemm`, where the weights stay in registers for mma.sync.)  The weights of a stage program stay in the decode kernel's packed tiles: eight or sixteen warps read a tile
// step each with one 128-bit load per lane, convert it to bf16 pieces that hold its value and write the swizzled operand
// into shared memory, so a prompt reads the same bytes from HBM as a decode step does and needs no second copy of the
// model.  (The 0.8B model does keep one: mk_prefill_08b.cu.)
//
// Operand layout in global memory ("slabs"): a matrix of R token rows and K columns is stored as K / 64 slabs of R
// rows x 128 bytes, the 16-byte pieces of a row swizzled with its number (piece p of row r sits at p ^ (r & 7)).
// Any run of rows that starts at a multiple of eight is then one contiguous, ready-to-use K-major SWIZZLE_128B tile:
// the producer brings it with one untiled bulk copy, and no tensor map is needed.
#pragma once
#include <cuda_fp16.h>

#include "../../include/mk_stage.h"
#include "mk_device.cuh"

namespace mkp {
using mk::bf_hi;
using mk::bf_lo;
using mk::mbar_arrive;
using mk::mbar_expect_tx;
using mk::mbar_init;
using mk::mbar_try_wait;
using mk::sigmoid_f;
using mk::silu_f;
using mk::smem_u32;
using mk::softplus_f;
using mk::u64;
using mk::warp_max;
using mk::warp_sum;

// A pass is a chain of some hundred short kernels, launched with programmatic stream serialisation: a kernel's CTAs come up
// while the one before drains, and wait here for its end before they touch memory that any kernel of the chain writes.  Every
// kernel of the chain calls this first thing (a CTA that left without it would let the next kernel start too early), or behind a
// prologue that reads nothing but the packed weights.  (512 tokens of the 0.8B model, 231 launches: 5.79 ms without the attribute, 5.28 with it.)
//   The next kernel's CTAs come up once every CTA has called chain_release or left.  A kernel that needs tensor memory calls it only
// when it owns it: the next one may allocate before it waits (rows_gemm of dense products does), an allocation waits without a
// limit, and columns that it took ahead of a CTA still to allocate would never come free.
__device__ __forceinline__ void chain_acquire() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() {
    chain_acquire();
    chain_release();
}

constexpr int ERR_TIMEOUT = -2;
enum { WP_EMPTY = 301, WP_FULL, WP_DONE, WP_DRAIN };

// Byte offset of column `c` of row `row` inside a slab array with `rows` rows per slab (bf16 elements).
__host__ __device__ __forceinline__ size_t slab_offset(int rows, int row, int c) {
    return ((size_t)(c >> 6) * rows + row) * 128 + (size_t)((((c >> 3) & 7) ^ (row & 7)) << 4) + (size_t)(c & 7) * 2;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
// Eight consecutive columns c .. c + 7 of a row into PIECES slabs (piece i + 1 is what the pieces before it lost).
template <int PIECES>
__device__ __forceinline__ void store_slab8(uint8_t* x, size_t piece_stride, int rows, int row, int c, float (&v)[8]) {
    uint8_t* dst = x + slab_offset(rows, row, c);
#pragma unroll
    for (int p = 0; p < PIECES; p++) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            w[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
            if (p + 1 < PIECES) {
                v[2 * i] -= bf_lo(w[i]);
                v[2 * i + 1] -= bf_hi(w[i]);
            }
        }
        *reinterpret_cast<uint4*>(dst + (size_t)p * piece_stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// ---- matrix product ----------------------------------------------------------------------------------------
// How the weights come: packed tiles of a format, or bf16 slabs.  Block-scaled FP8 has three forms: few tokens per tile leave
// room in tensor memory for an accumulator per 128-column block, and the epilogue adds them with their scales
// (W_FP8_BLOCK, the decode kernel's arithmetic); many tokens do not, and the scaled weights enter as bf16 pieces.  A value
// has 4 bits: with scales that are bf16 values (8 bits; the record says so) two pieces hold the product exactly
// (W_FP8_PIECES2), at twice the MMAs; with any fp32 scale three hold its fp32 value (W_FP8_PIECES3).
enum { W_MXFP4 = 0, W_FP8, W_FP8_BLOCK, W_FP8_PIECES2, W_FP8_PIECES3, W_BF16, W_SLAB };
template <int FMT> constexpr int weight_pieces = FMT == W_FP8_PIECES3 ? 3 : (FMT == W_FP8_PIECES2 ? 2 : 1);
enum { OUT_STORE = 0, OUT_ADD, OUT_GLU };

struct GemmArgs {
    // weights: [group][split][tile][chunk] blocks (stage/pack.py), or slabs
    const uint8_t* w;
    size_t w_gstride;            // bytes between groups
    int tiles, unit_steps, chunk_steps, chunk_bytes, kc;
    int w_rows;                  // W_SLAB: rows per slab
    const float* row_scale;      // per weight row, or null
    size_t rs_gstride;
    int rs_pairs;                // OUT_GLU: the scales alternate gate, up (the 0.8B layout) instead of following the tiles
    // token operand
    const uint8_t* x;
    size_t x_piece;              // bytes between its pieces
    int x_rows;                  // rows per slab
    // output
    float* out;
    long long out_stride;        // floats between token rows
    uint8_t* act;                // OUT_GLU: slab array of the activations
    size_t act_piece;
    int act_rows, act_cols;      // activation columns (n_valid pairs)
    int n_valid;                 // weight rows that exist
    int rows;                    // token rows that exist (dense)
    int nt;                      // tokens per tile (a multiple of 16; <= 384, with pieces or per-block accumulators 256)
    int kbs;                     // 64-column blocks of K
    int blocks;                  // experts_gemm: 128-row blocks of a group
    int ksplit;                  // CTAs that share K; > 1: fp32 partials [split][part_rows][n_valid] in `part`
    float* part;
    int part_rows;
    bool leave;                  // the partials are left to rows_in
    int gelu;
    // routed groups: items[i] = {group, first row, rows, 0}, n_items on the device
    const int4* items;
    const int* n_items;
    int stages;
    int* status;
    long long spin_limit_ns;
};

constexpr int A_BYTES = 128 * 128;                     // one 64-column block of 128 weight rows
constexpr int MAX_STAGES = 8;
struct GemmBars {
    uint64_t full[MAX_STAGES], empty[MAX_STAGES], done;
    uint64_t block_full[2], block_read[2];      // drained products: the two accumulators of the first piece
    uint32_t tmem;
    volatile int dead;
};

static __device__ __noinline__ bool wait_slow(volatile int* dead, const GemmArgs& A, uint64_t* b, uint32_t parity, int site) {
    u64 t0 = 0;
#pragma unroll 1
    for (unsigned it = 0;; it++) {
        if (mbar_try_wait(b, parity)) return true;
        if ((it & 63u) == 63u) {
            if (*dead) return false;
            const u64 now = mk::globaltimer();
            if (!t0) t0 = now;
            else if (now - t0 > (u64)A.spin_limit_ns) {
                *dead = 1;
                if (atomicCAS(A.status, 0, ERR_TIMEOUT) == 0) {
                    A.status[1] = site;
                    A.status[2] = (int)blockIdx.x;
                    A.status[3] = (int)threadIdx.x;
                }
                return false;
            }
        }
    }
}
template <class Bars>
__device__ __forceinline__ bool wait(Bars& B, const GemmArgs& A, uint64_t* b, uint32_t parity, int site) {
    return mbar_try_wait(b, parity) || wait_slow(&B.dead, A, b, parity, site);
}

// K-major SWIZZLE_128B operand: rows of 128 bytes, eight-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t operand_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t e2m1x2_f16(uint32_t b) {
    uint32_t r;
    asm("{\n .reg .b8 t;\n .reg .b16 h;\n cvt.u16.u32 h, %1;\n cvt.u8.u16 t, h;\n cvt.rn.f16x2.e2m1x2 %0, t;\n}\n" : "=r"(r) : "r"(b));
    return r;
}
// Two e4m3 values (bytes `sel` picks) moved to the bf16 fields: the values times 2^-120, subnormals included.
__device__ __forceinline__ uint32_t e4m3_as_bf16(uint32_t w, uint32_t sel) {
    const uint32_t b = __byte_perm(w, 0u, sel);                      // each byte in the upper half of its 16 bits
    return (b & 0x80008000u) | ((b >> 4) & 0x07F007F0u);
}
// The bits of a half moved to the bf16 fields: the value times 2^-112 (halves of at most 7 mantissa bits, no subnormals).
__device__ __forceinline__ uint32_t f16_as_bf16(uint32_t h) { return (h & 0x80008000u) | ((h >> 3) & 0x0FFF0FFFu); }

// Raw bytes of one 64-column block of a 16-row tile, as lane (g, q) holds them.
template <int FMT> struct Raw { uint4 q[FMT == W_BF16 ? 4 : (FMT == W_MXFP4 ? 1 : 2)]; uint32_t s[weight_pieces<FMT> > 1 ? 2 : 1]; };

// Walks the 64-column blocks of one tile: its units follow one another.
template <int FMT>
struct Walk {
    static constexpr int STEPS = FMT == W_BF16 ? 4 : (FMT == W_MXFP4 ? 1 : 2);      // 512-byte steps per 64 columns
    const uint8_t *p, *s;      // this lane's bytes of the next step; the current chunk's scales
    int left;                  // steps left in the chunk
    __device__ __forceinline__ void start(const GemmArgs& A, const uint8_t* w, int tile, int kb, int lane) {
        constexpr int STEP_K = 64 / STEPS;
        const int split = kb * 64 / A.kc, at = (kb * 64 - split * A.kc) / STEP_K;
        const size_t unit = (size_t)(A.unit_steps / A.chunk_steps) * A.chunk_bytes;
        const int within = at % A.chunk_steps;
        const uint8_t* chunk = w + ((size_t)tile * (A.kbs * 64 / A.kc) + split) * unit + (size_t)(at / A.chunk_steps) * A.chunk_bytes;
        left = A.chunk_steps - within;
        p = chunk + within * 512 + lane * 16;
        s = chunk + A.chunk_steps * 512 + (FMT == W_MXFP4 ? within * 32 + (lane >> 2) * 4 : (within >> 2) * 8);
    }
    __device__ __forceinline__ void load(const GemmArgs& A, Raw<FMT>& r) {
        if (FMT == W_MXFP4) r.s[0] = __ldg(reinterpret_cast<const uint32_t*>(s));
        if constexpr (weight_pieces<FMT> > 1) {
            const uint2 x = __ldg(reinterpret_cast<const uint2*>(s));
            r.s[0] = x.x;
            r.s[1] = x.y;
        }
#pragma unroll
        for (int i = 0; i < STEPS; i++) {
            r.q[i] = __ldg(reinterpret_cast<const uint4*>(p));
            step(A);
        }
    }
    __device__ __forceinline__ void skip(const GemmArgs& A) {
#pragma unroll
        for (int i = 0; i < STEPS; i++) step(A);
    }
    __device__ __forceinline__ void step(const GemmArgs& A) {
        p += 512;
        if (FMT == W_MXFP4) s += 32;
        if (weight_pieces<FMT> > 1 && (left & 3) == 1) s += 8;
        if (--left == 0) {
            left = A.chunk_steps;
            p += A.chunk_bytes - A.chunk_steps * 512;
            s += A.chunk_bytes - (FMT == W_MXFP4 ? A.chunk_steps * 32 : A.chunk_steps * 2);
        }
    }
};

// Two scaled values as bf16 pieces: each takes the first eight bits of what the ones before it left.
__device__ __forceinline__ void split_scaled(uint32_t e, float s, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    float a = bf_lo(e) * s, b = bf_hi(e) * s;
    p0 = pack_bf16(a, b);
    a -= bf_lo(p0); b -= bf_hi(p0);
    p1 = pack_bf16(a, b);
    a -= bf_lo(p1); b -= bf_hi(p1);
    p2 = pack_bf16(a, b);
}
// One lane's share of a block as bf16: piece 0's v[row half][j] holds columns 16 j + 4 q + {0 .. 3}.
template <int FMT>
__device__ __forceinline__ void convert(const Raw<FMT>& r, uint2 (&pieces)[weight_pieces<FMT>][2][4]) {
    uint2 (&v)[2][4] = pieces[0];
    if constexpr (FMT == W_BF16) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[0][j] = make_uint2(r.q[j].x, r.q[j].y);
            v[1][j] = make_uint2(r.q[j].z, r.q[j].w);
        }
    } else if constexpr (FMT == W_MXFP4) {
        const uint32_t sc = r.s[0] & 0x7F7F7F7Fu;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            // scale group 0 (j = 0, 1): bits pre-arranged by the packer; three magnitude bits at 8..6 of a half are the
            // value times 2^-126.  Group 1 (j = 2, 3): plain nibbles, through f16: the value times 2^-112.
            const uint32_t w = h == 0 ? r.q[0].x : r.q[0].z, n = h == 0 ? r.q[0].y : r.q[0].w;
            // factors 2^(s - 1) and 2^(s - 15) in both halves: the scale byte moved to the exponent field, plus a constant
            const uint32_t m0 = __byte_perm(sc, 0u, h == 0 ? 0x4040 : 0x4242) * 128u + 0x3F003F00u;
            const uint32_t m1 = __byte_perm(sc, 0u, h == 0 ? 0x4141 : 0x4343) * 128u + 0x38003800u;
            v[h][0].x = mul_bf16x2((w & 0x80008000u) | ((w >> 3) & 0x01C001C0u), m0);
            v[h][0].y = mul_bf16x2(((w << 3) & 0x80008000u) | (w & 0x01C001C0u), m0);
            v[h][1].x = mul_bf16x2(((w << 1) & 0x80008000u) | ((w << 3) & 0x01C001C0u), m0);
            v[h][1].y = mul_bf16x2(((w << 2) & 0x80008000u) | ((w << 6) & 0x01C001C0u), m0);
            v[h][2].x = mul_bf16x2(f16_as_bf16(e2m1x2_f16(n)), m1);
            v[h][2].y = mul_bf16x2(f16_as_bf16(e2m1x2_f16(n >> 8)), m1);
            v[h][3].x = mul_bf16x2(f16_as_bf16(e2m1x2_f16(n >> 16)), m1);
            v[h][3].y = mul_bf16x2(f16_as_bf16(e2m1x2_f16(n >> 24)), m1);
        }
        if (r.s[0] & 0x80808080u) {            // scales of 2 and more: the top bit is worth 2^128, twice 2^64
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const uint32_t m = (r.s[0] >> (16 * h + 8 * (j >> 1) + 7)) & 1u ? 0x5F805F80u : 0x3F803F80u;
                    v[h][j].x = mul_bf16x2(mul_bf16x2(v[h][j].x, m), m);
                    v[h][j].y = mul_bf16x2(mul_bf16x2(v[h][j].y, m), m);
                }
        }
    } else {
        constexpr uint32_t UP = 0x7B807B80u;       // 2^120
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t w[4] = {r.q[i].x, r.q[i].y, r.q[i].z, r.q[i].w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int h = k >> 1, j = 2 * i + (k & 1);
                v[h][j].x = mul_bf16x2(e4m3_as_bf16(w[k], 0x1404), UP);
                v[h][j].y = mul_bf16x2(e4m3_as_bf16(w[k], 0x3424), UP);
                if constexpr (FMT == W_FP8_PIECES2) {
                    const uint32_t s = r.s[h] >> 16, ss = s | (s << 16), neg = 0xBF80BF80u;      // (a bf16 value: the lower half is zero)
                    const uint2 e = v[h][j];
                    uint2& lo = pieces[1][h][j];
                    v[h][j].x = mul_bf16x2(e.x, ss);
                    v[h][j].y = mul_bf16x2(e.y, ss);
                    lo.x = fma_bf16x2(e.x, ss, mul_bf16x2(v[h][j].x, neg));
                    lo.y = fma_bf16x2(e.y, ss, mul_bf16x2(v[h][j].y, neg));
                } else if constexpr (FMT == W_FP8_PIECES3) {
                    const float s = __uint_as_float(r.s[h]);
                    const uint2 e = v[h][j];
                    split_scaled(e.x, s, v[h][j].x, pieces[1][h][j].x, pieces[2][h][j].x);
                    split_scaled(e.y, s, v[h][j].y, pieces[1][h][j].y, pieces[2][h][j].y);
                }
            }
        }
    }
}

// Writes a lane's share of a tile into the swizzled operand.  Lanes of odd rows store their columns in the order
// j = 2, 3, 0, 1: the sixteen 8-byte stores of a half warp then fall into different banks.
__device__ __forceinline__ void store_operand(uint8_t* a, const uint32_t (&off)[4], bool odd, const uint2 (&v)[2][4]) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 4; i++) *reinterpret_cast<uint2*>(a + off[i] + h * 1024) = odd ? v[h][i ^ 2] : v[h][i];
}
// Sixteen accumulator columns of this lane's row.
__device__ __forceinline__ void load16(uint32_t tmem, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(tmem));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Scale of weight row n in 128-column block b of block-scaled FP8: behind the chunk's steps, one for the upper and one for
// the lower eight rows of a tile.
__device__ __forceinline__ float block_scale(const GemmArgs& A, int group, int n, int b) {
    const int tile = min(n >> 4, A.tiles - 1), split = b * 128 / A.kc, in = b - split * (A.kc / 128), per = A.chunk_steps / 4;
    const size_t unit = (size_t)(A.unit_steps / A.chunk_steps) * A.chunk_bytes;
    const uint8_t* chunk = A.w + (size_t)group * A.w_gstride + ((size_t)tile * (A.kbs * 64 / A.kc) + split) * unit + (size_t)(in / per) * A.chunk_bytes;
    return __ldg(reinterpret_cast<const float*>(chunk + A.chunk_steps * 512 + (in % per) * 8) + ((n >> 3) & 1));
}

// One CTA: 128 weight rows x nt token rows over a range of K.
//   warps 0 .. 8 CG - 1  CG groups of eight convert weight tiles into the A operand (group c takes every CG-th block of 64
//                        columns, warp w of a group tile w), then read the accumulators back (epilogue);
//   warp 8 CG            one lane brings the token operand (and, for slab weights, the A operand) with bulk copies;
//   warp 8 CG + 1        one lane issues the MMAs.
// grid: x = token tile (neighbouring CTAs share weights, so HBM reads them once), y = 128-row weight block, z = K split;
// routed groups: x = weight block, y = work item.
// PX: bf16 pieces of the token operand (3: fp32-exact inputs); weight pieces: see the formats.
// An accumulation in tensor memory rounds its sum towards zero, once per instruction.  Three-piece inputs stand for fp32 ones,
// and one accumulator for all of K left a 24-layer bf16 prompt five times as far from 64 bits as stepping (logits 1.9e-5 of
// their norm against 4.0e-6).  So the small products of pieces 2 and 3 have an accumulator of their own, and the first piece's
// sums are short:
//   DG = 0  as many accumulators as tensor memory has room for, each over its share of K;
//   DG > 0  two accumulators of one 64-column block each, in turn: the conversion warps, which have no weights to convert, add
//           them up in registers, DG groups of sixteen tokens per warp, while the other one is filled.
template <int FMT, int PX, int OUT, int CG, int DG, bool WIDE = false>
static __global__ void __launch_bounds__((8 * CG + 2) * 32, CG == 1 && DG == 0 ? 2 : 1) rows_gemm(const __grid_constant__ GemmArgs A) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int PW = weight_pieces<FMT>, CW = 8 * CG;
    constexpr int DIST = FMT == W_BF16 || FMT == W_FP8_PIECES3 ? 2 : (FMT == W_MXFP4 ? 6 : 4);        // blocks a lane requests ahead
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int group = 0, row0, rows, block, z = 0;
    if (A.items) {
        chain_acquire();
        if ((int)blockIdx.y >= __ldcg(A.n_items)) return;
        const int4 it = __ldcg(A.items + blockIdx.y);
        group = it.x;
        row0 = it.y;
        rows = it.z;
        block = blockIdx.x;
    } else {
        row0 = (int)blockIdx.x * A.nt;
        rows = min(A.nt, A.rows - row0);
        block = blockIdx.y;
        z = blockIdx.z;
    }
    const int nt = A.items ? (rows + 15) & ~15 : A.nt;         // columns this CTA multiplies
    const int kb0 = (int)((long long)A.kbs * z / A.ksplit), kb1 = (int)((long long)A.kbs * (z + 1) / A.ksplit);
    const uint32_t x_bytes = (uint32_t)nt * 128u, stage_bytes = PW * A_BYTES + PX * (uint32_t)A.nt * 128u;
    GemmBars& B = *reinterpret_cast<GemmBars*>(smem + (size_t)A.stages * stage_bytes);
    const int blocks128 = FMT == W_FP8_BLOCK ? A.kbs / 2 : 1;   // (K splits do not occur with per-block accumulators)
    const int first_accs = DG ? 2 : (PX > 1 ? min(512 / nt - 1, kb1 - kb0) : 1);
    int cols = 32;
    while (cols < nt * (PX > 1 ? 1 + first_accs : blocks128)) cols *= 2;
    if (threadIdx.x == 0) {
        for (int i = 0; i < A.stages; i++) {
            mbar_init(&B.full[i], FMT == W_SLAB ? 1 : 8 + 1);
            mbar_init(&B.empty[i], 1);
        }
        mbar_init(&B.done, 1);
        for (int i = 0; i < 2; i++) {
            mbar_init(&B.block_full[i], 1);
            mbar_init(&B.block_read[i], 8);
        }
        B.dead = 0;
        mk::fence_barrier_init();
    }
    if (warp == CW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&B.tmem)), "r"(cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = B.tmem;
    if (A.items) chain_release();
    else if (FMT == W_SLAB || warp >= CW) chain_wait();

    if (warp == CW) {
        if (lane == 0) {
            uint32_t slot = 0, phase = 0;
#pragma unroll 1
            for (int kb = kb0; kb < kb1; kb++) {
                if (!wait(B, A, &B.empty[slot], phase ^ 1u, WP_EMPTY)) break;
                uint8_t* st = smem + (size_t)slot * stage_bytes;
                mbar_expect_tx(&B.full[slot], PX * x_bytes + (FMT == W_SLAB ? A_BYTES : 0));
                if (FMT == W_SLAB)
                    mk::bulk_load(st, A.w + (size_t)group * A.w_gstride + ((size_t)kb * A.w_rows + (size_t)block * 128) * 128, A_BYTES, &B.full[slot], mk::policy_evict_first());
#pragma unroll
                for (int p = 0; p < PX; p++)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(smem_u32(st + PW * A_BYTES + (size_t)p * A.nt * 128)),
                                   "l"(A.x + (size_t)p * A.x_piece + ((size_t)kb * A.x_rows + row0) * 128), "r"(x_bytes), "r"(smem_u32(&B.full[slot])) : "memory");
                if (++slot == (uint32_t)A.stages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
            if (B.dead) {
                // a role gave up: copies in flight must land before the CTA leaves (their barrier may still await others,
                // so this waits a bounded time instead)
                const u64 t0 = mk::globaltimer();
                while (mk::globaltimer() - t0 < 1000000ull) {}
            }
        }
    } else if (warp == CW + 1) {
        if (lane == 0) {
            // f32 <- bf16 x bf16, M 128; an instruction has at most 256 columns, so a wide tile takes two
            const uint32_t n0 = WIDE ? (uint32_t)((nt / 2 + 15) & ~15) : (uint32_t)nt, n1 = (uint32_t)nt - n0;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n0 >> 3) << 17) | (8u << 24), idesc1 = (1u << 4) | (1u << 7) | (1u << 10) | ((n1 >> 3) << 17) | (8u << 24);
            uint32_t slot = 0, phase = 0, first = 1;
            int chunk = 0;                                        // of the first piece: its accumulator
            bool ok = true, begin = true;
#pragma unroll 1
            for (int kb = kb0; kb < kb1; kb++) {
                if ((DG && !wait(B, A, &B.block_read[(kb - kb0) & 1], (((kb - kb0) >> 1) & 1) ^ 1, WP_DRAIN)) || !wait(B, A, &B.full[slot], phase, WP_FULL)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t st = smem_u32(smem + (size_t)slot * stage_bytes);
#pragma unroll
                for (int px = 0; px < PX; px++)
#pragma unroll
                    for (int pw = 0; pw < PW; pw++) {
                        const uint64_t da = operand_desc(st + pw * A_BYTES), db = operand_desc(st + PW * A_BYTES + px * (uint32_t)A.nt * 128u);
                        const uint32_t d = tmem + (PX > 1 ? (uint32_t)(px ? 0 : (1 + chunk) * nt) : 0u) + (FMT == W_FP8_BLOCK ? (uint32_t)((kb >> 1) * nt) : 0u);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const bool starts = FMT == W_FP8_BLOCK ? !(kb & 1) : (PX > 1 && px == 0 ? begin : first != 0);
                            const uint32_t accumulate = !(starts && k == 0 && pw == 0 && px <= 1);
                            asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                                         ::"r"(d), "l"(da + 2 * k), "l"(db + 2 * k), "r"(idesc), "r"(accumulate));
                            if constexpr (WIDE)              // the rows past n0 (whole groups of eight)
                                asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                                             ::"r"(d + n0), "l"(da + 2 * k), "l"(db + (uint64_t)(n0 * 8) + 2 * k), "r"(idesc1), "r"(accumulate));
                        }
                    }
                first = 0;
                if (DG) {
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&B.block_full[chunk])) : "memory");
                    chunk ^= 1;
                } else if (PX > 1) {
                    const int next = (kb + 1 - kb0) * first_accs / (kb1 - kb0);
                    begin = next != chunk;
                    chunk = next;
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&B.empty[slot])) : "memory");
                if (++slot == (uint32_t)A.stages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
            if (ok) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&B.done)) : "memory");
        }
    } else {
        if constexpr (FMT != W_SLAB) {
            // warp = tile: its bytes are requested DIST blocks ahead, straight into registers
            const int w8 = warp & 7, tile = block * 8 + w8, kb_first = kb0 + (warp >> 3);
            const bool have = tile < A.tiles;
            if (!have)                       // rows past the matrix: zero in every slot, never written again
                for (int i = lane; i < A.stages * 128; i += 32) {
                    uint8_t* a = smem + (size_t)(i >> 7) * stage_bytes + (size_t)w8 * 2048 + (i & 127) * 16;
#pragma unroll
                    for (int p = 0; p < PW; p++) *reinterpret_cast<uint4*>(a + p * A_BYTES) = make_uint4(0u, 0u, 0u, 0u);
                }
            const int g = lane >> 2, q = lane & 3;
            // offsets of the lane's 8-byte pieces j = 0 .. 3 of a row: odd rows take j = 2, 3, 0, 1 (see store_operand)
            uint32_t off[4];
#pragma unroll
            for (int i = 0; i < 4; i++) off[i] = (uint32_t)(w8 * 2048 + g * 128 + (q & 1) * 8) + (((2 * (g & 1 ? i ^ 2 : i) + (q >> 1)) ^ g) << 4);
            Walk<FMT> walk;
            walk.start(A, A.w + (size_t)group * A.w_gstride, min(tile, A.tiles - 1), min(kb_first, kb1 - 1), lane);
            Raw<FMT> raw[DIST];
            int asked = kb_first;
            auto request = [&](Raw<FMT>& r) {
                if (asked < kb1) {
                    walk.load(A, r);
                    if (CG == 2) walk.skip(A);
                    asked += CG;
                }
            };
#pragma unroll
            for (int i = 0; i < DIST; i++) request(raw[i]);
            if (!A.items) chain_wait();
            uint32_t slot = (uint32_t)(warp >> 3), phase = 0;
            bool ok = true;
#pragma unroll 1
            for (int kb = kb_first; kb < kb1 && ok; kb += DIST * CG) {
#pragma unroll
                for (int i = 0; i < DIST; i++) {
                    if (kb + i * CG < kb1 && ok) {
                        uint2 v[PW][2][4];
                        convert<FMT>(raw[i], v);
                        request(raw[i]);
                        ok = __all_sync(0xffffffffu, wait(B, A, &B.empty[slot], phase ^ 1u, WP_EMPTY));   // the warp leaves together
                        if (ok && have) {
                            uint8_t* st = smem + (size_t)slot * stage_bytes;
#pragma unroll
                            for (int p = 0; p < PW; p++) store_operand(st + p * A_BYTES, off, g & 1, v[p]);
                        }
                        mk::fence_proxy_async();
                        __syncwarp();
                        if (ok && lane == 0) mbar_arrive(&B.full[slot]);
                        slot += CG;
                        if (slot >= (uint32_t)A.stages) {
                            slot -= A.stages;
                            phase ^= 1u;
                        }
                    }
                }
            }
        }
        // the sums of drained products: this lane's row, group g of sixteen tokens
        float sums[DG ? DG : 1][16];
        bool drained = true;
        if constexpr (DG > 0) {
#pragma unroll
            for (int g = 0; g < DG; g++)
#pragma unroll
                for (int i = 0; i < 16; i++) sums[g][i] = 0.f;
#pragma unroll 1
            for (int b = 0; b < kb1 - kb0 && drained; b++) {
                drained = __all_sync(0xffffffffu, wait(B, A, &B.block_full[b & 1], (b >> 1) & 1, WP_DRAIN));
                if (!drained) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int g = 0; g < DG; g++) {
                    const int c0 = (warp >> 2) * 16 + 32 * g;
                    if (c0 < nt) {
                        uint32_t r[16];
                        load16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((1 + (b & 1)) * nt + c0), r);
#pragma unroll
                        for (int i = 0; i < 16; i++) sums[g][i] += __uint_as_float(r[i]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&B.block_read[b & 1]);
            }
        }
        // ---- epilogue: lane = weight row, columns = tokens; each set of four warps takes every 2 CG-th group of 16 tokens
        const bool ok = drained && __all_sync(0xffffffffu, wait(B, A, &B.done, 0, WP_DONE));
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int sub = warp & 3, n = block * 128 + sub * 32 + lane;
            float rs = 1.f;
            if (A.row_scale && n < A.n_valid) rs = __ldg(A.row_scale + (size_t)group * A.rs_gstride + (A.rs_pairs ? 2 * ((n >> 4) * 8 + (n & 7)) + ((n >> 3) & 1) : n));
#pragma unroll(DG ? DG : 1)
            for (int g = 0; g < (DG ? DG : 16); g++) {
                const int c0 = (warp >> 2) * 16 + 32 * CG * g;
                if (c0 >= nt) break;
                float v[16];
                {
                    uint32_t r[16];
                    load16(tmem + ((uint32_t)(sub * 32) << 16) + (uint32_t)c0, r);
                    const float s0 = FMT == W_FP8_BLOCK ? block_scale(A, group, n, 0) : 1.f;
#pragma unroll
                    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]) * s0;
                    if (FMT == W_FP8_BLOCK) {
#pragma unroll 2
                        for (int b = 1; b < blocks128; b++) {
                            const float s = block_scale(A, group, n, b);
                            load16(tmem + ((uint32_t)(sub * 32) << 16) + (uint32_t)(b * nt + c0), r);
#pragma unroll
                            for (int i = 0; i < 16; i++) v[i] = fmaf(__uint_as_float(r[i]), s, v[i]);
                        }
                    }
                    if constexpr (DG > 0) {
#pragma unroll
                        for (int i = 0; i < 16; i++) v[i] += sums[g][i];
                    } else if (PX > 1) {
#pragma unroll 1
                        for (int a = 1; a <= first_accs; a++) {
                            load16(tmem + ((uint32_t)(sub * 32) << 16) + (uint32_t)(a * nt + c0), r);
#pragma unroll
                            for (int i = 0; i < 16; i++) v[i] += __uint_as_float(r[i]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] *= rs;
                if (A.ksplit > 1) {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (c0 + i < rows && n < A.n_valid) A.part[((size_t)z * A.part_rows + row0 + c0 + i) * A.n_valid + n] = v[i];
                } else if (OUT == OUT_GLU) {
                    // Rows 0-7 of a 16-row tile are gates, rows 8-15 their up rows.  The two lanes of a pair share the tokens:
                    // the gate's lane computes tokens 0-7, the up row's lane tokens 8-15; then the eight lanes of a half
                    // tile exchange, so that each holds eight neighbouring columns of one token and stores 16 bytes.
                    const bool hi = n & 8;
                    float y[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float other = __shfl_xor_sync(0xffffffffu, hi ? v[i] : v[i + 8], 8);
                        const float gate = hi ? other : v[i], up = hi ? v[i + 8] : other;
                        y[i] = (A.gelu ? 0.5f * gate * (1.f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate))) : silu_f(gate)) * up;
                    }
#pragma unroll
                    for (int o = 4; o; o >>= 1) {          // 8 x 8 transpose: afterwards y[c] is column c of token (lane & 7)
                        const bool u = lane & o;
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (!(i & o)) {
                                const float got = __shfl_xor_sync(0xffffffffu, u ? y[i] : y[i + o], o);
                                if (u) y[i] = got;
                                else y[i + o] = got;
                            }
                    }
                    const int t = c0 + (hi ? 8 : 0) + (lane & 7), col = (n >> 4) * 8;
                    if (t < rows && col < A.act_cols) store_slab8<PX>(A.act, A.act_piece, A.act_rows, row0 + t, col, y);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (c0 + i < rows && n < A.n_valid) {
                            float* o = A.out + (size_t)(row0 + c0 + i) * A.out_stride + n;
                            *o = OUT == OUT_ADD ? *o + v[i] : v[i];
                        }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
    }
    __syncthreads();
    if (warp == CW + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
    }
}

// Adds the K splits' partials in split order and runs the epilogue.
template <int PX, int OUT>
static __global__ void __launch_bounds__(256) rows_finish(const __grid_constant__ GemmArgs A) {
    chain_wait();
    const int t = blockIdx.y;
    const float* p = A.part + (size_t)t * A.n_valid;
    const size_t ss = (size_t)A.part_rows * A.n_valid;
    if (OUT == OUT_GLU) {
        const int col = blockIdx.x * 256 + threadIdx.x;
        if (col >= A.act_cols) return;
        const int n = (col >> 3) * 16 + (col & 7);
        float g = 0.f, u = 0.f;
        for (int z = 0; z < A.ksplit; z++) {
            g += p[z * ss + n];
            u += p[z * ss + n + 8];
        }
        float y = (A.gelu ? 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) : silu_f(g)) * u;
        uint8_t* dst = A.act + slab_offset(A.act_rows, t, col);
#pragma unroll
        for (int q = 0; q < PX; q++) {
            const __nv_bfloat16 b = __float2bfloat16_rn(y);
            *reinterpret_cast<__nv_bfloat16*>(dst + (size_t)q * A.act_piece) = b;
            y -= __bfloat162float(b);
        }
    } else {
        const int n = (blockIdx.x * 256 + threadIdx.x) * 4;
        if (n >= A.n_valid) return;
        float* o = A.out + (size_t)t * A.out_stride + n;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (((A.n_valid | (int)A.out_stride) & 3) == 0) {
            for (int z = 0; z < A.ksplit; z++) {
                const float4 a = *reinterpret_cast<const float4*>(p + z * ss + n);
                v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
            }
            float4* o4 = reinterpret_cast<float4*>(o);
            if (OUT == OUT_ADD) {
                const float4 b = *o4;
                v[0] += b.x; v[1] += b.y; v[2] += b.z; v[3] += b.w;
            }
            *o4 = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            for (int i = 0; i < 4 && n + i < A.n_valid; i++) {
                for (int z = 0; z < A.ksplit; z++) v[i] += p[z * ss + n + i];
                o[i] = OUT == OUT_ADD ? o[i] + v[i] : v[i];
            }
        }
    }
}

// ---- element-wise steps ------------------------------------------------------------------------------------
__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
    for (int i = 0; i < (int)blockDim.x / 32; i++) s += red[i];
    __syncthreads();
    return s;
}

// fp32 rows -> slabs: optional RMSNorm, rounding to bf16 (PIECES = 1, the model's activation type) or fp32-exact pieces.
// PARTS: the row is `x` plus the K splits' partial products `part` [split][rows][K], in split order, and is stored back first:
// the end of one product and the input of the next in one pass over the residual (511 x 1024, eight splits: 5.6 us against 5.4 + 4.3).
struct RowsIn {
    float* x;
    long long stride;
    int K, ksplit, rows;
    const float* part;
    const float* norm_w;
    float norm_off, eps, in_scale;
    uint8_t* out;
    size_t piece;
    int out_rows;
};
template <int PIECES, bool PARTS>
static __global__ void __launch_bounds__(256) rows_in(const __grid_constant__ RowsIn R) {
    chain_wait();
    __shared__ float red[8];
    const int row = blockIdx.x, K = R.K;
    float* src = R.x + (size_t)row * R.stride;
    float r = 1.f;
    if (R.norm_w) {
        float s = 0.f;
        for (int c = threadIdx.x * 4; c < K; c += 1024) {
            float4 a = *reinterpret_cast<const float4*>(src + c);
            if (PARTS) {
                const float* p = R.part + (size_t)row * K + c;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int z = 0; z < R.ksplit; z++, p += (size_t)R.rows * K) {
                    const float4 b = *reinterpret_cast<const float4*>(p);
                    v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
                }
                a = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
                *reinterpret_cast<float4*>(src + c) = a;
            }
            s += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
        }
        s = block_sum(s, red);                     // (its barriers also publish the stored row to the block)
        r = rsqrtf(s / (float)K + R.eps) * R.in_scale;
    }
    for (int c = threadIdx.x * 8; c < K; c += 2048) {
        const float4 a = *reinterpret_cast<const float4*>(src + c), b = *reinterpret_cast<const float4*>(src + c + 4);
        float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (R.norm_w) {
            const float4 wa = __ldg(reinterpret_cast<const float4*>(R.norm_w + c)), wb = __ldg(reinterpret_cast<const float4*>(R.norm_w + c + 4));
            const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = v[i] * r * (R.norm_off + w[i]);
        }
        store_slab8<PIECES>(R.out, R.piece, R.out_rows, row, c, v);
    }
}

// Row r = sequence * L + position of every array below; tokens are [L][M] (step-major, as mk_stage_args.tokens_in).
static __global__ void __launch_bounds__(256) embed_rows(const __nv_bfloat16* table, const int* tokens, int M, int L, int H, int vocab, float scale, float* h) {
    chain_wait();
    const int row = blockIdx.x, m = row / L, l = row - m * L;
    const int tok = max(0, min(vocab - 1, tokens[(size_t)l * M + m]));
    const uint32_t* src = reinterpret_cast<const uint32_t*>(table + (size_t)tok * H);
    float2* dst = reinterpret_cast<float2*>(h + (size_t)row * H);
    for (int c = threadIdx.x; c < H / 2; c += 256) {
        const uint32_t w = __ldg(src + c);
        float lo = bf_lo(w), hi = bf_hi(w);
        if (scale != 0.f) {
            lo = round_bf16(lo * scale);
            hi = round_bf16(hi * scale);
        }
        dst[c] = make_float2(lo, hi);
    }
}

// The last position of every sequence: its residual and the sums of squares per 16 elements, where a decode step leaves them.
static __global__ void __launch_bounds__(256) last_rows(const float* h, int L, int H, float* out, float* ssq) {
    chain_wait();
    const int m = blockIdx.x;
    const float* src = h + ((size_t)m * L + L - 1) * H;
    for (int g = threadIdx.x; g < H / 16; g += 256) {
        float s = 0.f;
        for (int i = 0; i < 16; i++) {
            const float v = src[g * 16 + i];
            out[(size_t)m * H + g * 16 + i] = v;
            s += v * v;
        }
        ssq[(size_t)m * (H / 16) + g] = s;
    }
}

static __global__ void advance_pos(int* pos, int M, int L) {
    chain_wait();
    if ((int)threadIdx.x < M) pos[threadIdx.x] += L;
}

// out = (base + rms(a) w_a [+ rms(b) w_b]) * scale
static __global__ void __launch_bounds__(256) vec_rows(int N, const float* base, const float* a, const float* wa, const float* b, const float* wb, float off, float eps,
                                                float scale, float* out) {
    chain_wait();
    __shared__ float red[8];
    const size_t o = (size_t)blockIdx.x * N;
    float sa = 0.f, sb = 0.f;
    for (int c = threadIdx.x; c < N; c += 256) {
        sa += a[o + c] * a[o + c];
        if (b) sb += b[o + c] * b[o + c];
    }
    const float ra = rsqrtf(block_sum(sa, red) / (float)N + eps);
    const float rb = b ? rsqrtf(block_sum(sb, red) / (float)N + eps) : 0.f;
    for (int c = threadIdx.x; c < N; c += 256) {
        float r = a[o + c] * ra * (off + wa[c]);
        if (b) r += b[o + c] * rb * (off + wb[c]);
        if (base) r += base[o + c];
        out[o + c] = r * scale;
    }
}

// ---- Gated DeltaNet ----------------------------------------------------------------------------------------
struct GdnArgs {
    const float* y;              // in-projection rows
    long long y_stride;
    int M, L, nkh, nvh, conv_dim;
    int q_off, k_off, v_off, z_off, b_off, a_off;
    const float *conv_w, *A_log, *dt_bias, *norm_w;
    float* conv_state;           // history rings; see `conv_slot`
    int ring, layout;            // ring length; 0: [M][conv_dim][ring], 1: the 0.8B kernel's per-task copies, 2: its per-head batched layout
    float* ssm;                  // [M][nvh][128 v][128 k]
    const int* pos;              // position of each sequence's first row
    int conv_bf16, l2_clamp;
    float eps, norm_eps;         // of the L2 norms, of the gated norm
    // scratch
    float* qkv;                  // [rows][conv_dim]: normalised q, k, and v
    float4* scal;                // [rows][nvh]: decay, beta
    float* gram;                 // [M][blocks of 8 positions][nvh][GRAM]: see gdn_gram
    float* o;                    // [rows][nvh * 128]
    uint8_t* out;                // slabs of the gated output
    size_t out_piece;
    int out_rows;
};

// Where the history of channel `ch` (q | k | v order) of sequence m lives; the 0.8B kernels keep q and k once per
// recurrence task of the head (8 of them), of which task `copy` is meant.
__device__ __forceinline__ float* conv_slot(const GdnArgs& G, int m, int ch, int copy) {
    const int qk = G.nkh * 128;
    if (G.layout == 0) return G.conv_state + ((size_t)m * G.conv_dim + ch) * G.ring;
    const int part = ch < qk ? 0 : (ch < 2 * qk ? 1 : 2), c = ch - part * qk, h = c >> 7, i = c & 127;
    if (G.layout == 2) return G.conv_state + (((size_t)m * G.nvh + h) * 384 + part * 128 + i) * G.ring;
    const int task = h * 8 + (part == 2 ? i >> 4 : copy);
    return G.conv_state + ((size_t)task * 272 + (part == 2 ? 256 + (i & 15) : part * 128 + i)) * G.ring;
}

// Causal conv1d + SiLU of every channel, L2 norms of q and k, and the scalars of the recurrence.  One warp per 128
// channels and CONV_ROWS consecutive rows, four channels per lane: the window slides through registers, so an input is read
// CONV_ROWS + 3 times in CONV_ROWS rows instead of four times a row.  (Eight rows a warp were a chain of 16 us whatever the shape; two are
// 1 to 3 % of a pass, one takes longer again.)
constexpr int CONV_ROWS = 2;
static __global__ void __launch_bounds__(256) gdn_conv(const __grid_constant__ GdnArgs G) {
    chain_wait();
    const int groups = (G.L + CONV_ROWS - 1) / CONV_ROWS, m = blockIdx.y / groups, l0 = (blockIdx.y - m * groups) * CONV_ROWS, lane = threadIdx.x & 31;
    const int blk = blockIdx.x * 8 + (threadIdx.x >> 5);                    // 128-channel block: q heads, k heads, v heads
    if (blk * 128 >= G.conv_dim) return;
    const int part = blk < G.nkh ? 0 : (blk < 2 * G.nkh ? 1 : 2);
    const int head = blk - part * G.nkh;
    const int col = (part == 0 ? G.q_off : (part == 1 ? G.k_off : G.v_off)) + head * 128 + 4 * lane;
    const int ch = blk * 128 + 4 * lane, pos = G.pos[m];
    const float* y = G.y + (size_t)m * G.L * G.y_stride + col;
    float w[4][4], x[4][4];                                                 // [tap][channel], oldest first
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(G.conv_w) + ch + i);
        w[0][i] = a.x; w[1][i] = a.y; w[2][i] = a.z; w[3][i] = a.w;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int l = l0 - 3 + d;
        if (l >= 0) {
            const float4 a = *reinterpret_cast<const float4*>(y + (size_t)l * G.y_stride);
            x[d + 1][0] = a.x; x[d + 1][1] = a.y; x[d + 1][2] = a.z; x[d + 1][3] = a.w;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (G.conv_bf16) x[d + 1][i] = round_bf16(x[d + 1][i]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) x[d + 1][i] = conv_slot(G, m, ch + i, 0)[(pos + l) & (G.ring - 1)];
        }
    }
    float4 in[CONV_ROWS];
#pragma unroll
    for (int r = 0; r < CONV_ROWS; r++)
        if (l0 + r < G.L) in[r] = *reinterpret_cast<const float4*>(y + (size_t)(l0 + r) * G.y_stride);
#pragma unroll
    for (int r = 0; r < CONV_ROWS; r++) {
        if (l0 + r >= G.L) break;
        const size_t row = (size_t)m * G.L + l0 + r;
        const float now[4] = {in[r].x, in[r].y, in[r].z, in[r].w};
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            x[0][i] = x[1][i]; x[1][i] = x[2][i]; x[2][i] = x[3][i];
            float a = x[0][i] * w[0][i];
            a = fmaf(x[1][i], w[1][i], a);
            a = fmaf(x[2][i], w[2][i], a);
            a = fmaf(now[i], w[3][i], a);
            x[3][i] = G.conv_bf16 ? round_bf16(now[i]) : now[i];
            v[i] = silu_f(a);
        }
        if (part < 2) {
            const float s = warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]);
            float inv = G.l2_clamp ? 1.f / fmaxf(sqrtf(s), G.eps) : 1.f / sqrtf(s + G.eps);
            if (part == 0) inv *= 0.08838834764831845f;                     // 128^-0.5
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] *= inv;
        }
        *reinterpret_cast<float4*>(G.qkv + row * G.conv_dim + ch) = make_float4(v[0], v[1], v[2], v[3]);
        if (part == 2 && lane == 0) {
            const float b = G.y[row * G.y_stride + G.b_off + head], a = G.y[row * G.y_stride + G.a_off + head];
            G.scal[row * G.nvh + head] = make_float4(expf(-expf(G.A_log[head]) * softplus_f(a + G.dt_bias[head])), sigmoid_f(b), 0.f, 0.f);
        }
    }
}

// The last `ring` inputs of every channel go back into the history rings, 128 channels of one ring slot per block.  Only after
// gdn_conv has read them: gdn_gram's last blocks do it.
__device__ __forceinline__ void put_history(const GdnArgs& G, int block) {
    const int per = (G.conv_dim + 127) / 128, ch = block % per * 128 + threadIdx.x, z = block / per % G.ring, m = block / (per * G.ring), l = G.L - 1 - z;
    if (ch >= G.conv_dim || l < 0) return;
    const int qk = G.nkh * 128, part = ch < qk ? 0 : (ch < 2 * qk ? 1 : 2);
    const int col = (part == 0 ? G.q_off : (part == 1 ? G.k_off : G.v_off)) + ch - part * qk;
    float v = G.y[((size_t)m * G.L + l) * G.y_stride + col];
    if (G.conv_bf16) v = round_bf16(v);
    const int slot = (G.pos[m] + l) & (G.ring - 1), copies = G.layout == 1 && part < 2 ? 8 : 1;
    for (int c = 0; c < copies; c++) conv_slot(G, m, ch, c)[slot] = v;
}

// The recurrence  s <- d s + beta (v - d s k) k,  o = s q  runs in blocks of SCAN = 8 positions.  With s the state before
// the block, P_t the product of its first t decays and delta_t = beta_t (v_t - the state's recall of k_t),
//     recall_t = P_t (s k_t) + sum_{i < t} (P_t / P_i) delta_i (k_i k_t)      o_t = P_t (s q_t) + sum_{i <= t} (P_t / P_i) delta_i (k_i q_t)
//     s       <- P_8 s + sum_i (P_8 / P_i) delta_i k_i,
// so the sixteen products s k_t, s q_t of a block reduce together instead of one by one, and what is sequential are eight
// scalar steps.
constexpr int SCAN = 8;
// Per block and value head: k_i k_t (i < t) and q_i k_t (i >= t) with the decays between the two positions, [t][i], then
// P_t, P_8 / P_t and beta_t (a position past the end decays by 1 and corrects by 0).  One warp per block and key head.
constexpr int GRAM = SCAN * SCAN + 3 * SCAN;
static __global__ void __launch_bounds__(128) gdn_gram(const __grid_constant__ GdnArgs G) {
    chain_wait();
    const int w = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, chunks = (G.L + SCAN - 1) / SCAN, blocks = (G.M * chunks * G.nkh + 3) / 4;
    if ((int)blockIdx.x >= blocks) {
        put_history(G, blockIdx.x - blocks);
        return;
    }
    if (w >= G.M * chunks * G.nkh) return;
    const int kh = w % G.nkh, c = (w / G.nkh) % chunks, m = w / (G.nkh * chunks), rep = G.nvh / G.nkh;
    float4 q[SCAN], k[SCAN];
#pragma unroll
    for (int t = 0; t < SCAN; t++) {
        q[t] = k[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int l = c * SCAN + t;
        if (l < G.L) {
            const float4* src = reinterpret_cast<const float4*>(G.qkv + ((size_t)m * G.L + l) * G.conv_dim + kh * 128) + lane;
            q[t] = src[0];
            k[t] = src[G.nkh * 32];
        }
    }
    float v[SCAN * SCAN];
#pragma unroll
    for (int t = 0; t < SCAN; t++)
#pragma unroll
        for (int i = 0; i < SCAN; i++) {
            const float4 a = k[t], b = i < t ? k[i] : q[i];
            v[t * SCAN + i] = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));
        }
#pragma unroll
    for (int o = 16, n = 32; o; o >>= 1, n >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (j < n) {
                const float send = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
                v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    // per value head: entry (t, i) takes the decays between the two positions
    for (int r = 0; r < rep; r++) {
        const int h = kh * rep + r, l = c * SCAN + (lane & 7);
        const float4 sc = l < G.L ? G.scal[((size_t)m * G.L + l) * G.nvh + h] : make_float4(1.f, 0.f, 0.f, 0.f);
        const float dec = sc.x;
        float d0 = 1.f, d1 = 1.f, p = 1.f;
        const int t = lane >> 2, i = (lane & 3) * 2;
#pragma unroll
        for (int j = 0; j < SCAN; j++) {
            const float dj = __shfl_sync(0xffffffffu, dec, j);
            d0 *= j > min(t, i) && j <= max(t, i) ? dj : 1.f;
            d1 *= j > min(t, i + 1) && j <= max(t, i + 1) ? dj : 1.f;
            p *= (lane < 8 ? j <= lane : j > (lane & 7)) ? dj : 1.f;
        }
        float* out = G.gram + (((size_t)m * chunks + c) * G.nvh + h) * GRAM;
        *reinterpret_cast<float2*>(out + 2 * lane) = make_float2(v[0] * d0, v[1] * d1);
        if (lane < 24) out[64 + lane] = lane < 16 ? p : sc.y;
    }
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 both(float a) { return ((u64)__float_as_uint(a) << 32) | __float_as_uint(a); }
__device__ __forceinline__ float sum2(u64 a) { return __uint_as_float((uint32_t)a) + __uint_as_float((uint32_t)(a >> 32)); }

// Four warps; sixteen lanes share two value rows of one head of one sequence (eight keys each, in registers, packed in pairs), so
// a CTA holds 16 rows and a head is eight CTAs.  What bounds a block is shared memory: a 16-byte read is four of its cycles, and
// every lane reads its keys of eight k and eight q.  Two rows a lane halve the reads per product, and the k's stay in registers
// for the update.  16 heads x 511 positions: 54 us (69 with eight lanes to one row; 207 position by position).
template <bool FOUR>      // four CTAs per SM
static __global__ void __launch_bounds__(128, FOUR ? 4 : 0) gdn_scan(const __grid_constant__ GdnArgs G) {
    chain_wait();
    constexpr int ROWS = 16, IN = 256 + ROWS;
    __shared__ __align__(16) float in_s[2][SCAN][IN];        // q | k | values
    __shared__ __align__(16) float mats[2][GRAM];            // what gdn_gram left for the block
    const int rep = G.nvh / G.nkh;
    const int m = blockIdx.z, h = blockIdx.y, v0 = blockIdx.x * ROWS, kh = h / rep;
    const int tid = threadIdx.x, part = tid & 15, r0 = (tid >> 4) * 2;       // the lanes' rows r0, r0 + 1; keys part * 4 + 64 i + {0..3}
    const int chunks = (G.L + SCAN - 1) / SCAN, key_dim = G.nkh * 128;
    float* st = G.ssm + (((size_t)m * G.nvh + h) * 128 + v0 + r0) * 128 + part * 4;
    u64 s[2][4];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(st + r * 128 + 64 * i);
            s[r][2 * i] = a.x;
            s[r][2 * i + 1] = a.y;
        }
    const size_t row0 = (size_t)m * G.L;
    const float* qk_src = G.qkv + row0 * G.conv_dim + ((tid & 32) ? key_dim : 0) + kh * 128 + 4 * (tid & 31);
    const float* v_src = G.qkv + row0 * G.conv_dim + 2 * key_dim + h * 128 + v0 + 4 * (tid & 3);
    const float* m_src = G.gram + ((size_t)m * chunks * G.nvh + h) * GRAM + 4 * (tid - 64);
    auto request = [&](int buf, int c) {
        const int l0 = c * SCAN;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int b = (tid >> 6) + 2 * j;
            mk::cp_async16(&in_s[buf][b][4 * (tid & 63)], qk_src + (size_t)min(l0 + b, G.L - 1) * G.conv_dim);
        }
        if (tid < 4 * SCAN) mk::cp_async16(&in_s[buf][tid >> 2][256 + 4 * (tid & 3)], v_src + (size_t)min(l0 + (tid >> 2), G.L - 1) * G.conv_dim);
        if (tid >= 64 && tid < 64 + GRAM / 4) mk::cp_async16(&mats[buf][4 * (tid - 64)], m_src + (size_t)c * G.nvh * GRAM);
        mk::cp_async_commit();
    };
    request(0, 0);
    const int mine = (part >> 3) & 1, mt = part & 7;                        // the row and the position whose products this lane ends up with
    float* o = G.o + row0 * (size_t)(G.nvh * 128) + h * 128 + v0 + r0 + mine;
#pragma unroll 1
    for (int c = 0, buf = 0; c < chunks; c++, buf ^= 1) {
        mk::cp_async_wait_all();
        __syncthreads();
        if (c + 1 < chunks) request(buf ^ 1, c + 1);
        const float* mat_s = mats[buf];
        // s k_t, s q_t of both rows over this lane's keys: value r * 16 + 2 t (k) and + 1 (q)
        u64 k[SCAN][4];
        float u[32];
#pragma unroll
        for (int t = 0; t < SCAN; t++) {
            const float* q = in_s[buf][t] + part * 4;
            const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(q + 128), k1 = *reinterpret_cast<const ulonglong2*>(q + 192);
            const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(q), q1 = *reinterpret_cast<const ulonglong2*>(q + 64);
            k[t][0] = k0.x; k[t][1] = k0.y; k[t][2] = k1.x; k[t][3] = k1.y;
#pragma unroll
            for (int r = 0; r < 2; r++) {
                u[16 * r + 2 * t] = sum2(fma2(s[r][3], k1.y, fma2(s[r][2], k1.x, fma2(s[r][1], k0.y, mul2(s[r][0], k0.x)))));
                u[16 * r + 2 * t + 1] = sum2(fma2(s[r][3], q1.y, fma2(s[r][2], q1.x, fma2(s[r][1], q0.y, mul2(s[r][0], q0.x)))));
            }
        }
        // sums over the sixteen lanes; every step halves what a lane carries
#pragma unroll
        for (int x = 8, n = 16; x; x >>= 1, n >>= 1) {
            const bool up = part & x;
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (j < n) {
                    const float send = up ? u[j] : u[j + n], keep = up ? u[j + n] : u[j];
                    u[j] = keep + __shfl_xor_sync(0xffffffffu, send, x);
                }
        }
        // the eight corrections of this lane's row, one after the other
        float delta[SCAN];
#pragma unroll
        for (int t = 0; t < SCAN; t++) {
            float recall = __shfl_sync(0xffffffffu, u[0], (tid & 24) | t) * mat_s[64 + t];
#pragma unroll
            for (int i = 0; i < SCAN; i++)
                if (i < t) recall = fmaf(mat_s[t * 8 + i], delta[i], recall);
            delta[t] = (in_s[buf][t][256 + r0 + mine] - recall) * mat_s[80 + t];
        }
        {
            float y = u[1] * mat_s[64 + mt];
#pragma unroll
            for (int i = 0; i < SCAN; i++)
                if (i <= mt) y = fmaf(mat_s[i * 8 + mt], delta[i], y);
            if (c * SCAN + mt < G.L) o[(size_t)(c * SCAN + mt) * (G.nvh * 128)] = y;
        }
        const u64 p = both(mat_s[64 + SCAN - 1]);
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int i = 0; i < 4; i++) s[r][i] = mul2(s[r][i], p);
#pragma unroll
        for (int t = 0; t < SCAN; t++) {
            const float e = delta[t] * mat_s[72 + t], other = __shfl_xor_sync(0xffffffffu, e, 8);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const u64 f = both(mine == r ? e : other);
#pragma unroll
                for (int i = 0; i < 4; i++) s[r][i] = fma2(k[t][i], f, s[r][i]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int i = 0; i < 2; i++) *reinterpret_cast<ulonglong2*>(st + r * 128 + 64 * i) = make_ulonglong2(s[r][2 * i], s[r][2 * i + 1]);
}

// Gated RMSNorm per head, into slabs: one half warp per head and row (eight columns per lane).
template <int PIECES>
static __global__ void __launch_bounds__(256) gdn_gate(const __grid_constant__ GdnArgs G) {
    chain_wait();
    const int row = blockIdx.y, h = blockIdx.x * 16 + (threadIdx.x >> 4), i = (threadIdx.x & 15) * 8;
    if (h >= G.nvh) return;
    const float* o = G.o + (size_t)row * (G.nvh * 128) + h * 128 + i;
    const float* z = G.y + (size_t)row * G.y_stride + G.z_off + h * 128 + i;
    float v[8], s = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        v[j] = o[j];
        s = fmaf(v[j], v[j], s);
    }
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
#pragma unroll
    for (int x = 8; x; x >>= 1) s += __shfl_xor_sync(mask, s, x);
    const float r = rsqrtf(s / 128.f + G.norm_eps);
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = v[j] * r * __ldg(G.norm_w + i + j) * (z[j] * sigmoid_f(z[j]));
    store_slab8<PIECES>(G.out, G.out_piece, G.out_rows, row, h * 128 + i, v);
}

// ---- attention -----------------------------------------------------------------------------------------------
struct AttnArgs {
    const float* y;
    long long y_stride;
    int M, L, nq, nkv;
    int q_off, q_hs, gate_off, k_off, v_off;
    int rot, pairs, window, q_bf16, norm_plain, v_norm;
    float eps, scale;
    const float *q_norm, *k_norm, *cos, *sin;
    void *k_cache, *v_cache;
    const int* bt;
    int max_pages, kv_shift;
    uint32_t s_page, s_head, s_pos;
    const int* pos;
    void* q;                     // [rows][nq][HD] prepared queries, bf16 (attn_rows) or fp32 (attn_rows_f32)
    float q_scale;               // fp32 queries: factor applied after the rotation
    uint8_t* out;                // slabs of the (gated) output
    size_t out_piece;
    int out_rows;
};

__device__ __forceinline__ size_t kv_offset(const AttnArgs& T, int m, int kvh, int p) {
    const int page = __ldg(T.bt + (size_t)m * T.max_pages + (p >> T.kv_shift));
    return (size_t)((uint32_t)page * T.s_page + (uint32_t)kvh * T.s_head + (uint32_t)(p & ((1 << T.kv_shift) - 1)) * T.s_pos);
}

// Norm, rotation and rounding of every head vector of a row: queries to `q`, keys and values into the paged cache.
// One warp per head vector; lane i holds dims i + 32 j, so both halves of a rotated pair are in one lane.
template <int HD, bool QF32, bool KVF32>
static __global__ void __launch_bounds__(256) attn_prepare(const __grid_constant__ AttnArgs T) {
    chain_wait();
    constexpr int N = HD / 32;
    const int row = blockIdx.y, m = row / T.L, lane = threadIdx.x & 31;
    const int hv = blockIdx.x * 8 + (threadIdx.x >> 5);                 // q heads, k heads, v heads
    if (hv >= T.nq + 2 * T.nkv) return;
    const int kind = hv < T.nq ? 0 : (hv < T.nq + T.nkv ? 1 : 2);
    const int head = kind == 0 ? hv : (kind == 1 ? hv - T.nq : hv - T.nq - T.nkv);
    const float* y = T.y + (size_t)row * T.y_stride;
    const float* src = kind == 0 ? y + T.q_off + (size_t)head * T.q_hs
                                 : (kind == 1 || T.v_off < 0 ? y + T.k_off + (size_t)head * HD : y + T.v_off + (size_t)head * HD);
    const int pos = T.pos[m] + (row - m * T.L);
    float v[N], s = 0.f;
#pragma unroll
    for (int j = 0; j < N; j++) {
        v[j] = src[lane + 32 * j];
        s = fmaf(v[j], v[j], s);
    }
    const float* nw = kind == 0 ? T.q_norm : (kind == 1 ? T.k_norm : nullptr);
    const float off = T.norm_plain ? 0.f : 1.f;
    if (kind < 2 || T.v_norm) {
        const float r = rsqrtf(warp_sum(s) / (float)HD + T.eps);
#pragma unroll
        for (int j = 0; j < N; j++) v[j] = v[j] * r * (nw ? off + __ldg(nw + lane + 32 * j) : 1.f);
    }
    if (kind < 2) {
        const int pd = T.rot == HD ? HD / 64 : T.rot / 64;               // distance of a pair in units of 32 dims
#pragma unroll
        for (int j = 0; j < N / 2; j++)
            if (j < pd && lane + 32 * j < T.pairs) {
                const size_t o = (size_t)pos * T.pairs + lane + 32 * j;
                const float c = __ldg(T.cos + o), sn = __ldg(T.sin + o);
#pragma unroll
                for (int d = 1; d <= N / 2; d++)                          // static register indexes
                    if (d == pd) {
                        const float a = v[j], b = v[j + d];
                        v[j] = a * c - b * sn;
                        v[j + d] = b * c + a * sn;
                    }
            }
    }
    const size_t o = kind == 0 ? ((size_t)row * T.nq + head) * HD : kv_offset(T, m, head, pos);
    void* dst = kind == 0 ? T.q : (kind == 1 ? T.k_cache : T.v_cache);
    if (kind == 0 ? QF32 : KVF32) {
        const float f = kind == 0 ? T.q_scale : 1.f;
#pragma unroll
        for (int j = 0; j < N; j++) reinterpret_cast<float*>(dst)[o + lane + 32 * j] = v[j] * f;
    } else {
#pragma unroll
        for (int j = 0; j < N; j++) reinterpret_cast<__nv_bfloat16*>(dst)[o + lane + 32 * j] = __float2bfloat16_rn(v[j]);
    }
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp16_zfill(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Causal attention of a block of positions over the paged bf16 cache.  A CTA owns one KV head of one sequence and
// 64 query rows (position, head of the group); blocks of 64 keys pass through shared memory.  Warp (r, d): rows 16 r ..
// 16 r + 15; it scores keys 32 d .. 32 d + 31 of the block and accumulates head dims [d HD / 2, (d + 1) HD / 2).
// Probabilities enter the second product as three bf16 pieces (24 bits), so only Q, K and V carry bf16 roundings, as in
// the decode step.  V arrives while the scores are computed, the next K while P x V runs.
constexpr int AT_ROWS = 64, AT_KEYS = 64, AT_PIECES = 3;
template <int HD> constexpr int attn_smem() { return 3 * AT_ROWS * HD * 2 + AT_PIECES * AT_ROWS * AT_KEYS * 2 + 4 * AT_ROWS * 4; }
template <int HD>
static __global__ void __launch_bounds__(256, 1) attn_rows(const __grid_constant__ AttnArgs T) {
    chain_wait();
    extern __shared__ __align__(128) uint8_t sm[];
    constexpr int RB = HD * 2, CH = RB / 16;                             // bytes and 16-byte pieces of a row
    uint8_t *q_s = sm, *k_s = q_s + AT_ROWS * RB, *v_s = k_s + AT_KEYS * RB, *p_s = v_s + AT_KEYS * RB;
    float* st_s = reinterpret_cast<float*>(p_s + AT_PIECES * AT_ROWS * AT_KEYS * 2);   // [2][64] maxima, [2][64] sums
    const int qpk = T.nq / T.nkv, bq = AT_ROWS / qpk;
    const int m = blockIdx.z, kvh = blockIdx.y, l0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * bq;      // long ones first
    const int np = min(bq, T.L - l0), pos0 = T.pos[m] + l0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rg = warp & 3, dh = warp >> 2, g = lane >> 2, t = lane & 3;
    // keys outside [low, last] are zeros and their pages are not touched: before a window there may be anything
    const int last = pos0 + np - 1, low = T.window ? max(0, pos0 - T.window + 1) : 0, first = low & ~(AT_KEYS - 1);
    const __nv_bfloat16 *kc = reinterpret_cast<const __nv_bfloat16*>(T.k_cache), *vc = reinterpret_cast<const __nv_bfloat16*>(T.v_cache);
    auto load_kv = [&](uint8_t* dst, const __nv_bfloat16* cache, int k0) {
#pragma unroll 4
        for (int i = tid; i < AT_KEYS * CH; i += 256) {
            const int key = i / CH, c = i - key * CH, p = k0 + key;
            cp16_zfill(smem_u32(dst + (size_t)key * RB + (((c & ~7) | ((c ^ key) & 7)) << 4)), cache + kv_offset(T, m, kvh, min(max(p, low), last)) + c * 8, p >= low && p <= last);
        }
        mk::cp_async_commit();
    };
    for (int i = tid; i < AT_ROWS * CH; i += 256) {
        const int r = i / CH, c = i - r * CH, p = r / qpk, hq = r - p * qpk;
        const bool live = p < np;
        const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(T.q) + (((size_t)m * T.L + l0 + (live ? p : 0)) * T.nq + kvh * qpk + hq) * HD + c * 8;
        cp16_zfill(smem_u32(q_s + (size_t)r * RB + (((c & ~7) | ((c ^ r) & 7)) << 4)), src, live);
    }
    load_kv(k_s, kc, first);
    float o[HD / 16][4], mx[2] = {-3.0e38f, -3.0e38f}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < HD / 16; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    int qp[2];                                                           // positions of this lane's two rows
#pragma unroll
    for (int i = 0; i < 2; i++) qp[i] = pos0 + min((16 * rg + g + 8 * i) / qpk, np - 1);
    const uint32_t qa = smem_u32(q_s) + (uint32_t)(16 * rg + (lane & 15)) * RB, qx = (lane & 7);
#pragma unroll 1
    for (int k0 = first; k0 <= last; k0 += AT_KEYS) {
        cp_wait<0>();
        __syncthreads();                                                 // K is here; everybody is done with V and P
        load_kv(v_s, vc, k0);
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll 4
        for (int kk = 0; kk < HD / 16; kk++) {
            uint32_t a[4];
            const uint32_t ca = 2 * kk + (lane >> 4);
            ldsm4(a, qa + (((ca & ~7u) | ((ca ^ qx) & 7)) << 4));
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const uint32_t key = 32 * dh + 16 * n + (lane & 7) + ((lane >> 4) << 3), cb = 2 * kk + ((lane >> 3) & 1);
                uint32_t b[4];
                ldsm4(b, smem_u32(k_s) + key * RB + (((cb & ~7u) | ((cb ^ key) & 7)) << 4));
                mma16816(s[2 * n], a, b[0], b[1]);
                mma16816(s[2 * n + 1], a, b[2], b[3]);
            }
        }
        // mask, scale, running maximum over both key halves
        float bm[2] = {-3.0e38f, -3.0e38f};
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int p = k0 + 32 * dh + 8 * n + 2 * t + (i & 1), r = i >> 1;
                const bool seen = p <= qp[r] && (!T.window || p > qp[r] - T.window);
                s[n][i] = seen ? s[n][i] * T.scale : -3.0e38f;
                bm[r] = fmaxf(bm[r], s[n][i]);
            }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            bm[r] = fmaxf(bm[r], __shfl_xor_sync(0xffffffffu, bm[r], 1));
            bm[r] = fmaxf(bm[r], __shfl_xor_sync(0xffffffffu, bm[r], 2));
            if (t == 0) st_s[dh * AT_ROWS + 16 * rg + g + 8 * r] = bm[r];
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + rg) : "memory");        // the two warps of these rows
        float f[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float nm = fmaxf(mx[r], fmaxf(bm[r], st_s[(dh ^ 1) * AT_ROWS + 16 * rg + g + 8 * r]));
            f[r] = __expf(mx[r] - nm);
            mx[r] = nm;
            sum[r] *= f[r];
        }
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                float p0 = s[n][2 * r] > -2.9e38f ? __expf(s[n][2 * r] - mx[r]) : 0.f, p1 = s[n][2 * r + 1] > -2.9e38f ? __expf(s[n][2 * r + 1] - mx[r]) : 0.f;
                sum[r] += p0 + p1;
                const uint32_t row = 16 * rg + g + 8 * r, c = 4 * dh + n;
#pragma unroll
                for (int q = 0; q < AT_PIECES; q++) {
                    const uint32_t w = pack_bf16(p0, p1);
                    *reinterpret_cast<uint32_t*>(p_s + q * AT_ROWS * AT_KEYS * 2 + row * 128 + ((c ^ (row & 7)) << 4) + t * 4) = w;
                    p0 -= bf_lo(w);
                    p1 -= bf_hi(w);
                }
            }
#pragma unroll
        for (int i = 0; i < HD / 16; i++) {
            o[i][0] *= f[0]; o[i][1] *= f[0];
            o[i][2] *= f[1]; o[i][3] *= f[1];
        }
        cp_wait<0>();
        __syncthreads();                                                 // V and P are here; everybody is done with K
        if (k0 + AT_KEYS <= last) load_kv(k_s, kc, k0 + AT_KEYS);
#pragma unroll
        for (int kk = 0; kk < AT_KEYS / 16; kk++) {
            uint32_t a[AT_PIECES][4];
#pragma unroll
            for (int q = 0; q < AT_PIECES; q++)
                ldsm4(a[q], smem_u32(p_s) + q * AT_ROWS * AT_KEYS * 2 + (uint32_t)(16 * rg + (lane & 15)) * 128 + (((2 * kk + (lane >> 4)) ^ qx) << 4));
#pragma unroll
            for (int n = 0; n < HD / 32; n++) {
                const uint32_t key = 16 * kk + (lane & 15), c = dh * (CH / 2) + 2 * n + (lane >> 4);
                uint32_t b[4];
                ldsm4_t(b, smem_u32(v_s) + key * RB + (((c & ~7u) | ((c ^ key) & 7)) << 4));
#pragma unroll
                for (int q = 0; q < AT_PIECES; q++) {
                    mma16816(o[2 * n], a[q], b[0], b[1]);
                    mma16816(o[2 * n + 1], a[q], b[2], b[3]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
        if (t == 0) st_s[(2 + dh) * AT_ROWS + 16 * rg + g + 8 * r] = sum[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int rr = 16 * rg + g + 8 * r, p = rr / qpk, hq = kvh * qpk + rr - p * qpk;
        if (p >= np) continue;
        const float inv = 1.f / (st_s[2 * AT_ROWS + rr] + st_s[3 * AT_ROWS + rr]);
        const int row = m * T.L + l0 + p;
        const float* gate = T.gate_off >= 0 ? T.y + (size_t)row * T.y_stride + T.q_off + (size_t)hq * T.q_hs + T.gate_off : nullptr;
#pragma unroll
        for (int n = 0; n < HD / 16; n++) {
            const int dim = dh * (HD / 2) + 8 * n + 2 * t;
            float a = o[n][2 * r] * inv, b = o[n][2 * r + 1] * inv;
            if (gate) {
                a *= sigmoid_f(gate[dim]);
                b *= sigmoid_f(gate[dim + 1]);
            }
            *reinterpret_cast<uint32_t*>(T.out + slab_offset(T.out_rows, row, hq * HD + dim)) = pack_bf16(a, b);
        }
    }
}

// The same for the 0.8B model, whose attention is exact to fp32: queries, probabilities and an fp32 cache enter the
// tensor cores as three bf16 pieces each, and of the nine piece products the six that reach above 2^-24 are formed (a
// bf16 cache is one piece: three products).  32 query rows per CTA (a 500-token prompt is then one CTA per SM), blocks of 32
// keys: warp (r, d) takes rows 16 r .. 16 r + 15, scores keys 8 d .. 8 d + 7 and accumulates head dims 64 d .. 64 d + 63.
// The fp32 rows of the next block wait in registers.
//   A block of keys takes 6 us, bound by the chain load - split - two products with a barrier each at one CTA per SM, and the last
// rows see all of them.  So the CTAs of a cluster share a row block's keys (attn_splits), and the first one adds the others'
// sums through distributed shared memory.
__device__ __forceinline__ int cluster_size() { uint32_t v; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(v)); return (int)v; }
__device__ __forceinline__ int cluster_rank() { uint32_t v; asm("mov.u32 %0, %%cluster_ctaid.x;" : "=r"(v)); return (int)v; }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float cluster_f1(const float* p, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float2 cluster_f2(const float* p, int rank) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(cluster_addr(p, rank)) : "memory");
    return v;
}
constexpr int AF_ROWS = 32, AF_KEYS = 32, AF_HD = 256, AF_RB = AF_HD * 2;
template <bool KVF32> constexpr int attn_f32_smem() { return 3 * AF_ROWS * AF_RB + 2 * (KVF32 ? 3 : 1) * AF_KEYS * AF_RB + 3 * AF_ROWS * AF_KEYS * 2 + 8 * AF_ROWS * 4; }
// Four consecutive columns c .. c + 3 of a row, as NP pieces of swizzled rows
template <int NP>
__device__ __forceinline__ void split4(uint8_t* base, size_t piece, int row, int c, float4 v) {
    uint8_t* dst = base + (size_t)row * AF_RB + ((((c >> 3) & ~7) | (((c >> 3) ^ row) & 7)) << 4) + (c & 4) * 2;
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const uint32_t a = pack_bf16(v.x, v.y), b = pack_bf16(v.z, v.w);
        *reinterpret_cast<uint2*>(dst + p * piece) = make_uint2(a, b);
        v.x -= bf_lo(a); v.y -= bf_hi(a); v.z -= bf_lo(b); v.w -= bf_hi(b);
    }
}
template <bool KVF32>
static __global__ void __launch_bounds__(256, 1) attn_rows_f32(const __grid_constant__ AttnArgs T) {
    chain_wait();
    extern __shared__ __align__(128) uint8_t sm[];
    constexpr int KP = KVF32 ? 3 : 1, QB = AF_ROWS * AF_RB, KB = AF_KEYS * AF_RB, PB = AF_ROWS * AF_KEYS * 2;
    constexpr int PER = AF_KEYS * AF_HD / 4 / 256;                        // groups of four columns per thread and block
    uint8_t *q_s = sm, *k_s = q_s + 3 * QB, *v_s = k_s + KP * KB, *p_s = v_s + KP * KB;
    float* st_s = reinterpret_cast<float*>(p_s + 3 * PB);
    const int qpk = T.nq / T.nkv, bq = AF_ROWS / qpk;
    const int ranks = cluster_size(), rank = cluster_rank();
    const int m = blockIdx.z, kvh = blockIdx.y, l0 = ((int)(gridDim.x - 1 - blockIdx.x) / ranks) * bq;
    const int np = min(bq, T.L - l0), pos0 = T.pos[m] + l0, last = pos0 + np - 1;
    const int share = (last / AF_KEYS + ranks) / ranks * AF_KEYS, first = rank * share, end = min(last + 1, first + share);    // this CTA's keys
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rg = warp & 1, dh = warp >> 1, g = lane >> 2, t = lane & 3;
    auto fetch = [&](const void* cache, int k0, float4 (&r)[PER]) {
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int key = (tid >> 6) + 4 * i, c = (tid & 63) * 4, p = k0 + key;
            r[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p <= last) {
                const size_t o = kv_offset(T, m, kvh, p) + c;
                if (KVF32) r[i] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(cache) + o);
                else {
                    const uint2 w = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(cache) + o);
                    r[i] = make_float4(bf_lo(w.x), bf_hi(w.x), bf_lo(w.y), bf_hi(w.y));
                }
            }
        }
    };
    auto place = [&](uint8_t* dst, const float4 (&r)[PER]) {
#pragma unroll
        for (int i = 0; i < PER; i++) split4<KP>(dst, KB, (tid >> 6) + 4 * i, (tid & 63) * 4, r[i]);
    };
    float4 kr[PER];
    fetch(T.k_cache, first, kr);
    for (int i = tid; i < AF_ROWS * AF_HD / 4; i += 256) {
        const int r = i / (AF_HD / 4), c = (i - r * (AF_HD / 4)) * 4, p = r / qpk, hq = r - p * qpk;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p < np) v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(T.q) + (((size_t)m * T.L + l0 + p) * T.nq + kvh * qpk + hq) * AF_HD + c);
        split4<3>(q_s, QB, r, c, v);
    }
    float o[AF_HD / 32][4], mx[2] = {-3.0e38f, -3.0e38f}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < AF_HD / 32; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    int qp[2];
#pragma unroll
    for (int i = 0; i < 2; i++) qp[i] = pos0 + min((16 * rg + g + 8 * i) / qpk, np - 1);
    const uint32_t qa = smem_u32(q_s) + (uint32_t)(16 * rg + (lane & 15)) * AF_RB, qx = lane & 7;
#pragma unroll 1
    for (int k0 = first; k0 < end; k0 += AF_KEYS) {
        __syncthreads();                                                 // everybody is done with the previous block
        place(k_s, kr);
        float4 vr[PER];
        fetch(T.v_cache, k0, vr);
        __syncthreads();
        float s[4] = {0.f, 0.f, 0.f, 0.f};                               // 16 rows x 8 keys
#pragma unroll 2
        for (int kk = 0; kk < AF_HD / 32; kk++) {
            uint32_t a[2][3][4], b[KP][4];
            const uint32_t key = 8 * dh + (lane & 7), cb = 4 * kk + (lane >> 3);
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const uint32_t ca = 4 * kk + 2 * h + (lane >> 4);
                    ldsm4(a[h][p], qa + p * QB + (((ca & ~7u) | ((ca ^ qx) & 7)) << 4));
                }
#pragma unroll
            for (int p = 0; p < KP; p++) ldsm4(b[p], smem_u32(k_s) + p * KB + key * AF_RB + (((cb & ~7u) | ((cb ^ key) & 7)) << 4));
#pragma unroll
            for (int p = 2; p >= 0; p--)                                  // small products first
#pragma unroll
                for (int r = KP - 1; r >= 0; r--)
                    if (p + r < 3) {
                        mma16816(s, a[0][p], b[r][0], b[r][1]);
                        mma16816(s, a[1][p], b[r][2], b[r][3]);
                    }
        }
        float bm[2] = {-3.0e38f, -3.0e38f};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int p = k0 + 8 * dh + 2 * t + (i & 1), r = i >> 1;
            s[i] = p <= qp[r] ? s[i] : -3.0e38f;
            bm[r] = fmaxf(bm[r], s[i]);
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            bm[r] = fmaxf(bm[r], __shfl_xor_sync(0xffffffffu, bm[r], 1));
            bm[r] = fmaxf(bm[r], __shfl_xor_sync(0xffffffffu, bm[r], 2));
            if (t == 0) st_s[dh * AF_ROWS + 16 * rg + g + 8 * r] = bm[r];
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + rg) : "memory");
        float f[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            float nm = mx[r];
#pragma unroll
            for (int d = 0; d < 4; d++) nm = fmaxf(nm, st_s[d * AF_ROWS + 16 * rg + g + 8 * r]);
            f[r] = __expf(mx[r] - nm);
            mx[r] = nm;
            sum[r] *= f[r];
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            float p0 = s[2 * r] > -2.9e38f ? __expf(s[2 * r] - mx[r]) : 0.f, p1 = s[2 * r + 1] > -2.9e38f ? __expf(s[2 * r + 1] - mx[r]) : 0.f;
            sum[r] += p0 + p1;
            const uint32_t row = 16 * rg + g + 8 * r;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const uint32_t w = pack_bf16(p0, p1);
                *reinterpret_cast<uint32_t*>(p_s + q * PB + row * 64 + ((dh ^ ((row >> 1) & 3)) << 4) + t * 4) = w;
                p0 -= bf_lo(w);
                p1 -= bf_hi(w);
            }
        }
#pragma unroll
        for (int i = 0; i < AF_HD / 32; i++) {
            o[i][0] *= f[0]; o[i][1] *= f[0];
            o[i][2] *= f[1]; o[i][3] *= f[1];
        }
        place(v_s, vr);
        if (k0 + AF_KEYS < end) fetch(T.k_cache, k0 + AF_KEYS, kr);
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < AF_KEYS / 16; kk++) {
            uint32_t a[3][4];
            const uint32_t row = 16 * rg + (lane & 15);
#pragma unroll
            for (int p = 0; p < 3; p++) ldsm4(a[p], smem_u32(p_s) + p * PB + row * 64 + (((2 * kk + (lane >> 4)) ^ ((row >> 1) & 3)) << 4));
#pragma unroll
            for (int n = 0; n < AF_HD / 64; n++) {
                const uint32_t key = 16 * kk + (lane & 15), c = dh * 8 + 2 * n + (lane >> 4);
                uint32_t b[KP][4];
#pragma unroll
                for (int p = 0; p < KP; p++) ldsm4_t(b[p], smem_u32(v_s) + p * KB + key * AF_RB + (((c & ~7u) | ((c ^ key) & 7)) << 4));
#pragma unroll
                for (int p = 2; p >= 0; p--)
#pragma unroll
                    for (int r = KP - 1; r >= 0; r--)
                        if (p + r < 3) {
                            mma16816(o[2 * n], a[p], b[r][0], b[r][1]);
                            mma16816(o[2 * n + 1], a[p], b[r][2], b[r][3]);
                        }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
        if (t == 0) st_s[(4 + dh) * AF_ROWS + 16 * rg + g + 8 * r] = sum[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int rr = 16 * rg + g + 8 * r;
        sum[r] = (st_s[4 * AF_ROWS + rr] + st_s[5 * AF_ROWS + rr]) + (st_s[6 * AF_ROWS + rr] + st_s[7 * AF_ROWS + rr]);
    }
    if (ranks > 1) {                             // the first CTA adds the others' sums to its own
        float* part = reinterpret_cast<float*>(k_s);
        constexpr int PR = AF_HD + 8;            // padded against bank conflicts
        static_assert(AF_ROWS * PR * 4 <= 2 * KP * KB + 3 * PB, "K, V and probabilities are read by now");
        if (rank) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int rr = 16 * rg + g + 8 * r;
#pragma unroll
                for (int n = 0; n < AF_HD / 32; n++)
                    *reinterpret_cast<float2*>(part + rr * PR + dh * (AF_HD / 4) + 8 * n + 2 * t) = make_float2(o[n][2 * r], o[n][2 * r + 1]);
                if (dh == 0 && t == 0) st_s[rr] = mx[r];
                if (dh == 1 && t == 0) st_s[AF_ROWS + rr] = sum[r];
            }
        }
        cluster_sync();
        if (rank == 0) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int rr = 16 * rg + g + 8 * r;
#pragma unroll 1
                for (int c = 1; c < ranks; c++) {
                    const float2 ms = make_float2(cluster_f1(st_s + rr, c), cluster_f1(st_s + AF_ROWS + rr, c));
                    const float nm = fmaxf(mx[r], ms.x), f = __expf(mx[r] - nm), fc = __expf(ms.x - nm);
                    mx[r] = nm;
                    sum[r] = fmaf(sum[r], f, ms.y * fc);
#pragma unroll
                    for (int n = 0; n < AF_HD / 32; n++) {
                        const float2 v = cluster_f2(part + rr * PR + dh * (AF_HD / 4) + 8 * n + 2 * t, c);
                        o[n][2 * r] = fmaf(o[n][2 * r], f, v.x * fc);
                        o[n][2 * r + 1] = fmaf(o[n][2 * r + 1], f, v.y * fc);
                    }
                }
            }
        }
        cluster_sync();                          // their shared memory has been read
        if (rank) return;
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int rr = 16 * rg + g + 8 * r, p = rr / qpk, hq = kvh * qpk + rr - p * qpk;
        if (p >= np) continue;
        const float inv = 1.f / sum[r];
        const int row = m * T.L + l0 + p;
        const float* gate = T.y + (size_t)row * T.y_stride + T.q_off + (size_t)hq * T.q_hs + T.gate_off;
#pragma unroll
        for (int n = 0; n < AF_HD / 32; n++) {
            const int dim = dh * (AF_HD / 4) + 8 * n + 2 * t;
            float a = o[n][2 * r] * inv * sigmoid_f(gate[dim]), b = o[n][2 * r + 1] * inv * sigmoid_f(gate[dim + 1]);
            uint8_t* dst = T.out + slab_offset(T.out_rows, row, hq * AF_HD + dim);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const uint32_t w = pack_bf16(a, b);
                *reinterpret_cast<uint32_t*>(dst + q * T.out_piece) = w;
                a -= bf_lo(w);
                b -= bf_hi(w);
            }
        }
    }
}

// ---- products of a few rows per expert -----------------------------------------------------------------------
// A routed group has a few dozen token rows, so its product is a stream of weights, and what limits it is what happens to a weight on
// the way: through shared memory into the tensor cores' operand (rows_gemm) it costs some 300 instructions per 16 x 64 tile,
// which kept the stream at 1.5 of 6.5 TB/s.  The packed tiles are the register fragments of mma.sync, so here they stay in the
// warp that loaded them: 9 instructions turn four fp8 bytes into two bf16 pairs and the MMA takes them as they are.
//   A unit is 128 weight rows (eight warps, a tile each) times the rows of a work item; CTAs take units in turn and warps run on
// from unit to unit, each at its own pace.  Token rows come in stages of 128 columns by bulk copies that warp 0 asks for.
//   Columns of a token row are stored (gather_rows, the epilogue below) in the order in which the fragments hold those of the
// weights: of sixteen columns the even ones, then the odd ones.  Block-scaled FP8 adds an accumulator per 128 columns with the
// block's scale to fp32 sums (the decode kernel's arithmetic); row scales are applied at the end.
//   Each warp's weights come through a ring of its own in shared memory, four pairs of blocks ahead.  (In registers, two pairs: 47 %
// of the issue slots used and gate and up 190 us, down 103.)
//   Bound by issue slots (60 % used, a fifth of the rest math-pipe throttle) and then by the stream: 256 experts x 15.6 rows,
// block-scaled, a layer's gate and up products (537 MB) 151 us, down (268 MB) 91 us, against 348 and 174 through the operand (83
// and 42 at the measured copy bandwidth).
// NT8: groups of eight tokens of the widest item.
constexpr int EX_STAGES = 5, EX_AHEAD = 4;
constexpr int EX_PAIR = 2048 + 16, EX_BARS = 128;      // bytes of two blocks of a tile and their scales; of the barriers
struct ExpertBars {
    uint64_t full[EX_STAGES], empty[EX_STAGES];
    volatile int dead;
};
static_assert(sizeof(ExpertBars) <= EX_BARS, "");
constexpr int experts_smem(int nt8) { return 1024 + EX_STAGES * 2 * nt8 * 8 * 128 + EX_BARS + 8 * EX_AHEAD * EX_PAIR; }
__device__ __forceinline__ uint4 lds16(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds8(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
// Four fp8 bytes as two pairs of bf16: bytes 0 and 2, bytes 1 and 3.
__device__ __forceinline__ void e4m3x4_bf16(uint32_t w, uint32_t& even, uint32_t& odd) {
    constexpr uint32_t UP = 0x7B807B80u;           // 2^120: the bits moved into the bf16 fields are the values times 2^-120, subnormals included
    even = mul_bf16x2(((w << 4) & 0x07F007F0u) | ((w << 8) & 0x80008000u), UP);
    odd = mul_bf16x2(((w >> 4) & 0x07F007F0u) | (w & 0x80008000u), UP);
}
// Offset of column c of a row whose sixteens are stored even columns first.
__device__ __forceinline__ size_t slab_offset_eo(int rows, int row, int c) { return slab_offset(rows, row, (c & ~15) | ((c & 1) << 3) | ((c & 15) >> 1)); }

template <bool BLOCKS, int OUT, int NT8>
static __global__ void __launch_bounds__(256, 2) experts_gemm(const __grid_constant__ GemmArgs A) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int X_KB = NT8 * 8 * 128;
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    ExpertBars& B = *reinterpret_cast<ExpertBars*>(smem + EX_STAGES * 2 * X_KB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    chain_wait();
    const int units = __ldcg(A.n_items) * A.blocks;
    auto item = [&](int u) { return __ldcg(A.items + min(u, units - 1) / A.blocks); };
    if ((int)blockIdx.x >= units) return;
    if (threadIdx.x == 0) {
        for (int i = 0; i < EX_STAGES; i++) {
            mbar_init(&B.full[i], 1);
            mbar_init(&B.empty[i], 8);
        }
        B.dead = 0;
        mk::fence_barrier_init();
    }
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    // Requests run EX_AHEAD pairs of blocks (64 columns each) ahead of the products, across units: each lane copies the bytes that it
    // will read to the warp's ring, and warp 0 asks for the token rows too.  (Block-scaled: a pair is four steps of one chunk with a
    // scale each for the tile's upper and lower eight rows.)
    Walk<W_FP8> walk;
    int ask_u = blockIdx.x, ask_kb = 0;
    uint32_t ask_slot = 0, ask_phase = 0;
    const uint32_t ring = smem_u32(smem + EX_STAGES * 2 * X_KB + EX_BARS + warp * (EX_AHEAD * EX_PAIR));
    uint32_t ask_at = 0, at = 0;                   // ring places of the next pair to ask for and to multiply
    int4 ask_it = item(blockIdx.x), ask_next = item(blockIdx.x + gridDim.x);
    auto ask_start = [&]() { walk.start(A, A.w + (size_t)ask_it.x * A.w_gstride, min(ask_u % A.blocks * 8 + warp, A.tiles - 1), 0, lane); };
    auto request = [&]() {
        if (ask_u < units) {
            const bool two = BLOCKS || ask_kb + 1 < A.kbs;
            const uint32_t to = ring + ask_at + lane * 16;
            if (BLOCKS) {
#pragma unroll
                for (int i = 0; i < 4; i++) mk::cp_async16(to + i * 512, walk.p + i * 512);
                if (lane == 0) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + 2048), "l"(walk.s) : "memory");
                walk.p += 2048;
                walk.s += 8;
                if ((walk.left -= 4) == 0) {
                    walk.left = A.chunk_steps;
                    walk.p += A.chunk_bytes - A.chunk_steps * 512;
                    walk.s += A.chunk_bytes - A.chunk_steps * 2;
                }
            } else {
                for (int i = 0; i < (two ? 4 : 2); i++) {
                    mk::cp_async16(to + i * 512, walk.p);
                    walk.step(A);
                }
            }
            if (warp == 0 && lane == 0 && wait(B, A, &B.empty[ask_slot], ask_phase ^ 1u, WP_EMPTY)) {
                const uint32_t bytes = (uint32_t)((ask_it.z + 7) & ~7) * 128u;
                mbar_expect_tx(&B.full[ask_slot], two ? 2 * bytes : bytes);
                for (int i = 0; i < (two ? 2 : 1); i++)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(smem_u32(smem + (size_t)(2 * ask_slot + i) * X_KB)), "l"(A.x + ((size_t)(ask_kb + i) * A.x_rows + ask_it.y) * 128), "r"(bytes),
                                   "r"(smem_u32(&B.full[ask_slot])) : "memory");
            }
            if (++ask_slot == EX_STAGES) {
                ask_slot = 0;
                ask_phase ^= 1u;
            }
            if ((ask_at += EX_PAIR) == EX_AHEAD * EX_PAIR) ask_at = 0;
            if ((ask_kb += 2) >= A.kbs) {
                ask_kb = 0;
                ask_u += gridDim.x;
                ask_it = ask_next;
                ask_next = item(ask_u + gridDim.x);
                if (ask_u < units) ask_start();
            }
        }
        mk::cp_async_commit();                     // (also when there is nothing left: waiting for all but EX_AHEAD - 1 then still waits for the pair)
    };
    ask_start();
#pragma unroll 1
    for (int i = 0; i < EX_AHEAD; i++) request();
    uint32_t slot = 0, phase = 0;
    const uint32_t frag = smem_u32(smem) + (uint32_t)(lane & 7) * 128, piece = lane >> 3, sw = lane & 7;
    int4 it = item(blockIdx.x);
#pragma unroll 1
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int4 next = item(u + gridDim.x);
        const int tile = u % A.blocks * 8 + warp;
        float sums[NT8][4];
        bool ok = true;
        // The unit's products for N8 groups of eight tokens, written out for each number: a loop that leaves at the number in hand took
        // a fifth more instructions, most of them branches (gate and up 200 us instead of 190).
        auto products = [&](auto n8) {
            constexpr int N8 = decltype(n8)::value;
            float acc[N8][4];
#pragma unroll
            for (int n = 0; n < N8; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[n][i] = sums[n][i] = 0.f;
            auto product = [&](uint32_t w, uint32_t x, bool fresh) {                     // fresh: the accumulators start over
                uint32_t a[4][4];                        // [16 columns][row g even, row g + 8 even, row g odd, row g + 8 odd]
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const uint4 q = lds16(w + i * 512);
                    e4m3x4_bf16(q.x, a[2 * i][0], a[2 * i][2]);
                    e4m3x4_bf16(q.y, a[2 * i + 1][0], a[2 * i + 1][2]);
                    e4m3x4_bf16(q.z, a[2 * i][1], a[2 * i][3]);
                    e4m3x4_bf16(q.w, a[2 * i + 1][1], a[2 * i + 1][3]);
                }
#pragma unroll
                for (int n = 0; n < N8; n++) {
                    uint32_t b[2][4];
#pragma unroll
                    for (int h = 0; h < 2; h++) ldsm4(b[h], x + n * 1024 + (((4 * h + piece) ^ sw) << 4));
                    if (fresh) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
                    for (int j = 0; j < 4; j++) mma16816(acc[n], a[j], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
                }
            };
#pragma unroll 1
            for (int kb = 0; kb < A.kbs; kb += 2) {
                ok = __all_sync(0xffffffffu, wait(B, A, &B.full[slot], phase, WP_FULL));               // the warp leaves together
                if (!ok) break;
                cp_wait<EX_AHEAD - 1>();
                __syncwarp();
                const uint32_t x = frag + 2 * slot * X_KB, w = ring + at + lane * 16;
                product(w, x, BLOCKS);
                if (BLOCKS || kb + 1 < A.kbs) product(w + 1024, x + X_KB, false);
                if constexpr (BLOCKS) {
                    const float2 sc = lds8(ring + at + 2048);
#pragma unroll
                    for (int n = 0; n < N8; n++) {
                        sums[n][0] = fmaf(acc[n][0], sc.x, sums[n][0]);
                        sums[n][1] = fmaf(acc[n][1], sc.x, sums[n][1]);
                        sums[n][2] = fmaf(acc[n][2], sc.y, sums[n][2]);
                        sums[n][3] = fmaf(acc[n][3], sc.y, sums[n][3]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&B.empty[slot]);
                if (++slot == EX_STAGES) {
                    slot = 0;
                    phase ^= 1u;
                }
                if ((at += EX_PAIR) == EX_AHEAD * EX_PAIR) at = 0;
                request();
            }
            if constexpr (!BLOCKS)
#pragma unroll
                for (int n = 0; n < N8; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++) sums[n][i] = acc[n][i];
        };
        static_assert(NT8 == 4, "one case for every number of groups");
        const int groups = __shfl_sync(0xffffffffu, (it.z + 7) >> 3, 0);
        if (groups <= 1) products(std::integral_constant<int, 1>{});
        else if (groups == 2) products(std::integral_constant<int, 2>{});
        else if (groups == 3) products(std::integral_constant<int, 3>{});
        else products(std::integral_constant<int, 4>{});
        if (!ok) {
            if (warp == 0) {                     // copies in flight must land before the CTA leaves (see rows_gemm)
                const u64 t0 = mk::globaltimer();
                while (mk::globaltimer() - t0 < 1000000ull) {}
            }
            break;
        }
        // lane (g, t): rows g and g + 8 of the tile, tokens 2 t and 2 t + 1 of every eight
        const int r0 = tile * 16 + g;
        float rs0 = 1.f, rs1 = 1.f;
        if (A.row_scale && tile < A.tiles) {
            const float* rs = A.row_scale + (size_t)it.x * A.rs_gstride;
            if (r0 < A.n_valid) rs0 = __ldg(rs + r0);
            if (r0 + 8 < A.n_valid) rs1 = __ldg(rs + r0 + 8);
        }
        if (tile < A.tiles) {
#pragma unroll
            for (int n = 0; n < NT8; n++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int tok = 8 * n + 2 * t + i;
                    if (tok >= it.z) continue;
                    const float lo = sums[n][i] * rs0, hi = sums[n][2 + i] * rs1;
                    if (OUT == OUT_GLU) {            // rows 0-7 of a tile are gates, rows 8-15 their up rows
                        const int col = tile * 8 + g;
                        const float y = (A.gelu ? 0.5f * lo * (1.f + tanhf(0.7978845608028654f * (lo + 0.044715f * lo * lo * lo))) : silu_f(lo)) * hi;
                        if (col < A.act_cols) *reinterpret_cast<__nv_bfloat16*>(A.act + slab_offset_eo(A.act_rows, it.y + tok, col)) = __float2bfloat16_rn(y);
                    } else {
                        float* o = A.out + (size_t)(it.y + tok) * A.out_stride + r0;
                        if (r0 < A.n_valid) o[0] = lo;
                        if (r0 + 8 < A.n_valid) o[8] = hi;
                    }
                }
        }
        it = next;
    }
    mk::cp_async_wait_all();                       // (a warp that gave up has copies in flight)
}

// ---- expert routing --------------------------------------------------------------------------------------------
struct RouteArgs {
    const float* logits;
    int rows, stride, experts, topk, kind;
    const float* expert_scale;
    int4* items;                 // {expert, first row, rows, 0}
    int* n_items;
    int* counts;                 // [experts] tokens per expert, then [experts] fill counters, then [experts] first rows
    int* slot;                   // [rows][8] row of the token's k-th expert (ascending expert id) in the gathered order
    float* weight;               // [rows][8]
    float* gate;                 // [rows] shared expert's gate
    int* ids_out;                // [sequences][topk] the last position's experts in rank order, or null
    int L;
    int nt;
};

// One warp per token: the top-k experts (ties to the lower id), their weights, and the count per expert.
static __global__ void __launch_bounds__(256) route_rows(const __grid_constant__ RouteArgs R) {
    chain_wait();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= R.rows) return;
    const float* lg = R.logits + (size_t)row * R.stride;
    const int per = R.experts / 32;
    float v[8];
    bool used[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        v[i] = i < per ? lg[lane + 32 * i] : 0.f;
        used[i] = i >= per;
    }
    float top0 = 0.f, wsum = 0.f, myw = 0.f;
    int myid = 0x7fffffff;
#pragma unroll 1
    for (int k = 0; k < R.topk; k++) {
        u64 best = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (!used[i]) {
                const u64 key = mk::score_key(v[i], lane + 32 * i);
                best = key > best ? key : best;
            }
        best = mk::warp_max_u64(best);
        const int id = max(0, min(R.experts - 1, mk::key_index(best)));
        float mine = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (i == (id >> 5)) {
                mine = v[i];
                if (lane == (id & 31)) used[i] = true;
            }
        const float sc = __shfl_sync(0xffffffffu, mine, id & 31);
        if (k == 0) top0 = sc;
        const float w = __expf(sc - top0);
        wsum += w;
        if (lane == k) {
            myw = w;
            myid = id;
        }
    }
    // rank among the token's experts: ascending id, the order in which their products are added
    int rank = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) rank += __shfl_sync(0xffffffffu, myid, k) < myid;
    if (lane < R.topk) {
        R.slot[(size_t)row * 8 + rank] = myid;                           // the expert for now; route_slots turns it into a row
        R.weight[(size_t)row * 8 + rank] = myw / wsum * (R.kind == 1 && R.expert_scale ? R.expert_scale[myid] : 1.f);
        atomicAdd(R.counts + myid, 1);
        if (R.ids_out && row % R.L == R.L - 1) R.ids_out[(row / R.L) * R.topk + lane] = myid;
    }
    if (R.kind == 0 && lane == 0) R.gate[row] = sigmoid_f(lg[R.experts]);
}

// Lays the experts' tokens out one after the other (each expert from a multiple of 16 rows) and lists the tiles.
static __global__ void __launch_bounds__(256) route_plan(const __grid_constant__ RouteArgs R) {
    chain_wait();
    __shared__ int rows_s[256], tiles_s[256];
    const int e = threadIdx.x, n = e < R.experts ? R.counts[e] : 0;
    const int rows = (n + 15) & ~15, tiles = (n + R.nt - 1) / R.nt;
    rows_s[e] = rows;
    tiles_s[e] = tiles;
    __syncthreads();
    for (int d = 1; d < 256; d <<= 1) {
        const int a = e >= d ? rows_s[e - d] : 0, b = e >= d ? tiles_s[e - d] : 0;
        __syncthreads();
        rows_s[e] += a;
        tiles_s[e] += b;
        __syncthreads();
    }
    const int first = rows_s[e] - rows, item = tiles_s[e] - tiles;
    if (e < R.experts) {
        R.counts[2 * R.experts + e] = first;
        for (int i = 0; i < tiles; i++) R.items[item + i] = make_int4(e, first + i * R.nt, min(R.nt, n - i * R.nt), 0);
    }
    if (e == 255) *R.n_items = tiles_s[255];
}

static __global__ void __launch_bounds__(256) route_slots(const __grid_constant__ RouteArgs R) {
    chain_wait();
    const int i = blockIdx.x * 256 + threadIdx.x, row = i >> 3, k = i & 7;
    if (row >= R.rows || k >= R.topk) return;
    const int e = R.slot[i];
    R.slot[i] = R.counts[2 * R.experts + e] + atomicAdd(R.counts + R.experts + e, 1);
}

// Copies every token's slab row to the rows of its experts.  EO: of every sixteen columns the even ones first, as experts_gemm
// reads them.
template <bool EO>
static __global__ void __launch_bounds__(256) gather_rows(const uint8_t* x, int x_rows, const int* slot, int topk, int kbs, uint8_t* out, int out_rows) {
    chain_wait();
    const int row = blockIdx.x;
    for (int i = threadIdx.x; i < kbs * 4; i += 256) {
        const int kb = i >> 2, c = 2 * (i & 3);
        const uint8_t* src = x + ((size_t)kb * x_rows + row) * 128;
        uint4 a = *reinterpret_cast<const uint4*>(src + ((c ^ (row & 7)) << 4)), b = *reinterpret_cast<const uint4*>(src + (((c + 1) ^ (row & 7)) << 4));
        if (EO) {
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            a = make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410), __byte_perm(w[4], w[5], 0x5410), __byte_perm(w[6], w[7], 0x5410));
            b = make_uint4(__byte_perm(w[0], w[1], 0x7632), __byte_perm(w[2], w[3], 0x7632), __byte_perm(w[4], w[5], 0x7632), __byte_perm(w[6], w[7], 0x7632));
        }
        for (int k = 0; k < topk; k++) {
            const int s = slot[(size_t)row * 8 + k];
            uint8_t* dst = out + ((size_t)kb * out_rows + s) * 128;
            *reinterpret_cast<uint4*>(dst + ((c ^ (s & 7)) << 4)) = a;
            *reinterpret_cast<uint4*>(dst + (((c + 1) ^ (s & 7)) << 4)) = b;
        }
    }
}

// Weighted sum of a token's expert outputs (ascending expert id, then the shared expert), stored or added.
static __global__ void __launch_bounds__(256) combine_rows(const float* y, int N, const int* slot, const float* weight, int topk, const float* shared, const float* gate,
                                                    int add, float* out, long long out_stride) {
    chain_wait();
    const int row = blockIdx.x;
    for (int c = threadIdx.x * 4; c < N; c += 1024) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < topk; k++) {
            const float w = weight[(size_t)row * 8 + k];
            const float4 v = *reinterpret_cast<const float4*>(y + (size_t)slot[(size_t)row * 8 + k] * N + c);
            s.x = fmaf(v.x, w, s.x); s.y = fmaf(v.y, w, s.y); s.z = fmaf(v.z, w, s.z); s.w = fmaf(v.w, w, s.w);
        }
        if (shared) {
            const float w = gate[row];
            const float4 v = *reinterpret_cast<const float4*>(shared + (size_t)row * N + c);
            s.x = fmaf(v.x, w, s.x); s.y = fmaf(v.y, w, s.y); s.z = fmaf(v.z, w, s.z); s.w = fmaf(v.w, w, s.w);
        }
        float4* o = reinterpret_cast<float4*>(out + (size_t)row * out_stride + c);
        if (add) {
            const float4 b = *o;
            s.x += b.x; s.y += b.y; s.z += b.z; s.w += b.w;
        }
        *o = s;
    }
}

}  // namespace mkp
