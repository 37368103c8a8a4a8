// Stage-machine decode megakernel for sm_100a: one CTA per SM, one cooperative launch for n_steps
// decode steps of up to eight sequences.
//
// What a step does is a program of mk_stage_desc records (include/mk_stage.h) in device memory.
// Every CTA has 16 consumer warps and one scout warp:
//
//   * every consumer warp owns a few slots of a shared-memory ring and feeds them itself: a lane copies (cp.async) the very
//     bytes it will multiply, four tile steps ahead at a time, so a slot needs no barrier and no other warp has to notice
//     that it is free.  The stream runs ahead across stage boundaries: weights of the next matrix land while the warp
//     waits at a grid barrier.  It never depends on activations, except for the routed expert list;
//   * the scout walks the program ahead of the consumers and leaves each GEMV stage's geometry (this CTA's tiles and
//     columns) in shared memory, so that a warp that runs into the next stage does not wait for global memory;
//   * a GEMV stage is cut into panels of input columns (usually one: the whole row) and 16-row tiles.  A CTA stages one
//     panel's input and takes an even share of the panel's tiles; its sixteen warps take even shares of the CTA's weight
//     chunks, in order, so a warp multiplies whole rows and at most shares its first and its last tile with its
//     neighbours (summed through shared memory).  The weight bytes become fp16 in registers (bf16 stays bf16) and
//     multiply with `mma.sync.m16n8k16`: the weight tile is the 16-row A operand, the sequences are the eight B columns,
//     so one to eight sequences cost the same number of instructions;
//   * with several panels every CTA publishes its 16 x 8 partial tiles as words that carry their own tag, and one CTA per
//     tile (they take turns) polls the panels' words and adds them in a fixed order; then the epilogue runs
//     (store, residual add with sums of squares for the next RMSNorm, GLU, logits + arg-max);
//   * with tensor parallelism the epilogue of a row-parallel GEMV first pushes the tile into every
//     rank's mailbox with plain peer stores (value and sequence tag in one 64-bit word), polls its own
//     mailbox and adds the ranks' tiles in rank order, so every rank holds the same bits;
//   * stages meet at a grid barrier (one atomic counter in global memory, bounded wait).
//
// Every wait is bounded: a wait that runs out records MK_ERR_TIMEOUT and its site in the status words,
// after which every wait in every CTA returns at once, the remaining stages are skipped, every warp
// waits for its copies in flight and the kernel returns.
#pragma once
#include <cuda_fp16.h>

#include "../../include/mk_stage.h"
#include "mk_device.cuh"

namespace mks {
using namespace mk;

constexpr int SLOT_BYTES = 4352;                  // largest chunk of the packed format: 8 tile steps of 512 bytes + 256 bytes of scales
constexpr int BLOCK_STEPS = 4;                    // one ring slot: four tile steps and their scales
constexpr int BLOCK_BYTES = BLOCK_STEPS * 512 + 128;
constexpr int XS_BYTES = 82432;                   // staged GEMV input: 8 columns x 5120 fp16 + padding; also mixer scratch and shared tiles
constexpr int MAX_GROUPS = 72;                    // routed experts of one step (8 x 8) + shared / dense groups
constexpr int MISC_BYTES = 10752;
constexpr int SMEM_TOTAL = 232448;                // 227 KB
constexpr int MIN_RING_DEPTH = 4, MAX_RING_DEPTH = 5;   // ring slots per consumer warp: as many as the launch's input staging area leaves room for
constexpr int MAX_SEGS = 16;                      // K splits (of all groups) of one panel of a stage that adds its groups up
constexpr int TILE_BYTES = 16 * 512;              // what each warp adds to a tile that the warp before it started
constexpr int GEO_RING = 4;                       // stage records in shared memory: the scout is up to three stages ahead
constexpr int ATTN_MAX_CHUNK = 256;               // positions per attention task (score buffer)
constexpr int MAILBOX_TILES = 1024;               // output tiles of a row-parallel GEMV one all-reduce can carry
constexpr int MAILBOX_BYTES = 2 * MAILBOX_TILES * MKS_MAX_RANKS * 128 * 8 + 2 * MKS_MAX_RANKS * MKS_MAX_BATCH * 16;
static_assert((size_t)16 * MIN_RING_DEPTH * BLOCK_BYTES + XS_BYTES + MISC_BYTES <= SMEM_TOTAL, "shared memory of one SM");

// wait sites (status[1])
enum { WS_SCOUT = 101, WS_BARRIER, WS_MAILBOX, WS_KEYS, WS_TILE };

struct Args {
    const mk_stage_desc* prog;
    int n_stages, M, n_steps;
    int* tok;
    int* pos;
    int* tokens_out;
    unsigned long long* bar;
    unsigned long long bar_base;
    int* status;
    long long spin_limit_ns;
    unsigned long long* prof;
    int tp, rank;
    unsigned long long* mailbox[MKS_MAX_RANKS];
    unsigned long long ar_base;
    const int* tokens_in;    // [n_tokens_in][M] forced inputs of the first steps, or null
    int n_tokens_in;
    const int* row_valid;    // [M] 0 = padding row, or null
    int prof_cta;            // the CTA whose timestamps go to `prof`
    int xs_bytes;            // input staging / mixer scratch area of this launch
    int ring_depth;          // ring slots per consumer warp
    uint32_t tile_tag;       // tag of this launch's first partial tiles
    int clear_tiles;         // 1: words of partial tiles are left zero (a captured launch, which runs again with the same tags)
};

// Everything the threads of a CTA share lives in shared memory, behind the ring and the input staging
// area; what is per thread (identity, ring position) travels in registers.  A per-thread context struct
// handed to the stage functions by reference would sit in local memory: 544 threads' copies do not fit
// the few KB of L1 that the shared-memory carve-out leaves, and every field access would cost an L2 trip.
// One GEMV stage as this CTA sees it (written by the scout, read by every warp).
struct Geo {
    const uint8_t* w;              // weights of group 0 (or of expert 0)
    const uint8_t* w_shared;       // weights of the last group of a routed stage, or null
    u64 gstride, w_bytes;
    int T, S, G;                   // tiles and K splits of a group, groups
    int n_chunks, chunk_steps, chunk_bytes;
    int ebps;                      // scale bytes per tile step
    int reduce, routed;
    int Q, P, panel;               // K splits a tile adds up, panels they are cut into, this CTA's panel (-1: all, one after another)
    int t0, t1;                    // this CTA's tiles (of all groups, unless the groups are added up)
    int g0, ng;                    // groups these tiles lie in, when every group has an input of its own (else 0, 1)
    int nb;                        // batches: one staged input each
    uint32_t stage;                // the stage this entry describes (counted over the launch)
    int beside;                    // CTAs this stage leaves to the one behind it (0: it has the whole grid, or the rest of it)
};
// A warp's share of a batch: chunks [c, c1), tile by tile.
struct Share {
    const uint8_t* src;            // chunk c
    int c, c1, per;                // per: chunks of every warp's share but the last ones'
    int cpt, tl, k;                // chunks of one tile; chunk c as tile of the batch and chunk of the tile
};
// The stream's registers (the same in every lane but for what is said to be the lane's own).
struct Feed {
    const uint8_t* src;            // next step of the current chunk (of the whole run, where chunks are steps alone); this lane's bytes
    int steps, left;               // steps left in it, chunks left in the run behind it
    int eoff;                      // from src to the scales of that step (this lane's)
    int ebps, cs;                  // scale bytes per step, steps per chunk
    int gap;                       // bytes from a chunk's last step to the next chunk: its scales and padding
    int ahead;                     // blocks requested and not yet multiplied
    uint32_t rd;                   // shared-memory address of the next block to multiply (this lane's part)
};
// Where a consumer warp's weight stream stands: ahead of the multiplication by up to the ring's depth.
struct Cur {
    const uint8_t* src;            // the current run of consecutive chunks
    int left;                      // its chunks
    int rest;                      // chunks of the batch behind the run
    int run, jump;                 // chunks of a whole run, bytes from one's end to the next
    int chunk_bytes, chunk_steps;
    int ebps;                      // scale bytes per tile step (behind a chunk's steps)
    int tile, seg, seg0, seg1;     // the run behind the current one, if the runs belong to several matrices; the batch's K splits
    uint32_t gn, now;              // stages entered; the stage the warp multiplies in
    int b, nb;                     // batches of the stage begun, all of them
    // the registers of the stream between two GEMV stages
    Feed f;                        // (the first lane's)
};

struct Shared {
    u64 keys_s[8];                 // best key per sequence
    mk_stage_desc desc[GEO_RING];  // stage n's record in entry n % GEO_RING
    Geo geo[GEO_RING];             // and, for a GEMV stage, its geometry
    Share share[GEO_RING][NCW];    // its first batch's
    Cur cur[NCW];
    unsigned long long* prof;      // this stage's timestamp row (CTA 0, last step) or null
    Args A;                        // the launch arguments
    uint32_t tag0;                 // stage barriers passed before this launch
    float red[16 + 17 * 8];        // block-reduction scratch
    float xinv[MAX_SEGS * 8];      // factor that undoes the power-of-two scaling of a staged column (of every K split, when groups are added up)
    int xmax[MAX_SEGS * 8];        // its largest magnitude, then its scale
    float rstd[8];                 // 1/rms of the staged input
    int tok_s[8];
    int pos_s[8];
    int valid_s[8];                // 0: a padding row of this launch
    int r_ids[64];                 // [8][8] routed expert ids per sequence
    float r_w[64];                 // [8][8] routing weights
    float coef[MAX_GROUPS * 8];    // weight of group g for sequence m
    int glist[MAX_GROUPS];         // expert id of group g
    unsigned gmask[8];             // bitmap of the selected experts
    int n_groups;
    volatile int abort_flag;
    volatile unsigned route_seq;
    volatile unsigned described;   // stages the scout has described
    volatile unsigned completed;   // stages all warps of this CTA have left
    int flag;
    // dynamic shared memory: [this block | staging area of A.xs_bytes | 16 x A.ring_depth ring slots]
    __device__ __forceinline__ uint8_t* xs() { return reinterpret_cast<uint8_t*>(this) + MISC_BYTES; }
    __device__ __forceinline__ uint8_t* ring() { return reinterpret_cast<uint8_t*>(this) + MISC_BYTES + A.xs_bytes; }
};
static_assert(sizeof(Shared) <= MISC_BYTES, "the shared block fits its area");

// thread identity from the special registers: cheaper than a struct that travels through the stack
__device__ __forceinline__ int tid_() { return (int)threadIdx.x; }
__device__ __forceinline__ int warp_() { return (int)(threadIdx.x >> 5); }
__device__ __forceinline__ int lane_() { return (int)(threadIdx.x & 31); }
__device__ __forceinline__ int cta_() { return (int)blockIdx.x; }
__device__ __forceinline__ int grid_() { return (int)gridDim.x; }
constexpr int PROF_FIELDS = 8;  // per stage: entered, input staged, work done, barrier passed, then up to three marks inside staging or attention
__device__ __forceinline__ void prof_mark(Shared& S, int field) {
    if (S.prof && tid_() == 0) S.prof[field] = globaltimer();
}

// ---- bounded waits ---------------------------------------------------------------------------------------
struct Spin2 {
    uint32_t it = 0;
    u64 t0 = 0;
};
__device__ __noinline__ u64 spin_slow2(volatile int* abort_flag, int* status, u64 limit_ns, u64 t0, int where) {
    if (*abort_flag) return ~0ull;
    if (ld_volatile_i32(status) != 0) {
        *abort_flag = 1;
        return ~0ull;
    }
    const u64 now = globaltimer();
    if (!t0) return now;
    if (now - t0 > limit_ns) {
        if (atomicCAS(status, 0, -2) == 0) {
            status[1] = where;
            status[2] = (int)blockIdx.x;
            status[3] = (int)threadIdx.x;
        }
        __threadfence();
        *abort_flag = 1;
        return ~0ull;
    }
    return t0;
}
#define MKS_SPIN_FAIL(S, s, where) \
    ((((++(s).it) & 255u) == 0) && (((s).t0 = spin_slow2(&(S).abort_flag, (S).A.status, (u64)(S).A.spin_limit_ns, (s).t0, (where))) == ~0ull))

__device__ __forceinline__ u64 ld_acquire_u64(const unsigned long long* p) {
    u64 v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ u64 ld_relaxed_sys_u64(const unsigned long long* p) {
    u64 v;
    asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_sys_u64(unsigned long long* p, u64 v) {
    chaos_delay();
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Grid barrier over the consumer threads of all CTAs: one arrival per CTA on a counter that only grows.
// The arrival is a release (everything this CTA wrote before the preceding CTA barrier is visible to
// whoever observes the count), the poll an acquire; no sequentially-consistent fence is needed.
__device__ __forceinline__ void red_release_add_u64(unsigned long long* p, unsigned long long v) {
    chaos_delay();
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// Only thread 0 waits here; the CTA barrier in front of the next stage holds the others.
__device__ __forceinline__ void grid_barrier(Shared& S, const Args& A, u64& bar_n) {
    bar_n++;
    consumer_sync();
    if (tid_() == 0 && !S.abort_flag) {
        red_release_add_u64(A.bar, 1ull);
        const u64 target = A.bar_base + bar_n * (u64)grid_();
        Spin2 s;
        while (ld_acquire_u64(A.bar) < target) {
            if (MKS_SPIN_FAIL(S, s, WS_BARRIER)) break;
        }
    }
    __syncwarp();
}

// ---- conversions -----------------------------------------------------------------------------------------
// Two e2m1 values in the low byte of `b` -> f16x2 (low nibble in the low half).
__device__ __forceinline__ uint32_t cvt_e2m1x2(uint32_t b) {
    uint32_t r;
    asm("{\n .reg .b8 t;\n .reg .b16 h;\n cvt.u16.u32 h, %1;\n cvt.u8.u16 t, h;\n cvt.rn.f16x2.e2m1x2 %0, t;\n}\n" : "=r"(r) : "r"(b));
    return r;
}
// Two e4m3 values in the low 16 bits of `b` -> f16x2.
__device__ __forceinline__ uint32_t cvt_e4m3x2(uint32_t b) {
    uint32_t r;
    asm("{\n .reg .b16 h;\n cvt.u16.u32 h, %1;\n cvt.rn.f16x2.e4m3x2 %0, h;\n}\n" : "=r"(r) : "r"(b));
    return r;
}
// Two signed bytes (low 16 bits of `b`, already xor 0x80) -> f16x2: 0x6400 | u is the half 1024 + u.
__device__ __forceinline__ uint32_t cvt_s8x2(uint32_t bx, uint32_t sel) {
    const uint32_t h = __byte_perm(bx, 0x64646464u, sel);             // [0x64, b1, 0x64, b0] as two halves
    const __half2 v = *reinterpret_cast<const __half2*>(&h);
    const __half2 r = __hsub2(v, __floats2half2_rn(1152.f, 1152.f));  // 1024 + 128
    return *reinterpret_cast<const uint32_t*>(&r);
}

// (not `volatile`: the instruction has no effect beyond its outputs, and the compiler must be free to interleave
// independent accumulator chains -- a warp issues in order, and a dependent MMA behind its producer stalls it)
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float gelu_tanh_f(float x) {
    return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float ldcg_f(const float* p) { return __ldcg(p); }

// ---- geometry of a GEMV stage (shared by scout, weight streams and multiplication) ---------------------------------
// Column stride of the staged input in bytes: a multiple of 128 plus 32, so that the eight columns'
// 8-byte fragment reads of a half warp fall into different banks.
__host__ __device__ __forceinline__ int xs_stride_bytes(int cols) { return ((cols * 2 + 127) / 128) * 128 + 32; }
// K splits of `kc` columns of `ncols` staged columns (sequences x pieces) that fit `xs_bytes`.
__host__ __device__ __forceinline__ int max_panel_splits(int xs_bytes, int kc, int ncols, int pieces, bool reduce) {
    int w = (xs_bytes / ncols - 32) / 128 * 64 / kc;
    if (reduce) w = min(w, MAX_SEGS);
    return max(w, 1);
}
// What a stage costs the busiest CTA, in bytes of weight stream (about 83 per ns), if its R tiles x Q splits are cut into P
// panels: the weights of its tiles (whole chunks per warp count half: the other warps keep the memory busy); the input it
// stages (every CTA reads its panel's fp32 columns from L2: about 0.12 ns a value); and with more than one panel the exchange:
// one round trip through L2 (about 1.5 us) and 16-byte words of partial tiles, written once and read once.
// (In floats: the scout compares them while the CTA waits for a routed stage.)
__host__ __device__ __forceinline__ float panel_cost(int R, int Q, int P, int n_chunks, int chunk_bytes, int kc, int M, int grid) {
    const int tiles = (R * P + grid - 1) / grid, w = (Q + P - 1) / P;
    const int chunks = tiles * w * n_chunks, even = (chunks + NCW - 1) / NCW * NCW;
    return 0.5f * (float)(chunks + even) * (float)chunk_bytes + (float)(w * kc) * (float)M * 10.f + (P > 1 ? 120000.f + (float)(tiles * M) * 256.f : 0.f);
}

// Every lane of the scout calls this: the number of panels, from P0 (what the staging area allows) up to half the grid
// (each panel then has a CTA).
__device__ __forceinline__ int pick_panels(int R, int Q, int P0, int n_chunks, int chunk_bytes, int kc, int M, int grid) {
    const int P1 = min(Q, grid / 2);
    if (P0 >= P1) return P0 == P1 ? P0 : 0;
    float best = 3.0e38f;
    int at = 0;
    for (int P = P0 + lane_(); P <= P1; P += 32) {
        const float k = panel_cost(R, Q, P, n_chunks, chunk_bytes, kc, M, grid);
        if (k < best) {
            best = k;
            at = P;
        }
    }
    __syncwarp();
    const int low = __reduce_min_sync(0xffffffffu, __float_as_int(best));          // (positive floats compare like their bits)
    return (int)__reduce_min_sync(0xffffffffu, __float_as_int(best) == low ? (unsigned)at : ~0u);
}

// One batch of a stage: a staged input (K splits [seg0, seg1) of a panel) and the tiles [t0, t1) it multiplies.
struct Batch {
    int panel, seg0, seg1, t0, t1, grp;
};
__device__ __forceinline__ Batch geo_batch(const Geo& g, int b) {
    Batch r;
    const int pb = g.ng == 1 ? b : b / g.ng, gb = b - pb * g.ng;
    r.panel = g.panel >= 0 ? g.panel : pb;
    r.seg0 = g.P == 1 ? 0 : g.Q * r.panel / g.P;
    r.seg1 = g.P == 1 ? g.Q : g.Q * (r.panel + 1) / g.P;
    r.t0 = g.t0; r.t1 = g.t1; r.grp = 0;
    if (g.ng > 1 || g.g0 > 0) {
        r.grp = g.g0 + gb;
        r.t0 = max(r.t0, r.grp * g.T);
        r.t1 = min(r.t1, (r.grp + 1) * g.T);
    }
    return r;
}
// Weight bytes of group `grp`: experts of a routed stage come from the routing list, the shared expert last.
__device__ __forceinline__ const uint8_t* group_weights(const Shared& S, const Geo& g, int grp) {
    if (!g.routed) return g.w + (size_t)grp * g.gstride;
    if (g.w_shared && grp == g.G - 1) return g.w_shared;
    return g.w + (size_t)reinterpret_cast<const volatile int*>(S.glist)[grp] * g.gstride;
}
__device__ __forceinline__ const float* group_row_scale(const Shared& S, const mk_stage_desc& d, int grp, int G) {
    const float* s = reinterpret_cast<const float*>(d.p[MKS_P_ROW_SCALE]);
    if (!s) return nullptr;
    if (d.i[MKS_I_GROUPS] >= 0) return s + (size_t)grp * d.p[MKS_P_RS_GSTRIDE];
    if (d.p[MKS_P_W_SHARED] && grp == G - 1) return reinterpret_cast<const float*>(d.p[MKS_P_RS_SHARED]);
    return s + (size_t)S.glist[grp] * d.p[MKS_P_RS_GSTRIDE];
}

// ---- the weight stream of a consumer warp --------------------------------------------------------------------
// A warp requests its own weights, block by block (four tile steps), in the order it multiplies them: lane j copies the 16
// bytes per step that lane j will read, and right after a block has been read the slot takes the next request.  So all of the
// ring but one block is in flight, and nobody polls for free slots.  (A 95 MB MXFP4 matrix: 34 us for its stage; a producer
// warp that filled two slots of a whole chunk per consumer warp streamed at 3.0 TB/s where the same loop with the data in
// place runs at 5.9.)
__device__ __noinline__ void stream_error(Shared& S, uint32_t stage, int where) {
    if (atomicCAS(S.A.status, 0, -5) == 0) {
        S.A.status[1] = (int)stage;
        S.A.status[2] = cta_();
        S.A.status[3] = where;
    }
    S.abort_flag = 1;
}
// Weights of K split `seg` (of all groups, if they are added up) of tile `tile` (of all groups, if they are not).
__device__ __forceinline__ const uint8_t* split_weights(const Shared& S, const Geo& g, int tile, int seg) {
    int grp = 0;
    if (g.reduce) {
        grp = g.S == 1 ? seg : seg / g.S;
        seg -= grp * g.S;
    } else if (g.G > 1) {
        grp = tile / g.T;
        tile -= grp * g.T;
    }
    return group_weights(S, g, grp) + (size_t)((tile * g.S + seg) * g.n_chunks) * g.chunk_bytes;
}
constexpr int FEW_WARPS = 4;
// Warp w's share of a batch.
__device__ __forceinline__ Share batch_share(const Shared& S, const Geo& g, const Batch& bt, int w) {
    Share r;
    r.cpt = (bt.seg1 - bt.seg0) * g.n_chunks;
    // Equal shares of whole chunks, the first warps first: as long as the longest share is no longer, every warp without one
    // is a partial tile less to add.  Fewer chunks than warps go to FEW_WARPS: two or three chunks in a row cost less than
    // the exchange.  (Both rules together, 8 and 6 layers: 27B x1 per step 1417 -> 1373 us, x8 1699 -> 1656 us, 35B-A3B x8
    // 1531 -> 1493 us, 26B x4 1419 -> 1413 us; the second one's own part was not measured.)
    const int n = (bt.t1 - bt.t0) * r.cpt, warps = n < NCW && n > FEW_WARPS ? FEW_WARPS : NCW;
    r.per = (n + warps - 1) / warps;
    r.c = min(n, w * r.per);
    r.c1 = min(n, r.c + r.per);
    if (g.routed && !g.reduce) {
        // many tiles of many experts: cut as evenly as chunks allow.  `per` then holds minus the batch's chunks, from which
        // multiply() finds the warp that has a tile's last chunk.
        r.per = -n;
        r.c = n * w / NCW;
        r.c1 = n * (w + 1) / NCW;
    }
    r.tl = r.c / r.cpt;
    r.k = r.c - r.tl * r.cpt;
    const int sg = r.k / g.n_chunks;
    r.src = r.c < r.c1 ? split_weights(S, g, bt.t0 + r.tl, bt.seg0 + sg) + (size_t)(r.k - sg * g.n_chunks) * g.chunk_bytes : nullptr;
    return r;
}
// The next run of consecutive chunks; false if the scout has not described the stage it belongs to.  The whole warp calls it
// and every lane computes the same; its first lane writes the cursor back.
__device__ __noinline__ bool next_run(Shared& S) {
    Cur& c = S.cur[warp_()];
    const uint8_t* src = c.src;
    int rest = c.rest, run = c.run, left = 0;
    if (rest > 0) {
        const Geo& g = S.geo[(c.gn - 1) % GEO_RING];
        if (g.G == 1) {
            src += c.left * c.chunk_bytes + c.jump;            // the same columns of the next tile
        } else {
            const int tile = c.tile, seg = c.seg;
            src = split_weights(S, g, tile, seg);
            __syncwarp();
            if (lane_() == 0) {
                const bool end = !g.reduce || seg + 1 == c.seg1;
                c.seg = end ? c.seg0 : seg + 1;
                c.tile = end ? tile + 1 : tile;
            }
        }
        left = min(run, rest);
        rest -= left;
    } else {
        uint32_t gn = c.gn;
        int b = c.b, nb = c.nb;
        const unsigned described = __shfl_sync(0xffffffffu, S.described, 0);
        __threadfence_block();
        __syncwarp();
#pragma unroll 1
        while (left == 0) {
            if (b == nb) {                                     // next stage
                // (stages before the warp's own are over, and their entries may describe later ones by now)
                if ((int)(c.now - gn) > 0) gn = c.now;
                b = nb = 0;
                if ((int)(described - gn) <= 0) break;
                if (S.geo[gn % GEO_RING].stage != gn) {
                    stream_error(S, gn, -1);
                    break;
                }
                nb = S.geo[gn++ % GEO_RING].nb;
                if (nb == 0) continue;
            }
            const Geo& g = S.geo[(gn - 1) % GEO_RING];
            const Batch bt = geo_batch(g, b);
            Share sh;
            if (b == 0) sh = S.share[(gn - 1) % GEO_RING][warp_()];
            else sh = batch_share(S, g, bt, warp_());
            b++;
            rest = sh.c1 - sh.c;
            if (rest == 0) continue;
            src = sh.src;
            run = sh.cpt;
            left = run - sh.k;
            int seg = bt.seg0, tile = bt.t0 + sh.tl + 1;
            if (g.reduce) {
                run = g.n_chunks;                              // one K split of one matrix at a time
                seg = sh.k / run;
                left = run - (sh.k - seg * run);
                seg += bt.seg0 + 1;
                if (seg == bt.seg1) seg = bt.seg0;
                else tile--;
            }
            left = min(left, rest);
            rest -= left;
            // self-check: the copies must be aligned and stay inside the matrix the record describes
            if ((reinterpret_cast<size_t>(src) & 15) ||
                (g.w_bytes && g.G == 1 && (size_t)(src - g.w) + (size_t)((long long)rest * g.chunk_bytes) > (size_t)g.w_bytes)) {
                stream_error(S, gn, left);
                left = rest = 0;
                break;
            }
            __syncwarp();
            if (lane_() == 0) {
                c.run = run;
                c.jump = (g.S * g.n_chunks - sh.cpt) * g.chunk_bytes;
                c.chunk_bytes = g.chunk_bytes; c.chunk_steps = g.chunk_steps; c.ebps = g.ebps;
                c.tile = tile; c.seg = seg; c.seg0 = bt.seg0; c.seg1 = bt.seg1;
            }
        }
        __syncwarp();
        if (lane_() == 0) {
            c.gn = gn; c.b = b; c.nb = nb;
        }
    }
    __syncwarp();
    if (lane_() == 0) {
        c.src = src; c.left = left; c.rest = rest;
    }
    __syncwarp();
    return left > 0;
}
__device__ __forceinline__ void next_chunk(Feed& f) {
    f.src += f.gap;
    f.left--;
    f.steps = f.cs;
    f.eoff = f.cs * 512 - lane_() * 12;
}
// Fill the warp's free slots.  The caller has ordered the warp's reads of the freed slots before this (a warp barrier).
// Every free slot gets a group of copies, an empty one when there is nothing to request: then at least ring_depth - 1
// groups lie behind the next block to multiply, and waiting for all but that many waits for the block.
__device__ __forceinline__ void feed(Shared& S, Feed& f, int depth, uint32_t ring_end) {
    int n_free = depth - f.ahead;
#pragma unroll 1
    for (; n_free > 0; n_free--) {
        if (f.steps == 0) {
            if (f.left > 0) {
                next_chunk(f);
            } else {
                if (!next_run(S)) break;
                const Cur& c = S.cur[warp_()];
                f.ebps = c.ebps;
                f.gap = c.chunk_bytes - c.chunk_steps * 512;
                f.cs = f.gap ? c.chunk_steps : c.chunk_steps * c.left;
                f.left = f.gap ? c.left : 1;
                f.src = c.src + lane_() * 16 - f.gap;
                next_chunk(f);
            }
        }
        const int n = min(BLOCK_STEPS, f.steps);
        uint32_t wr = f.rd + f.ahead * BLOCK_BYTES;
        if (wr >= ring_end) wr -= depth * BLOCK_BYTES;
#pragma unroll 1
        for (int u = 0; u < n; u++) cp_async16(wr + u * 512, f.src + u * 512);
        if (lane_() * 4 < n * f.ebps) cp_async4(wr + BLOCK_STEPS * 512 - lane_() * 12, f.src + f.eoff);
        cp_async_commit();
        f.src += n * 512;
        f.steps -= n;
        f.eoff += n * (f.ebps - 512);
        f.ahead++;
    }
#pragma unroll 1
    for (; n_free > 0; n_free--) cp_async_commit();
}
// The same where only slot `wr` is free and a whole block can be requested (nearly always).
__device__ __forceinline__ void feed_one(Feed& f, uint32_t wr) {
#pragma unroll
    for (int u = 0; u < BLOCK_STEPS; u++) cp_async16(wr + u * 512, f.src + u * 512);
    if (lane_() < f.ebps) cp_async4(wr + BLOCK_STEPS * 512 - lane_() * 12, f.src + f.eoff);
    cp_async_commit();
    f.src += BLOCK_STEPS * 512;
    f.eoff += BLOCK_STEPS * (f.ebps - 512);
    f.steps -= BLOCK_STEPS;
    f.ahead++;
    if (f.steps == 0 && f.left > 0) next_chunk(f);
}
// All but depth - 1 groups of copies have landed.
__device__ __forceinline__ void wait_block(int depth) {
    static_assert(MIN_RING_DEPTH == 4 && MAX_RING_DEPTH == 5, "one wait per ring depth");
    if (depth == 4) cp_async_wait<3>();
    else cp_async_wait<4>();
}

// ---- scout ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool scout_wait(Shared& S, volatile unsigned* word, unsigned at_least) {
    Spin2 sp;
    bool stop = false;
#pragma unroll 1
    while (!__all_sync(0xffffffffu, (int)(*word - at_least) >= 0)) {      // (the warp leaves together)
        // (the consumers' own waits end a launch that is stuck; this bound is only the scout's last resort)
        if (lane_() == 0 && ((++sp.it) & 255u) == 0 &&
            (sp.t0 = spin_slow2(&S.abort_flag, S.A.status, 8 * (u64)S.A.spin_limit_ns, sp.t0, WS_SCOUT)) == ~0ull) stop = true;
        stop = stop || S.abort_flag != 0;
        if (__any_sync(0xffffffffu, stop)) return false;
        __nanosleep(40);
    }
    __threadfence_block();
    __syncwarp();
    return true;
}
// Two GEMV stages without a barrier between them do not depend on each other, and a small one is all latency: they share the
// grid in proportion to their weights, at least a CTA per tile of a small one (up to a tenth of the grid: an estimate).  One
// after the other, the gates' projection behind a 35B-A3B DeltaNet layer's qkvz, and in a 26B layer the router behind the
// dense gate and up and the experts' down behind the dense one, cost their whole latency, 13 to 20 us each.  -> CTAs of the second.
__device__ __forceinline__ int side_by_side(const mk_stage_desc& a, const mk_stage_desc& b, int n_groups, int grid) {
    const float ta = (float)a.i[MKS_I_TILES] * (a.i[MKS_I_GROUPS] < 0 ? n_groups : a.i[MKS_I_GROUPS]);
    const float tb = (float)b.i[MKS_I_TILES] * (b.i[MKS_I_GROUPS] < 0 ? n_groups : b.i[MKS_I_GROUPS]);
    const float ba = ta * a.i[MKS_I_SPLITS] * (a.i[MKS_I_UNIT_STEPS] / a.i[MKS_I_CHUNK_STEPS]) * a.i[MKS_I_CHUNK_BYTES];
    const float bb = tb * b.i[MKS_I_SPLITS] * (b.i[MKS_I_UNIT_STEPS] / b.i[MKS_I_CHUNK_STEPS]) * b.i[MKS_I_CHUNK_BYTES];
    const int least = max(2, grid / 10);
    int k = (int)((float)grid * bb / (ba + bb));
    k = max(k, min((int)tb, least));
    k = min(k, grid - min((int)ta, least));
    return max(1, min(grid - 1, k));
}
__device__ __noinline__ void scout_main(Shared& S, const Args& A) {
    constexpr int DESC_WORDS = (int)(sizeof(mk_stage_desc) / 4);
    unsigned n = 0, routes = 0;
#pragma unroll 1
    for (int step = 0; step < A.n_steps; step++) {
#pragma unroll 1
        for (int si = 0; si < A.n_stages; si++, n++) {
            uint32_t words[(DESC_WORDS + 31) / 32];
#pragma unroll
            for (int i = 0; i < (DESC_WORDS + 31) / 32; i++)
                if (lane_() + 32 * i < DESC_WORDS) words[i] = __ldg(reinterpret_cast<const uint32_t*>(&A.prog[si]) + lane_() + 32 * i);
            // the stage that had this entry is over
            if (n >= GEO_RING && !scout_wait(S, &S.completed, n - GEO_RING + 1)) return;
            mk_stage_desc& d = S.desc[n % GEO_RING];
            Geo& g = S.geo[n % GEO_RING];
#pragma unroll
            for (int i = 0; i < (DESC_WORDS + 31) / 32; i++)
                if (lane_() + 32 * i < DESC_WORDS) reinterpret_cast<uint32_t*>(&d)[lane_() + 32 * i] = words[i];
            __syncwarp();
            if (d.op == MKS_OP_ROUTE) routes++;
            if (d.op != MKS_OP_GEMV) {
                if (lane_() == 0) {
                    g.nb = 0;
                    g.beside = 0;
                    g.stage = n;
                    __threadfence_block();
                    S.described = n + 1;
                }
                continue;
            }
            if (d.i[MKS_I_GROUPS] < 0 && !scout_wait(S, &S.route_seq, routes)) return;       // the expert list
            const int T = d.i[MKS_I_TILES], Sp = d.i[MKS_I_SPLITS], kc = d.i[MKS_I_KC], pieces = d.i[MKS_I_PIECES];
            const bool routed = d.i[MKS_I_GROUPS] < 0, reduce = d.i[MKS_I_REDUCE_GROUPS] != 0;
            const int G = routed ? *reinterpret_cast<const volatile int*>(&S.n_groups) : d.i[MKS_I_GROUPS];
            const int n_chunks = d.i[MKS_I_UNIT_STEPS] / d.i[MKS_I_CHUNK_STEPS], cb = d.i[MKS_I_CHUNK_BYTES];
            const int R = reduce ? T : G * T, Q = reduce ? G * Sp : Sp;
            const int w = max_panel_splits(A.xs_bytes, kc, A.M * pieces, pieces, reduce);
            int P = 1, panel = 0, c0 = 0, nc = 0, nb = 0, t0 = 0, t1 = 0;
            // the CTAs of this stage: all of them, unless it runs beside its neighbour
            int grid = grid_(), cta = cta_(), beside = 0;
            const int before = si > 0 ? S.geo[(n - 1) % GEO_RING].beside : 0;
            if (before > 0) {
                cta -= grid - before;
                grid = before;
            } else if ((d.flags & MKS_FLAG_NO_BARRIER) && si + 1 < A.n_stages && R > 0 && Q > 0 && grid > 1) {     // (one CTA cannot be shared)
                const mk_stage_desc& nx = A.prog[si + 1];
                if (nx.op == MKS_OP_GEMV && __ldg(&nx.i[MKS_I_TILES]) > 0) {
                    // every CTA must see the same number of groups, also when only the second stage is a routed one
                    if (nx.i[MKS_I_GROUPS] < 0 && !scout_wait(S, &S.route_seq, routes)) return;
                    beside = side_by_side(d, nx, *reinterpret_cast<const volatile int*>(&S.n_groups), grid);
                    grid -= beside;
                }
            }
            nc = grid;
            if (R > 0 && Q > 0 && cta >= 0 && cta < grid) {
                const int P0 = (Q + w - 1) / w;
                P = pick_panels(R, Q, P0, n_chunks, cb, kc, A.M, grid);
                if (P == 0) {
                    P = P0;                                    // more panels than half the CTAs: every CTA goes through all of them
                    panel = P > 1 ? -1 : 0;
                }
                if (P > 1 && panel >= 0) {
                    // panel p has the CTAs [grid q0 / Q, grid q1 / Q), q0 and q1 its first split and the next panel's
                    panel = cta * P / grid;
                    auto first = [&](int p) { return (grid * (Q * p / P) + Q - 1) / Q; };
                    while (panel > 0 && first(panel) > cta) panel--;
                    while (panel + 1 < P && first(panel + 1) <= cta) panel++;
                    c0 = first(panel);
                    nc = first(panel + 1) - c0;
                }
                const int k = cta - c0;
                t0 = (int)((unsigned)R * (unsigned)k / (unsigned)nc);   // (fewer than 2^24 units)
                t1 = (int)((unsigned)R * (unsigned)(k + 1) / (unsigned)nc);
                nb = t1 > t0 ? (panel < 0 ? P : 1) : 0;
            }
            if (lane_() == 0) {
                g.w = reinterpret_cast<const uint8_t*>(d.p[MKS_P_W]);
                g.w_shared = reinterpret_cast<const uint8_t*>(d.p[MKS_P_W_SHARED]);
                g.gstride = d.p[MKS_P_W_GSTRIDE];
                g.w_bytes = d.p[MKS_P_W_BYTES];
                g.T = T; g.S = Sp; g.G = G;
                g.n_chunks = n_chunks; g.chunk_steps = d.i[MKS_I_CHUNK_STEPS]; g.chunk_bytes = cb;
                g.ebps = d.i[MKS_I_FMT] == MKS_FMT_MXFP4 ? 32 : (d.i[MKS_I_BLOCK_SCALES] ? 2 : 0);
                g.reduce = reduce; g.routed = routed;
                g.Q = Q; g.P = P; g.panel = panel;
                g.t0 = t0; g.t1 = t1;
                g.g0 = 0; g.ng = 1;
                if (!reduce && d.i[MKS_I_X_GSTRIDE] != 0 && nb) {   // a staged input per group
                    g.g0 = t0 / T;
                    g.ng = (t1 - 1) / T - g.g0 + 1;
                }
                g.nb = nb * g.ng;
                g.stage = n;
                g.beside = beside;
            }
            __syncwarp();
            if (g.nb && lane_() < NCW) S.share[n % GEO_RING][lane_()] = batch_share(S, g, geo_batch(g, 0), lane_());
            __threadfence_block();
            __syncwarp();
            if (lane_() == 0) S.described = n + 1;
        }
    }
}

// ---- GEMV input staging ------------------------------------------------------------------------------------
// Stage K splits [seg0, seg1) of every sequence's input: normalise, round to bf16 (the model's activation type) and
// store as fp16 scaled by a power of two per column (bf16 weights: as bf16, unscaled).  Column `m` of the staged matrix
// is sequence m; with two pieces column M + m holds what fp16 lost of sequence m, so that the products see an
// fp32-exact input.  When groups are added up, consecutive splits belong to different groups: each has its own input,
// its own scale, and nothing to stage for a sequence that gives it no weight.
//
// What matters here is the number of dependent L2 round trips (about 0.7 us each on this part), not bytes: XB input
// loads and their norm weights per thread are in flight at once, the first of them together with the sums of squares
// behind 1/rms.  And the size of the code: every stage runs through it once, at the speed of instruction fetch.
constexpr int XB = 4;       // float4 groups per thread and round

// 1/rms of sequence `warp` from the 16-element sums of squares of the whole input vector: all loads of a lane in flight
// together (up to 8192 elements), added in a fixed order.
__device__ __forceinline__ float row_rstd(const mk_stage_desc& d, int m) {
    const int K = d.i[MKS_I_K_TOTAL], n16 = K / 16;
    const float* row = reinterpret_cast<const float*>(d.p[MKS_P_X_SSQ]) + (size_t)m * n16;
    float s = 0.f;
#pragma unroll 1
    for (int j0 = lane_(); j0 < n16; j0 += 512) {
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; u++) v[u] = j0 + 32 * u < n16 ? ldcg_f(row + j0 + 32 * u) : 0.f;
#pragma unroll
        for (int u = 0; u < 16; u++) s += v[u];
    }
    return rsqrtf(warp_sum(s) / (float)K + d.f[MKS_F_EPS]) * (d.f[MKS_F_IN_SCALE] != 0.f ? d.f[MKS_F_IN_SCALE] : 1.f);
}
// Exponent of the scale of a column whose largest magnitude has these bits: a = f * 2^e with f in [0.5, 1), the scale 2^(14 - e).
__device__ __forceinline__ int scale_exponent(int bits) {
    const int e = bits > 0 && bits < 0x7f800000 ? ((bits >> 23) & 0xff) - 126 : 0;
    return max(-100, min(100, 14 - e));
}
// Four and more sequences, one piece, no adding up of groups: four sequences' values of one column group at a time, the next
// four requested before the present ones are used.  (All 8 x 5120 values of a 27B layer: 10.5 us with a round trip per four.)
__device__ __noinline__ void stage_wide(Shared& S, const mk_stage_desc& d, int seg0, int seg1, int grp0) {
    const int kc = d.i[MKS_I_KC], M = S.A.M, cols = (seg1 - seg0) * kc, stride = xs_stride_bytes(cols);
    const bool norm = d.i[MKS_I_PROLOGUE] == MKS_P_NORM, bf16 = d.i[MKS_I_FMT] == MKS_FMT_BF16;
    const int xstride = d.i[MKS_I_X_STRIDE], c4n = cols >> 2;
    const float* x = reinterpret_cast<const float*>(d.p[MKS_P_X]) + (size_t)grp0 * d.i[MKS_I_X_GSTRIDE] + (size_t)seg0 * kc;
    const float* nw = reinterpret_cast<const float*>(d.p[MKS_P_NORM_W]) + (size_t)seg0 * kc;
    const float noff = d.f[MKS_F_NORM_OFF], bound = d.f[MKS_F_IN_BOUND];
    const bool final_form = bf16 || bound > 0.f;               // see stage_x
    float fscale = 1.f;
    if (tid_() < 8) {
        S.xmax[tid_()] = 0;
        if (bf16) S.xinv[tid_()] = 1.f;
    }
    if (!bf16 && final_form) {
        const int be = ((__float_as_int(bound) >> 23) & 0xff) - 126;          // bound < 2^be
        const int e = max(-100, min(100, 15 - be));
        fscale = __int_as_float((127 + e) << 23);
        if (tid_() < 8) S.xinv[tid_()] = __int_as_float((127 - e) << 23);
    }
    const int total = (c4n + NCT - 1) / NCT * ((M + 3) >> 2);
    float4 xn[4], wn = make_float4(0.f, 0.f, 0.f, 0.f);
    int li = tid_(), lm = 0;
    auto request = [&]() {
        if (norm && lm == 0 && li < c4n) wn = __ldg(reinterpret_cast<const float4*>(nw) + li);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            xn[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (li < c4n && lm + u < M) xn[u] = __ldcg(reinterpret_cast<const float4*>(x + (size_t)(lm + u) * xstride) + li);
        }
    };
    request();
    if (norm && warp_() < M) {
        const float r = row_rstd(d, warp_());
        if (lane_() == 0) S.rstd[warp_()] = r;
    }
    __syncwarp();
    consumer_sync();
    prof_mark(S, 4);
#pragma unroll 1
    for (int it = 0; it < total; it++) {
        float4 xv[4];
        const float4 w = wn;
        const int c4 = li, m0 = lm;
#pragma unroll
        for (int u = 0; u < 4; u++) xv[u] = xn[u];
        lm += 4;
        if (lm >= M) {
            lm = 0;
            li += NCT;
        }
        if (it + 1 < total) request();
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int m = m0 + u;
            if (m >= M) break;
            float v[4] = {xv[u].x, xv[u].y, xv[u].z, xv[u].w};
            if (norm) {
                const float r = S.rstd[m];
                v[0] = v[0] * r * (noff + w.x); v[1] = v[1] * r * (noff + w.y);
                v[2] = v[2] * r * (noff + w.z); v[3] = v[3] * r * (noff + w.w);
            }
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
            uint2 out = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            if (final_form) {
                if (!bf16) {
                    const __half2 a2 = __floats2half2_rn(bf_lo(out.x) * fscale, bf_hi(out.x) * fscale);
                    const __half2 b2 = __floats2half2_rn(bf_lo(out.y) * fscale, bf_hi(out.y) * fscale);
                    out = make_uint2(*reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&b2));
                }
            } else {
                // magnitudes of bf16 values compare like their bits
                const uint32_t a = max(max(out.x & 0x7FFFu, (out.x >> 16) & 0x7FFFu), max(out.y & 0x7FFFu, (out.y >> 16) & 0x7FFFu));
                const uint32_t mx = __reduce_max_sync(0xffffffffu, a);
                if (lane_() == 0) atomicMax(&S.xmax[m], (int)(mx << 16));
            }
            if (c4 < c4n) *reinterpret_cast<uint2*>(S.xs() + m * stride + c4 * 8) = out;
        }
    }
    if (final_form) return;                                    // the caller's barrier publishes it
    __syncwarp();
    consumer_sync();
    prof_mark(S, 5);
    if (tid_() < M) S.xinv[tid_()] = __int_as_float((127 - scale_exponent(S.xmax[tid_()])) << 23);
    // bf16 -> scaled fp16 in place, each thread its own column groups
#pragma unroll 1
    for (int c4 = tid_(); c4 < c4n; c4 += NCT) {
#pragma unroll 4
        for (int m = 0; m < M; m++) {
            const float sc = __int_as_float((127 + scale_exponent(S.xmax[m])) << 23);
            uint2* q = reinterpret_cast<uint2*>(S.xs() + m * stride + c4 * 8);
            const uint2 b = *q;
            const __half2 a2 = __floats2half2_rn(bf_lo(b.x) * sc, bf_hi(b.x) * sc), b2 = __floats2half2_rn(bf_lo(b.y) * sc, bf_hi(b.y) * sc);
            *q = make_uint2(*reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&b2));
        }
    }
}
// Routed groups that are added up (an expert's down projection), one piece, no norm: few sequences give a group any weight, so
// a warp takes one (K split, sequence) pair at a time, finds its scale by itself and leaves the other columns zero.  (The
// general staging below goes through all of them: 11 us for the ten experts of a panel at eight sequences.)
__device__ __noinline__ void stage_routed(Shared& S, const mk_stage_desc& d, int seg0, int seg1, int n_splits) {
    const int kc = d.i[MKS_I_KC], M = S.A.M, nseg = seg1 - seg0, stride = xs_stride_bytes(nseg * kc);
    const bool bf16 = d.i[MKS_I_FMT] == MKS_FMT_BF16;
    const float* x = reinterpret_cast<const float*>(d.p[MKS_P_X]);
    for (int i = tid_(); i < M * stride / 16; i += NCT) reinterpret_cast<uint4*>(S.xs())[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid_() < nseg * 8) S.xinv[tid_()] = 1.f;
    __syncwarp();
    consumer_sync();
    prof_mark(S, 4);
#pragma unroll 1
    for (int p = warp_(); p < nseg * M; p += NCW) {
        const int sg = p / M, m = p - sg * M, grp = n_splits == 1 ? seg0 + sg : (seg0 + sg) / n_splits;
        if (S.coef[grp * 8 + m] == 0.f) continue;
        const float* src = x + (size_t)grp * d.i[MKS_I_X_GSTRIDE] + (size_t)m * d.i[MKS_I_X_STRIDE] + (size_t)(seg0 + sg - grp * n_splits) * kc;
        uint8_t* dst = S.xs() + m * stride + sg * kc * 2;
        uint32_t mx = 0;
#pragma unroll 1
        for (int e = lane_() * 4; e < kc; e += 512) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = e + u * 128 < kc ? __ldcg(reinterpret_cast<const float4*>(src + e + u * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v[u].x, v[u].y), hi = __floats2bfloat162_rn(v[u].z, v[u].w);
                const uint2 b = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                mx = max(max(mx, max(b.x & 0x7FFFu, (b.x >> 16) & 0x7FFFu)), max(b.y & 0x7FFFu, (b.y >> 16) & 0x7FFFu));   // magnitudes compare like their bits
                if (e + u * 128 < kc) *reinterpret_cast<uint2*>(dst + (e + u * 128) * 2) = b;
            }
        }
        __syncwarp();
        if (!bf16) {
            const int ex = scale_exponent((int)(__reduce_max_sync(0xffffffffu, mx) << 16));
            const float sc = __int_as_float((127 + ex) << 23);
            if (lane_() == 0) S.xinv[sg * 8 + m] = __int_as_float((127 - ex) << 23);
#pragma unroll 2
            for (int e = lane_() * 4; e < kc; e += 128) {      // the lane's own values
                uint2* q = reinterpret_cast<uint2*>(dst + e * 2);
                const uint2 b = *q;
                const __half2 a2 = __floats2half2_rn(bf_lo(b.x) * sc, bf_hi(b.x) * sc), b2 = __floats2half2_rn(bf_lo(b.y) * sc, bf_hi(b.y) * sc);
                *q = make_uint2(*reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&b2));
            }
        }
        __syncwarp();
    }
}
// (PLAIN: one piece, no adding up of groups: nearly every stage)
template <bool PLAIN>
__device__ __forceinline__ void stage_x(Shared& S, const mk_stage_desc& d, int seg0, int seg1, int grp0, int n_splits) {
    const int kc = d.i[MKS_I_KC], M = S.A.M;
    const bool reduce = !PLAIN && d.i[MKS_I_REDUCE_GROUPS] != 0, norm = d.i[MKS_I_PROLOGUE] == MKS_P_NORM;
    const bool bf16 = d.i[MKS_I_FMT] == MKS_FMT_BF16, two = !PLAIN && d.i[MKS_I_PIECES] == 2;
    const int nseg = seg1 - seg0, cols = nseg * kc, stride = xs_stride_bytes(cols);
    const float* x = reinterpret_cast<const float*>(d.p[MKS_P_X]);
    const float* nw = reinterpret_cast<const float*>(d.p[MKS_P_NORM_W]);
    const int xstride = d.i[MKS_I_X_STRIDE], gstride = d.i[MKS_I_X_GSTRIDE];
    const float noff = d.f[MKS_F_NORM_OFF];
    const int c4n = cols >> 2, k4n = kc >> 2;
    const int total = (c4n + NCT - 1) / NCT * M;                      // a thread's groups: column group tid + i NCT of sequence m, m fastest
    const int nscale = reduce ? nseg * 8 : 8;
    // A bound on |input| known to the host (a normed vector cannot exceed sqrt(K) max|weight|) fixes the power-of-two
    // scale of the fp16 copy up front: the values then go to shared memory in their final form in one pass.
    const float bound = d.f[MKS_F_IN_BOUND];
    const bool fixed_scale = bound > 0.f && !bf16 && !two;
    // what a pass over the input leaves: final values; bf16 copies and their largest magnitudes; the latter alone
    enum { FINAL, COPY, LARGEST };
    int mode = bf16 || fixed_scale ? FINAL : (two ? LARGEST : COPY);
    bool first = true;
    const bool once = PLAIN && mode == COPY && total <= XB;           // the bf16 values of the only round wait in registers
    float4 xv[XB], wv[XB];
    float fscale = 1.f;
    if (tid_() < nscale) {
        S.xmax[tid_()] = 0;
        if (bf16) S.xinv[tid_()] = 1.f;
    }
    if (fixed_scale) {
        const int be = ((__float_as_int(bound) >> 23) & 0xff) - 126;          // bound < 2^be
        const int e = max(-100, min(100, 15 - be));
        fscale = __int_as_float((127 + e) << 23);
        if (tid_() < nscale) S.xinv[tid_()] = __int_as_float((127 - e) << 23);
    }
#pragma unroll 1
    for (;;) {
        int li = tid_(), lm = 0, pi = tid_(), pm = 0;                 // the next group to request, to work on
#pragma unroll 1
        for (int base = 0; base < total; base += XB) {
#pragma unroll
            for (int u = 0; u < XB; u++) {
                xv[u] = wv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (base + u < total && li < c4n) {
                    int grp = grp0, o = seg0 * kc + li * 4;
                    if (reduce) {
                        const int sg = li / k4n;
                        grp = n_splits == 1 ? seg0 + sg : (seg0 + sg) / n_splits;
                        o = (seg0 + sg - grp * n_splits) * kc + (li - sg * k4n) * 4;
                    }
                    if (!reduce || S.coef[grp * 8 + lm] != 0.f) xv[u] = __ldcg(reinterpret_cast<const float4*>(x + (size_t)grp * gstride + lm * xstride + o));
                    if (norm) wv[u] = __ldg(reinterpret_cast<const float4*>(nw + o));
                }
                if (++lm == M) {
                    lm = 0;
                    li += NCT;
                }
            }
            if (first) {
                first = false;
                if (norm && warp_() < M) {                         // while the other warps only wait for x
                    const float r = row_rstd(d, warp_());
                    if (lane_() == 0) S.rstd[warp_()] = r;
                }
                __syncwarp();
                consumer_sync();
                prof_mark(S, 4);
            }
#pragma unroll
            for (int u = 0; u < XB; u++) {
                if (base + u >= total) break;
                const int c4 = pi, m = pm;
                const bool live = c4 < c4n;
                if (++pm == M) {
                    pm = 0;
                    pi += NCT;
                }
                const int sg = reduce ? c4 / k4n : 0;
                float v[4] = {xv[u].x, xv[u].y, xv[u].z, xv[u].w};
                if (norm) {
                    const float r = S.rstd[m];
                    v[0] = v[0] * r * (noff + wv[u].x); v[1] = v[1] * r * (noff + wv[u].y);
                    v[2] = v[2] * r * (noff + wv[u].z); v[3] = v[3] * r * (noff + wv[u].w);
                }
                if (!two) {
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] = bf16_round(v[i]);
                }
                if (once) xv[u] = make_float4(v[0], v[1], v[2], v[3]);
                if (mode != FINAL) {
                    // (magnitudes compare like their bits) a warp's 32 groups are one sequence's and lie in at most two splits
                    const int bits = live ? __float_as_int(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])))) : 0;
                    const int s0 = PLAIN ? 0 : __shfl_sync(0xffffffffu, sg, 0);
                    const int a = __reduce_max_sync(0xffffffffu, sg == s0 ? bits : 0);
                    if (lane_() == 0 && a > 0) atomicMax(&S.xmax[s0 * 8 + m], a);
                    if (!PLAIN) {
                        const int b = __reduce_max_sync(0xffffffffu, sg != s0 ? bits : 0);
                        if (lane_() == 0 && b > 0) atomicMax(&S.xmax[s0 * 8 + 8 + m], b);
                    }
                }
                if (live && mode != LARGEST && !once) {
                    uint8_t* dst = S.xs() + m * stride + c4 * 8;
                    const bool as_bf16 = bf16 || mode == COPY;
                    if (!as_bf16) {
                        const float sc = two ? __int_as_float(S.xmax[sg * 8 + m]) : fscale;
#pragma unroll
                        for (int i = 0; i < 4; i++) v[i] *= sc;
                    }
                    uint32_t hi[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const __nv_bfloat162 b2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                        const __half2 h2 = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                        hi[i] = as_bf16 ? *reinterpret_cast<const uint32_t*>(&b2) : *reinterpret_cast<const uint32_t*>(&h2);
                        if (two) {                                 // what the first piece lost
                            v[2 * i] -= bf16 ? __low2float(b2) : __low2float(h2);
                            v[2 * i + 1] -= bf16 ? __high2float(b2) : __high2float(h2);
                        }
                    }
                    *reinterpret_cast<uint2*>(dst) = make_uint2(hi[0], hi[1]);
                    if (two) {
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const __nv_bfloat162 b2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                            const __half2 h2 = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                            hi[i] = bf16 ? *reinterpret_cast<const uint32_t*>(&b2) : *reinterpret_cast<const uint32_t*>(&h2);
                        }
                        *reinterpret_cast<uint2*>(dst + M * stride) = make_uint2(hi[0], hi[1]);
                    }
                }
            }
        }
        if (mode == FINAL) return;                                 // the caller's barrier publishes it
        __syncwarp();
        consumer_sync();
        prof_mark(S, 5);
        if (once) {
            int m = 0, c4 = tid_();
#pragma unroll
            for (int u = 0; u < XB; u++) {
                if (u >= total) break;
                const int e = scale_exponent(S.xmax[m]);
                const float sc = __int_as_float((127 + e) << 23);
                if (c4 < c4n) {
                    const __half2 a2 = __floats2half2_rn(xv[u].x * sc, xv[u].y * sc), b2 = __floats2half2_rn(xv[u].z * sc, xv[u].w * sc);
                    *reinterpret_cast<uint2*>(S.xs() + m * stride + c4 * 8) =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&b2));
                }
                if (tid_() == 0) S.xinv[m] = __int_as_float((127 - e) << 23);
                if (++m == M) {
                    m = 0;
                    c4 += NCT;
                }
            }
            return;
        }
        if (tid_() < nscale && (tid_() & 7) < M) {
            const int e = scale_exponent(S.xmax[tid_()]);
            S.xmax[tid_()] = (127 + e) << 23;
            S.xinv[tid_()] = __int_as_float((127 - e) << 23);
            if (two) S.xinv[tid_() + M] = __int_as_float((127 - e) << 23);
        }
        __syncwarp();
        consumer_sync();
        prof_mark(S, 6);
        if (mode == COPY) break;
        mode = FINAL;
    }
    // bf16 -> scaled fp16 in place, eight values per thread and turn
    const int c8n = cols >> 3, k8n = kc >> 3;
#pragma unroll 1
    for (int c8 = tid_(); c8 < c8n; c8 += NCT) {
        const int sg = reduce ? c8 / k8n : 0;
#pragma unroll 1
        for (int m = 0; m < M; m++) {
            uint4* pq = reinterpret_cast<uint4*>(S.xs() + m * stride) + c8;
            uint4 q = *pq;
            const float sc = __int_as_float(S.xmax[sg * 8 + m]);
            auto conv = [&](uint32_t w) {
                const __half2 h = __floats2half2_rn(bf_lo(w) * sc, bf_hi(w) * sc);
                return *reinterpret_cast<const uint32_t*>(&h);
            };
            q.x = conv(q.x); q.y = conv(q.y); q.z = conv(q.z); q.w = conv(q.w);
            *pq = q;
        }
    }
}

// ---- tensor-parallel all-reduce of one output tile -------------------------------------------------------------
// Mailbox of a rank: [2 halves][MAILBOX_TILES][ranks][128] 64-bit words (value | tag << 32), then the key
// exchange area [2][ranks][8][2].  Each lane owns four words of the tile.
__device__ __noinline__ float4 allreduce_tile(Shared& S, const Args& A, u64 seq, int tile, float4 in) {
    const float acc[4] = {in.x, in.y, in.z, in.w};
    const uint32_t tag = (uint32_t)seq;
    const size_t base = (((size_t)(seq & 1) * MAILBOX_TILES + tile) * MKS_MAX_RANKS);
#pragma unroll 1
    for (int r = 0; r < A.tp; r++) {
        unsigned long long* dst = A.mailbox[r] + (base + A.rank) * 128 + lane_() * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) st_relaxed_sys_u64(dst + i, ((u64)tag << 32) | __float_as_uint(acc[i]));
    }
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int r = 0; r < A.tp; r++) {
        const unsigned long long* src = A.mailbox[A.rank] + (base + r) * 128 + lane_() * 4;
        u64 w[4];
        Spin2 s;
        bool fail = false;
#pragma unroll 1
        for (;;) {                                               // the warp leaves together
            bool ok = true;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                w[i] = ld_relaxed_sys_u64(src + i);
                ok = ok && (uint32_t)(w[i] >> 32) == tag;
            }
            if (__all_sync(0xffffffffu, ok)) break;
            if (!ok && MKS_SPIN_FAIL(S, s, WS_MAILBOX)) fail = true;
            if (__any_sync(0xffffffffu, fail)) return in;         // (the abort flag is set)
        }
#pragma unroll
        for (int i = 0; i < 4; i++) sum[i] += __uint_as_float((uint32_t)w[i]);
    }
    return make_float4(sum[0], sum[1], sum[2], sum[3]);
}

// ---- GEMV stage (consumers) ----------------------------------------------------------------------------------
// Lane (g = lane / 4, t = lane % 4) of a warp holds, per tile step, 8 bytes of row g and 8 bytes of row g + 8: the
// values that MMA j of the step multiplies with input columns k0 + 16 j + 4 t + {0, 1, 2, 3}.  Its accumulators are
// rows g, g + 8 x sequences 2t, 2t + 1.
//
// (volatile: they stay behind the wait for the copies they read)
__device__ __forceinline__ uint4 lds_u4(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float2 lds_f2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
// One tile step: accumulates into acc / acc2 (two chains where a warp's own MMAs would wait for each other).
template <int FMT>
__device__ __forceinline__ void tile_step(uint32_t sl, uint32_t sc, int st, const uint8_t* xk, float (&acc)[4], float (&acc2)[4]) {
    const uint4 wq = lds_u4(sl);
    if (FMT == MKS_FMT_MXFP4) {
        // The conversion unit (cvt ... e2m1x2) is the scarcest pipe of this loop, so only half of the
        // values go through it.  The 32 columns of scale group 0 (MMAs 0 and 1) arrive with their bits
        // pre-arranged by the packer: every 32-bit word yields four f16x2 registers with shifts and masks
        // alone (sign at bit 15, the three magnitude bits at 11..9 of each half: the value times 2^-14).  Scale group 1 (MMAs 2 and 3) keeps plain nibbles.
        const uint32_t scw = lds_u32(sc);
        float t0[4] = {0.f, 0.f, 0.f, 0.f};                                    // scale group 0: MMAs 0, 1
        float u0[4] = {0.f, 0.f, 0.f, 0.f};                                    // scale group 1: MMAs 2, 3
        uint2 b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const uint2*>(xk + j * 32);
        {
            const uint32_t lo = wq.x, hi = wq.z;                  // row g, row g + 8
            uint32_t a[4];
            a[0] = lo & 0x8E008E00u;
            a[1] = hi & 0x8E008E00u;
            a[2] = (lo << 3) & 0x8E008E00u;
            a[3] = (hi << 3) & 0x8E008E00u;
            mma_f16(t0, a, b[0].x, b[0].y);
            a[0] = ((lo << 1) & 0x80008000u) | ((lo << 6) & 0x0E000E00u);
            a[1] = ((hi << 1) & 0x80008000u) | ((hi << 6) & 0x0E000E00u);
            a[2] = ((lo << 2) & 0x80008000u) | ((lo << 9) & 0x0E000E00u);
            a[3] = ((hi << 2) & 0x80008000u) | ((hi << 9) & 0x0E000E00u);
            mma_f16(t0, a, b[1].x, b[1].y);
        }
        {
            const uint32_t lo = wq.y, hi = wq.w;
            uint32_t a[4];
            a[0] = cvt_e2m1x2(lo);
            a[2] = cvt_e2m1x2(lo >> 8);
            a[1] = cvt_e2m1x2(hi);
            a[3] = cvt_e2m1x2(hi >> 8);
            mma_f16(u0, a, b[2].x, b[2].y);
            a[0] = cvt_e2m1x2(lo >> 16);
            a[2] = cvt_e2m1x2(lo >> 24);
            a[1] = cvt_e2m1x2(hi >> 16);
            a[3] = cvt_e2m1x2(hi >> 24);
            mma_f16(u0, a, b[3].x, b[3].y);
        }
        // e8m0 scales: bytes [row g: group 0, group 1, row g + 8: group 0, group 1]; group 0 is collected in `acc`, which takes
        // back the 2^14 at the end of the tile
        const float s00 = __uint_as_float((scw << 23) & 0x7F800000u), s01 = __uint_as_float((scw << 15) & 0x7F800000u);
        const float s10 = __uint_as_float((scw << 7) & 0x7F800000u), s11 = __uint_as_float((scw >> 1) & 0x7F800000u);
        acc[0] = fmaf(t0[0], s00, acc[0]); acc[1] = fmaf(t0[1], s00, acc[1]);
        acc[2] = fmaf(t0[2], s10, acc[2]); acc[3] = fmaf(t0[3], s10, acc[3]);
        acc2[0] = fmaf(u0[0], s01, acc2[0]); acc2[1] = fmaf(u0[1], s01, acc2[1]);
        acc2[2] = fmaf(u0[2], s11, acc2[2]); acc2[3] = fmaf(u0[3], s11, acc2[3]);
    } else if (FMT == MKS_FMT_FP8) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t lo = j == 0 ? wq.x : wq.y, hi = j == 0 ? wq.z : wq.w;
            uint32_t a[4];
            a[0] = cvt_e4m3x2(lo);
            a[2] = cvt_e4m3x2(lo >> 16);
            a[1] = cvt_e4m3x2(hi);
            a[3] = cvt_e4m3x2(hi >> 16);
            const uint2 b = *reinterpret_cast<const uint2*>(xk + j * 32);
            mma_f16(acc, a, b.x, b.y);
        }
    } else if (FMT == MKS_FMT_INT8) {
        const uint32_t x0 = wq.x ^ 0x80808080u, x1 = wq.y ^ 0x80808080u, x2 = wq.z ^ 0x80808080u, x3 = wq.w ^ 0x80808080u;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t lo = j == 0 ? x0 : x1, hi = j == 0 ? x2 : x3;
            uint32_t a[4];
            a[0] = cvt_s8x2(lo, 0x4140);
            a[2] = cvt_s8x2(lo, 0x4342);
            a[1] = cvt_s8x2(hi, 0x4140);
            a[3] = cvt_s8x2(hi, 0x4342);
            const uint2 b = *reinterpret_cast<const uint2*>(xk + j * 32);
            mma_f16(j == 0 ? acc : acc2, a, b.x, b.y);
        }
    } else {
        uint32_t a[4] = {wq.x, wq.z, wq.y, wq.w};                 // row g: (x, y), row g + 8: (z, w)
        const uint2 b = *reinterpret_cast<const uint2*>(xk);
        if (st & 2) mma_bf16(acc2, a, b.x, b.y);
        else mma_bf16(acc, a, b.x, b.y);
    }
}

// Partial tiles of a stage with several panels: [tile][panel][8 sequences][8 row pairs][2] words (value | tag << 32); only
// live sequences' columns are written and read.  A launch's tags are its own (the host counts them over all launches, apart
// from the barrier counter, which a caller may start over); a captured launch runs again with the same ones, so there the
// words are left zero, which no tag is (cleared in every launch: 1 to 2.5 % of a step).
__device__ __forceinline__ unsigned long long* tile_words(unsigned long long* part, int tile_panel) {
    return part + (size_t)tile_panel * 128 + (lane_() & 3) * 32 + (lane_() >> 2) * 2;
}
__device__ __noinline__ void clear_tile(Shared& S, unsigned long long* src, int P) {
    const int m0 = 2 * (lane_() & 3);
#pragma unroll 1
    for (int p = 0; p < P; p++, src += 128) {
        if (m0 < S.A.M) __stcg(reinterpret_cast<ulonglong2*>(src), make_ulonglong2(0ull, 0ull));
        if (m0 + 1 < S.A.M) __stcg(reinterpret_cast<ulonglong2*>(src + 16), make_ulonglong2(0ull, 0ull));
    }
}
__device__ __forceinline__ void publish_tile(unsigned long long* dst, uint32_t tag, int M, const float (&v)[4]) {
    chaos_delay();
    const u64 t = (u64)tag << 32;
    const int m0 = 2 * (lane_() & 3);
    if (m0 < M) asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(dst), "l"(t | __float_as_uint(v[0])), "l"(t | __float_as_uint(v[2])) : "memory");
    if (m0 + 1 < M) asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(dst + 16), "l"(t | __float_as_uint(v[1])), "l"(t | __float_as_uint(v[3])) : "memory");
}
// The sum of the P partial tiles at `src`, in panel order, four panels' words in flight.  False: a wait ran out.
__device__ __forceinline__ bool collect_tile(Shared& S, const unsigned long long* src, uint32_t tag, int P, float (&acc)[4]) {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    const int m0 = 2 * (lane_() & 3);
    const bool l0 = m0 < S.A.M, l1 = m0 + 1 < S.A.M;
#pragma unroll 1
    for (int p0 = 0; p0 < P; p0 += 4) {
        u64 w[4][4];
        Spin2 s;
        bool fail = false;
#pragma unroll 1
        for (;;) {                                               // the warp leaves together
            bool ok = true;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                w[u][0] = w[u][1] = w[u][2] = w[u][3] = (u64)tag << 32;
                if (p0 + u < P) {
                    const unsigned long long* q = src + (size_t)(p0 + u) * 128;
                    if (l0) asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w[u][0]), "=l"(w[u][2]) : "l"(q) : "memory");
                    if (l1) asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w[u][1]), "=l"(w[u][3]) : "l"(q + 16) : "memory");
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int i = 0; i < 4; i++) ok = ok && (uint32_t)(w[u][i] >> 32) == tag;
            if (__all_sync(0xffffffffu, ok)) break;
            if (!ok && MKS_SPIN_FAIL(S, s, WS_TILE)) fail = true;
            if (__any_sync(0xffffffffu, fail)) return false;
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (p0 + u < P)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[i] += __uint_as_float((uint32_t)w[u][i]);
    }
    return true;
}

// Epilogue of a finished tile (`row_tile` counts the tiles of all groups, unless the groups were added up).  False: a wait
// ran out.
__device__ __noinline__ bool finish_tile(Shared& S, const mk_stage_desc& d, u64 ar_seq, int row_tile, float4 in) {
    float acc[4] = {in.x, in.y, in.z, in.w};
    const int g = lane_() >> 2, t = lane_() & 3, epi = d.i[MKS_I_EPILOGUE];
    const int T = d.i[MKS_I_TILES];
    const int grp = row_tile < T ? 0 : row_tile / T, tile = row_tile - grp * T;
    if (d.i[MKS_I_ALLREDUCE] != 0 && S.A.tp > 1) {
        const float4 r = allreduce_tile(S, S.A, ar_seq, tile, make_float4(acc[0], acc[1], acc[2], acc[3]));
        if (__any_sync(0xffffffffu, S.abort_flag != 0)) return false;
        acc[0] = r.x; acc[1] = r.y; acc[2] = r.z; acc[3] = r.w;
    }
    // rows g, g + 8 of the tile x sequences 2t, 2t + 1
    const int ostride = d.i[MKS_I_OUT_STRIDE], nvalid = d.i[MKS_I_N_VALID];
    const int row = epi == MKS_E_GLU ? tile * 8 + g : tile * 16 + g;
    float* out = reinterpret_cast<float*>(d.p[MKS_P_OUT]) + (size_t)grp * d.i[MKS_I_OUT_GSTRIDE] + (size_t)(2 * t) * ostride + row;
    const bool l0 = 2 * t < S.A.M, l1 = 2 * t + 1 < S.A.M;
    const bool va = row < nvalid, vb = epi != MKS_E_GLU && row + 8 < nvalid;
    if (epi == MKS_E_RESID) {
        if (l0) { acc[0] += ldcg_f(out); acc[2] += ldcg_f(out + 8); }
        if (l1) { acc[1] += ldcg_f(out + ostride); acc[3] += ldcg_f(out + ostride + 8); }
    }
    float* ssq = epi == MKS_E_STORE || epi == MKS_E_RESID ? reinterpret_cast<float*>(d.p[MKS_P_OUT_SSQ]) : nullptr;
    float a = acc[0], b = acc[2];
    bool live = l0;
#pragma unroll 1
    for (int q = 0; q < 2; q++) {
        if (epi == MKS_E_GLU) a = (d.i[MKS_I_ACT] == MKS_ACT_GELU_TANH ? gelu_tanh_f(a) : silu_f(a)) * b;
        if (epi == MKS_E_LOGITS) {
            const float cap = d.f[MKS_F_SOFTCAP];
            if (cap > 0.f) {
                a = cap * tanhf(a / cap);
                b = cap * tanhf(b / cap);
            }
            const int r0 = (int)d.p[MKS_P_ROW_BASE] + row;
            u64 k = va ? score_key(a, r0) : 0;
            const u64 k2 = vb ? score_key(b, r0 + 8) : 0;
            k = k2 > k ? k2 : k;
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                const u64 other = __shfl_xor_sync(0xffffffffu, k, o);
                k = other > k ? other : k;
            }
            if (g == 0 && live) atomicMax(reinterpret_cast<unsigned long long*>(&S.keys_s[2 * t + q]), (unsigned long long)k);
        }
        if (live) {
            if (va) __stcg(out, a);
            if (vb) __stcg(out + 8, b);
        }
        if (ssq) {                                              // the sums of squares a later norm of this vector needs (whole tiles only)
            float s2 = a * a + b * b;
            // sum over the eight lanes that share t (the 16 rows of the tile), in a fixed order
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (g == 0 && live) __stcg(ssq + (size_t)(2 * t + q) * (nvalid / 16) + tile, s2);
        }
        if (S.A.M == 1) break;
        a = acc[1]; b = acc[3];
        live = l1;
        out += ostride;
    }
    return true;
}

// What happens to a tile's sum over this CTA's panel.  False: a wait ran out.
__device__ __forceinline__ bool deliver(Shared& S, const mk_stage_desc& d, const Geo& gm, u64 ar_seq, uint32_t tag, int panel, int row_tile, const float (&v)[4]) {
    if (gm.P == 1) return finish_tile(S, d, ar_seq, row_tile, make_float4(v[0], v[1], v[2], v[3]));
    publish_tile(tile_words(reinterpret_cast<unsigned long long*>(d.p[MKS_P_PART]), row_tile * gm.P + panel), tag, S.A.M, v);
    return true;
}

// A batch of a stage, input staged: this warp's chunks, tile by tile.  The first and the last tile may be shared with the
// warps before and behind.  One call per batch: a call per tile spilled the caller's registers around each, and spills of
// 544 threads do not fit the L1 that the shared-memory carve-out leaves.
template <int FMT>
__device__ __forceinline__ bool multiply(Shared& S, const mk_stage_desc& d, const Geo& gm, const Batch bt, int b, u64 ar_seq, uint32_t tag, uint32_t n_stage) {
    constexpr int STEP_BYTES = (FMT == MKS_FMT_MXFP4 ? 4 : (FMT == MKS_FMT_BF16 ? 1 : 2)) * 32;   // staged input bytes of one tile step
    const int depth = S.A.ring_depth;
    Feed f = S.cur[warp_()].f;
    f.src += lane_() * 16;
    f.eoff -= lane_() * 12;
    f.rd += lane_() * 16;
    const int ring_bytes = depth * BLOCK_BYTES;
    const uint32_t ring_end = smem_u32(S.ring()) + (warp_() + 1) * ring_bytes;
    __syncwarp();
    if (lane_() == 0) S.cur[warp_()].now = n_stage;
    __syncwarp();
    const int stride = xs_stride_bytes((bt.seg1 - bt.seg0) * d.i[MKS_I_KC]), chunk_steps = gm.chunk_steps, n_chunks = gm.n_chunks;
    const Share sh = b == 0 ? S.share[n_stage % GEO_RING][warp_()] : batch_share(S, gm, bt, warp_());
    const bool scales = FMT == MKS_FMT_MXFP4 || (FMT == MKS_FMT_FP8 && gm.ebps != 0);
    const int cpt = sh.cpt, c1 = sh.c1;
    int c = sh.c, tl = sh.tl, k = sh.k;
    bool begun = k == 0, has_head = false, ok = true;
    float sum[4] = {0.f, 0.f, 0.f, 0.f}, head[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    while (c < c1 && ok) {
        // consecutive chunks of one tile: one K split's at a time when groups are added up
        float s0 = 1.f, s1 = 1.f, f0 = 1.f, f1 = 1.f, x0, x1;
        int ke = cpt;
        {
            int sg = 0, grp = 0, tile = bt.t0 + tl;
            if (gm.reduce) {
                sg = n_chunks == 1 ? k : k / n_chunks;
                ke = (sg + 1) * n_chunks;
                grp = gm.S == 1 ? bt.seg0 + sg : (bt.seg0 + sg) / gm.S;
                f0 = S.coef[grp * 8 + 2 * (lane_() & 3)];
                f1 = S.coef[grp * 8 + 2 * (lane_() & 3) + 1];
            } else if (tile >= gm.T) {
                grp = tile / gm.T;
                tile -= grp * gm.T;
            }
            const float* rs = group_row_scale(S, d, grp, gm.G);
            if (rs) {
                s0 = __ldg(rs + tile * 16 + (lane_() >> 2));
                s1 = __ldg(rs + tile * 16 + (lane_() >> 2) + 8);
            }
            x0 = S.xinv[sg * 8 + 2 * (lane_() & 3)];
            x1 = S.xinv[sg * 8 + 2 * (lane_() & 3) + 1];
        }
        const int run = min(ke - k, c1 - c);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        {
            float acc2[4] = {0.f, 0.f, 0.f, 0.f};
            float tot[4] = {0.f, 0.f, 0.f, 0.f};                // block-scaled FP8: the sum over 128-column blocks
            // lanes beyond the staged columns read a live one (their accumulators are never used): predicated zeros cost a tenth of the loop
            const uint8_t* xk = S.xs() + min(lane_() >> 2, S.A.M * d.i[MKS_I_PIECES] - 1) * stride + (lane_() & 3) * 8 + k * chunk_steps * STEP_BYTES;
            // the stream's blocks end where a chunk with scales or padding, or a run of chunks, ends
            int steps = run * chunk_steps, in = gm.chunk_bytes != chunk_steps * 512 ? chunk_steps : steps;
            const uint32_t sc_off = BLOCK_STEPS * 512 - lane_() * 16 + (lane_() >> 2) * 4;
#pragma unroll 1
            while (steps > 0) {
                __syncwarp();                                  // the warp has read the block before
                if (f.ahead == depth - 1 && f.steps >= BLOCK_STEPS) {
                    feed_one(f, f.rd == ring_end - ring_bytes + lane_() * 16 ? ring_end - BLOCK_BYTES + lane_() * 16 : f.rd - BLOCK_BYTES);
                } else {
                    feed(S, f, depth, ring_end);
                    if (f.ahead == 0) {                        // (a stream that was refused: the launch has failed)
                        ok = false;
                        break;
                    }
                }
                wait_block(depth);
                __syncwarp();
                const uint32_t sl = f.rd;
                const int ns = min(BLOCK_STEPS, in);
                if (ns == BLOCK_STEPS) {
#pragma unroll
                    for (int st = 0; st < BLOCK_STEPS; st++, xk += STEP_BYTES) tile_step<FMT>(sl + st * 512, sl + sc_off + st * 32, st, xk, acc, acc2);
                } else {
#pragma unroll 1
                    for (int st = 0; st < ns; st++, xk += STEP_BYTES) tile_step<FMT>(sl + st * 512, sl + sc_off + st * 32, st, xk, acc, acc2);
                }
                if (FMT == MKS_FMT_FP8 && scales) {
                    // one scale per 128 k for rows 0-7 of the tile and one for rows 8-15 (a GLU tile pairs two matrices)
                    const float2 bs = lds_f2(sl + BLOCK_STEPS * 512 - lane_() * 16);
                    tot[0] = fmaf(acc[0] + acc2[0], bs.x, tot[0]); tot[1] = fmaf(acc[1] + acc2[1], bs.x, tot[1]);
                    tot[2] = fmaf(acc[2] + acc2[2], bs.y, tot[2]); tot[3] = fmaf(acc[3] + acc2[3], bs.y, tot[3]);
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                    acc2[0] = acc2[1] = acc2[2] = acc2[3] = 0.f;
                }
                steps -= ns;
                in -= ns;
                if (in == 0) in = chunk_steps;
                f.ahead--;
                f.rd += BLOCK_BYTES;
                if (f.rd >= ring_end) f.rd -= ring_bytes;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i] = acc[i] * (FMT == MKS_FMT_MXFP4 ? 16384.f : 1.f) + acc2[i] + (FMT == MKS_FMT_FP8 ? tot[i] : 0.f);
        }
        __syncwarp();
        // undo the input scaling, fold the second piece's columns onto the first
        acc[0] *= x0; acc[1] *= x1; acc[2] *= x0; acc[3] *= x1;
        if (d.i[MKS_I_PIECES] == 2) {
            // columns [0, M) + columns [M, 2M): lane t holds columns 2t, 2t + 1
            const int t = lane_() & 3;
            float add[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int src_col = 2 * t + (i & 1) + S.A.M;              // the partner column
                const int src = (lane_() & ~3) | ((src_col >> 1) & 3);
                const float same = __shfl_sync(0xffffffffu, acc[i], src), other = __shfl_sync(0xffffffffu, acc[i ^ 1], src);
                add[i] = (src_col & 1) == (i & 1) ? same : other;
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (2 * t + (i & 1) < S.A.M) acc[i] += add[i];
        }
        sum[0] = fmaf(acc[0] * s0, f0, sum[0]); sum[1] = fmaf(acc[1] * s0, f1, sum[1]);
        sum[2] = fmaf(acc[2] * s1, f0, sum[2]); sum[3] = fmaf(acc[3] * s1, f1, sum[3]);
        c += run;
        k += run;
        if (k == cpt || c == c1) {
            if (!begun) {
                // the warp that has the tile's beginning adds this to it
                has_head = true;
#pragma unroll
                for (int i = 0; i < 4; i++) head[i] = sum[i];
            } else if (k == cpt) {
                ok = deliver(S, d, gm, ar_seq, tag, bt.panel, bt.t0 + tl, sum) && ok;
            } else {
                break;                                             // c == c1, inside a tile that began here: `sum` is its first part
            }
            begun = true;
            sum[0] = sum[1] = sum[2] = sum[3] = 0.f;
            if (k == cpt) {
                k = 0;
                tl++;
            } else {
                k = 0;                                             // (the whole range lay inside another warp's tile)
            }
        }
    }
    __syncwarp();
    feed(S, f, depth, ring_end);
    if (lane_() == 0) {
        S.cur[warp_()].f = f;
    }
    __syncwarp();
    consumer_sync();                                             // the staging area is free: it takes the shared tiles
    float4* tiles = reinterpret_cast<float4*>(S.xs()) + lane_();
    tiles[warp_() * 32] = make_float4(head[0], head[1], head[2], head[3]);         // (zeros if there is none)
    __syncwarp();
    consumer_sync();
    if (k > 0 && c == c1 && c > sh.c && ok) {
        // the warps behind this one, up to the one that has the tile's last chunk
        const int end = (tl + 1) * cpt - 1, last = sh.per > 0 ? end / sh.per : (NCW * end + NCW - 1) / -sh.per;
#pragma unroll 4
        for (int v = warp_() + 1; v <= last; v++) {
            const float4 x = tiles[v * 32];
            sum[0] += x.x; sum[1] += x.y; sum[2] += x.z; sum[3] += x.w;
        }
        ok = deliver(S, d, gm, ar_seq, tag, bt.panel, bt.t0 + tl, sum);
    }
    __syncwarp();
    return ok;
}

template <int FMT>
__device__ __forceinline__ void gemv_stage(Shared& S, const mk_stage_desc& d, const Geo& gm, u64 ar_seq, uint32_t tag, uint32_t n_stage) {
    const bool logits = d.i[MKS_I_EPILOGUE] == MKS_E_LOGITS;
    if (logits && tid_() < 8) S.keys_s[tid_()] = 0;
    bool ok = true;                                              // no wait of this warp ran out
#pragma unroll 1
    for (int b = 0; b < gm.nb; b++) {
        const Batch bt = geo_batch(gm, b);
        __syncwarp();
        if (b) consumer_sync();                                  // everybody is done with the staging area
        if (d.i[MKS_I_PIECES] == 1 && !gm.reduce && S.A.M >= 4) stage_wide(S, d, bt.seg0, bt.seg1, bt.grp);
        else if (d.i[MKS_I_PIECES] == 1 && gm.reduce && d.i[MKS_I_PROLOGUE] != MKS_P_NORM) stage_routed(S, d, bt.seg0, bt.seg1, gm.S);
        else if (d.i[MKS_I_PIECES] == 1 && !gm.reduce) stage_x<true>(S, d, bt.seg0, bt.seg1, bt.grp, gm.S);
        else stage_x<false>(S, d, bt.seg0, bt.seg1, bt.grp, gm.S);
        __syncwarp();
        consumer_sync();
        if (b == 0) prof_mark(S, 1);
        const bool good = multiply<FMT>(S, d, gm, bt, b, ar_seq, tag, n_stage);
        ok = ok && good;
    }
    if (gm.P > 1 && gm.nb > 0) {
        // every partial tile of this CTA is on its way; now the sums it is responsible for: each P-th tile of its range
        const int step = gm.panel >= 0 ? gm.P : 1;
        const int first = gm.panel >= 0 ? gm.t0 + ((gm.panel - gm.t0) % gm.P + gm.P) % gm.P : gm.t0;
#pragma unroll 1
        for (int tl = first + warp_() * step; tl < gm.t1 && ok; tl += NCW * step) {
            float sum[4];
            unsigned long long* words = tile_words(reinterpret_cast<unsigned long long*>(d.p[MKS_P_PART]), tl * gm.P);
            ok = collect_tile(S, words, tag, gm.P, sum);
            if (ok && S.A.clear_tiles) clear_tile(S, words, gm.P);
            ok = ok && finish_tile(S, d, ar_seq, tl, make_float4(sum[0], sum[1], sum[2], sum[3]));
        }
    }
    __syncwarp();
    prof_mark(S, 2);
    if (logits) {
        // best key of every sequence over this CTA's rows -> keys[m][cta]
        __syncwarp();
        consumer_sync();
        u64* keys = reinterpret_cast<u64*>(d.p[MKS_P_KEYS]);
        if (tid_() < S.A.M) __stcg(reinterpret_cast<unsigned long long*>(keys + (size_t)tid_() * grid_() + cta_()), (unsigned long long)S.keys_s[tid_()]);
    }
}

}  // namespace mks
