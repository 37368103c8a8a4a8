// Prompts through a stage program, all positions at once (declarations: include/mk_stage.h).
//
// `mk_stage_prefill` walks the same program the decode kernel runs, but executes every stage for M x L token rows with
// the kernels of mk_prefill.cuh.  The program's per-step activation buffers ([M][width]) become arrays of M x L rows in
// the caller's workspace; weights, states and caches are used where they are.  Everything the LM head needs is left to
// one ordinary decode step with the prompt's last token, so the caller sees exactly what stepping through would leave.
#include <utility>
#include <vector>

#include "mk_prefill_host.h"

using namespace mkp;

namespace {

// What this path does not do exactly as the decode kernel does is refused as a whole, and the caller steps through the prompt.
// A record is taken only if all it reads is what earlier records of the program have written in the same form: here the
// per-step buffers are arrays of their own, with nothing in them that was there before, and products' inputs are kept as bf16
// slabs.  The check follows the records through the buffers without touching the device.
struct Flow {
    struct Rows { uint64_t base; int width; uint64_t ssq; std::vector<std::pair<int, int>> cols; };   // fp32 [M][width]; written columns; sums of squares of all of it
    struct Made { uint64_t key; int stride, width; };                                                 // slabs
    int M;
    std::vector<Rows> rows;
    std::vector<Made> slabs;

    Rows* find(uint64_t p) {
        for (auto& r : rows)
            if (p >= r.base && p < r.base + (uint64_t)r.width * 4) return &r;
        return nullptr;
    }
    bool reads(uint64_t p, int stride, int off, int n) {
        Rows* r = find(p);
        if (!r || r->width != stride || (p - r->base) % 16) return false;
        int at = (int)((p - r->base) / 4) + off;
        const int end = at + n;
        if (at < 0 || end > r->width) return false;
        for (bool more = true; more && at < end;) {
            more = false;
            for (auto& c : r->cols)
                if (c.first <= at && c.second > at) {
                    at = c.second;
                    more = true;
                }
        }
        return at >= end;
    }
    static bool apart(uint64_t a, uint64_t a_bytes, uint64_t b, uint64_t b_bytes) { return a + a_bytes <= b || b + b_bytes <= a; }
    bool writes(uint64_t p, int stride, int n, uint64_t ssq) {
        if (n > stride || stride % 4) return false;
        const uint64_t bytes = ((uint64_t)(M - 1) * stride + n) * 4;
        for (auto& m : slabs)
            if (!apart(p, bytes, m.key, (uint64_t)M * m.stride * 4)) return false;
        Rows* r = find(p);
        if (r) {
            const int at = (int)((p - r->base) / 4);
            if (r->width != stride || (p - r->base) % 16 || at + n > stride) return false;
            r->cols.push_back({at, at + n});
            r->ssq = at == 0 && n == stride ? ssq : 0;
            return true;
        }
        for (auto& o : rows)
            if (!apart(p, bytes, o.base, (uint64_t)M * o.width * 4)) return false;
        rows.push_back({p, stride, n == stride ? ssq : 0, {{0, n}}});
        return true;
    }
    bool makes(uint64_t key, int stride, int width) {
        if (width > stride || width % 64) return false;
        const uint64_t bytes = (uint64_t)M * stride * 4;
        for (auto& r : rows)
            if (!apart(key, bytes, r.base, (uint64_t)M * r.width * 4)) return false;
        for (auto& m : slabs) {
            if (m.key == key && m.stride == stride) {
                m.width = width;
                return true;
            }
            if (!apart(key, bytes, m.key, (uint64_t)M * m.stride * 4)) return false;
        }
        slabs.push_back({key, stride, width});
        return true;
    }
    // all columns of a vector, and the sums of squares its norm is computed from
    bool normed(uint64_t p, int n, uint64_t ssq) {
        Rows* r = find(p);
        return r && r->base == p && r->width == n && ssq && r->ssq == ssq;
    }
    // a product's input
    bool operand(const mk_stage_desc& d, int K) {
        for (auto& m : slabs)
            if (m.key == d.p[MKS_P_X]) return d.i[MKS_I_PROLOGUE] == MKS_P_PLAIN && m.stride == d.i[MKS_I_X_STRIDE] && m.width == K;
        if (!reads(d.p[MKS_P_X], d.i[MKS_I_X_STRIDE], 0, K)) return false;
        return d.i[MKS_I_PROLOGUE] == MKS_P_PLAIN || (d.i[MKS_I_PROLOGUE] == MKS_P_NORM && normed(d.p[MKS_P_X], K, d.p[MKS_P_X_SSQ]));
    }
};

const char* refuse(const mk_stage_desc* prog, int n_stages, int M) {
    Flow F;
    F.M = M;
    const mk_stage_desc& e = prog[0];
    const int H = e.i[MKS_I_HIDDEN];
    if (H < 16 || H % 16 || !F.writes(e.p[MKS_P_H], H, H, e.p[MKS_P_H_SSQ])) return "the embedding's width";
    const mk_stage_desc *route = nullptr, *up = nullptr;       // the last routing, and the routed gate and up products behind it
    for (int s = 1; s < n_stages; s++) {
        const mk_stage_desc& d = prog[s];
        if (d.op == MKS_OP_GEMV) {
            const int kc = d.i[MKS_I_KC], K = kc * d.i[MKS_I_SPLITS], n = d.i[MKS_I_N_VALID], epi = d.i[MKS_I_EPILOGUE];
            const bool routed = d.i[MKS_I_GROUPS] < 0, glu = epi == MKS_E_GLU;
            if (d.i[MKS_I_PIECES] != 1) return "two-piece inputs";
            if (d.i[MKS_I_ALLREDUCE]) return "tensor parallelism";
            if (d.i[MKS_I_FMT] == MKS_FMT_INT8) return "int8 weights";
            if (kc % 64) return "columns per split are not whole 64-column blocks";
            if (d.i[MKS_I_GROUPS] != 1 && d.i[MKS_I_GROUPS] != -1) return "fixed groups";
            if (d.i[MKS_I_PROLOGUE] == MKS_P_NORM && d.i[MKS_I_K_TOTAL] != K) return "a norm over more than the stage's columns";
            if (epi == MKS_E_LOGITS) {
                // the head runs behind the prompt, on the last position's residual alone
                if (s != n_stages - 1 || routed || d.p[MKS_P_X] != e.p[MKS_P_H] || d.i[MKS_I_X_STRIDE] != H || K != H ||
                    (d.i[MKS_I_PROLOGUE] == MKS_P_NORM && d.p[MKS_P_X_SSQ] != e.p[MKS_P_H_SSQ])) return "an LM head that does not end the program on its residual";
                continue;
            }
            if (n < 1 || n > d.i[MKS_I_TILES] * (glu ? 8 : 16)) return "more output columns than tiles";
            if (!routed) {
                if (d.i[MKS_I_REDUCE_GROUPS]) return "one group to add up";
                if (!F.operand(d, K)) return "an input that no earlier stage leaves in this form";
                if (glu) {
                    if (!F.makes(d.p[MKS_P_OUT], d.i[MKS_I_OUT_STRIDE], n)) return "activations that overlap another buffer or are not whole 64-column blocks";
                    continue;
                }
            } else {
                if (!route) return "routed products without a routing";
                if (d.i[MKS_I_SPLITS] != 1) return "split experts";
                if (d.p[MKS_P_W_SHARED] && route->i[MKS_I_ROUTE_KIND] != 0) return "a shared expert without a gate";
                if (glu) {
                    if (d.i[MKS_I_REDUCE_GROUPS] || d.i[MKS_I_X_GSTRIDE] || n % 64 || !F.operand(d, K)) return "routed gate and up products of another form";
                    up = &d;
                    continue;
                }
                if (!up || !d.i[MKS_I_REDUCE_GROUPS] || d.i[MKS_I_PROLOGUE] != MKS_P_PLAIN || d.p[MKS_P_X] != up->p[MKS_P_OUT] || K != up->i[MKS_I_N_VALID] ||
                    d.i[MKS_I_X_STRIDE] != up->i[MKS_I_OUT_STRIDE] || d.i[MKS_I_X_GSTRIDE] != up->i[MKS_I_OUT_GSTRIDE] ||
                    !d.p[MKS_P_W_SHARED] != !up->p[MKS_P_W_SHARED]) return "routed products that do not follow their gate and up products";
                if (n % 4) return "routed outputs that are not whole float4s";
            }
            if (epi == MKS_E_RESID && !F.reads(d.p[MKS_P_OUT], d.i[MKS_I_OUT_STRIDE], 0, n)) return "a sum onto something no earlier stage writes";
            if (!F.writes(d.p[MKS_P_OUT], d.i[MKS_I_OUT_STRIDE], n, d.p[MKS_P_OUT_SSQ])) return "an output that overlaps another buffer";
        } else if (d.op == MKS_OP_GDN) {
            const int key = d.i[MKS_I_NKH] * 128, val = d.i[MKS_I_NVH] * 128, stride = d.i[MKS_I_Y_STRIDE];
            const uint64_t y = d.p[MKS_P_Y];
            if (d.i[MKS_I_CONV_DIM] != 2 * key + val || (d.i[MKS_I_Q_OFF] | d.i[MKS_I_K_OFF] | d.i[MKS_I_V_OFF]) % 4) return "DeltaNet channels";
            if (!F.reads(y, stride, d.i[MKS_I_Q_OFF], key) || !F.reads(y, stride, d.i[MKS_I_K_OFF], key) || !F.reads(y, stride, d.i[MKS_I_V_OFF], val) ||
                !F.reads(y, stride, d.i[MKS_I_Z_OFF], val) || !F.reads(y, stride, d.i[MKS_I_B_OFF], d.i[MKS_I_NVH]) || !F.reads(y, stride, d.i[MKS_I_A_OFF], d.i[MKS_I_NVH]))
                return "DeltaNet inputs that no earlier stage writes";
            if (!F.makes(d.p[MKS_P_Y2], d.i[MKS_I_Y2_STRIDE], val)) return "DeltaNet outputs that overlap another buffer";
        } else if (d.op == MKS_OP_ATTN) {
            const int nq = d.i[MKS_I_NQ], nkv = d.i[MKS_I_NKV], HD = d.i[MKS_I_HD], rot = d.i[MKS_I_ROT], stride = d.i[MKS_I_A_Y_STRIDE];
            const uint64_t y = d.p[MKS_P_A_Y];
            if (d.i[MKS_I_KV_F32] || !d.i[MKS_I_Q_BF16]) return "fp32 attention";
            if (nq % nkv) return "query heads per KV head";
            if (rot < 64 || rot > HD || rot % 64 || d.i[MKS_I_ROPE_PAIRS] > rot / 2) return "rotated dims that are not whole 64-dim blocks";
            bool ok = F.reads(y, stride, d.i[MKS_I_A_K_OFF], nkv * HD) && (d.i[MKS_I_A_V_OFF] < 0 || F.reads(y, stride, d.i[MKS_I_A_V_OFF], nkv * HD));
            for (int h = 0; h < nq; h++) {
                const int q = d.i[MKS_I_A_Q_OFF] + h * d.i[MKS_I_A_Q_HSTRIDE];
                ok = ok && F.reads(y, stride, q, HD) && (d.i[MKS_I_A_GATE_OFF] < 0 || F.reads(y, stride, q + d.i[MKS_I_A_GATE_OFF], HD));
            }
            if (!ok) return "attention inputs that no earlier stage writes";
            if (!F.makes(d.p[MKS_P_A_Y2], d.i[MKS_I_A_Y2_STRIDE], nq * HD)) return "attention outputs that overlap another buffer";
        } else if (d.op == MKS_OP_ROUTE) {
            if (!F.reads(d.p[MKS_P_LOGITS], d.i[MKS_I_LOGIT_STRIDE], 0, d.i[MKS_I_EXPERTS] + (d.i[MKS_I_ROUTE_KIND] == 0))) return "router logits that no earlier stage writes";
            route = &d;
            up = nullptr;
        } else if (d.op == MKS_OP_VEC) {
            const int N = d.i[MKS_I_VEC_N];
            if (N == 0) continue;
            if (!F.normed(d.p[MKS_P_VEC_A], N, d.p[MKS_P_VEC_A_SSQ]) || (d.p[MKS_P_VEC_B] && !F.normed(d.p[MKS_P_VEC_B], N, d.p[MKS_P_VEC_B_SSQ])))
                return "a vector step's term without its sums of squares";
            if (d.p[MKS_P_VEC_BASE] && (!F.reads(d.p[MKS_P_VEC_BASE], N, 0, N))) return "a vector step's base that no earlier stage writes";
            if (!F.writes(d.p[MKS_P_VEC_OUT], N, N, d.p[MKS_P_VEC_OUT_SSQ]) || F.find(d.p[MKS_P_VEC_OUT])->base != d.p[MKS_P_VEC_OUT]) return "a vector step's output";
        } else {
            return "an embedding inside the program";
        }
    }
    return nullptr;
}

struct Buffer { uint64_t base; int width; float* rows; };
struct Have { uint64_t key; const void* norm; float in_scale, eps, off; int K; };      // what x_scratch holds
struct Slab { uint64_t key; const void* norm; float in_scale; uint8_t* x; int rows, width; };

struct Exec {
    const mk_stage_desc* prog;
    int n_stages, M, L, rows, xrows = 0, sms;
    struct Tiling { int n, nt, ksplit; } tile[2];          // of the token rows: at most 256 and at most 384 a tile
    const int* tokens;
    int* pos;
    int* status;
    long long spin;
    cudaStream_t st;
    bool h_last = false;
    Arena arena;
    std::vector<Buffer> bufs;
    std::vector<Slab> slabs;
    uint8_t* x_scratch = nullptr;        // slabs made from fp32 rows; reused by every stage that needs new ones
    Have x_have = {};
    struct { uint64_t key; int ksplit; } left = {};       // a residual whose last addend waits as partial products in `part`
    float* part = nullptr;
    size_t part_floats = 0;
    // DeltaNet / attention / routing scratch
    float *qkv = nullptr, *o = nullptr, *gram = nullptr;
    float4* scal = nullptr;
    __nv_bfloat16* q = nullptr;
    RouteArgs route;
    uint8_t* xg = nullptr;               // gathered slabs
    int slot_rows = 0, max_items = 0;
    bool few = false;                                     // the routed products are those of experts_gemm
    float *yg = nullptr, *ys = nullptr;
    uint8_t *act_g = nullptr, *act_s = nullptr;

    Buffer* find(uint64_t p) {
        for (auto& b : bufs)
            if (p >= b.base && p < b.base + (uint64_t)b.width * 4) return &b;
        return nullptr;
    }
    // the row array behind a per-step buffer, at the same column offset
    float* at(uint64_t p) {
        Buffer* b = find(p);
        return b ? b->rows + (p - b->base) / 4 : nullptr;
    }
    void add(uint64_t p, int width) {
        if (p && !find(p)) bufs.push_back({p, width, nullptr});
    }
    Slab* slab(uint64_t key) {
        for (auto& s : slabs)
            if (s.key == key) return &s;
        return nullptr;
    }
    void need_slab(uint64_t key, int width) {
        Slab* s = slab(key);
        if (!s) slabs.push_back({key, nullptr, 0.f, nullptr, xrows, width});
        else if (width > s->width) s->width = width;
    }
    void written(uint64_t p) {           // fp32 rows change: slabs made from them are stale
        if (find(x_have.key) == find(p)) x_have.key = 0;
    }

    static int format(const mk_stage_desc& d) {
        switch (d.i[MKS_I_FMT]) {
            case MKS_FMT_MXFP4: return W_MXFP4;
            case MKS_FMT_FP8: return d.i[MKS_I_BLOCK_SCALES] == 2 ? W_FP8_PIECES2 : (d.i[MKS_I_BLOCK_SCALES] ? W_FP8_PIECES3 : W_FP8);
            case MKS_FMT_BF16: return W_BF16;
            default: return -1;
        }
    }

    // How a dense product is cut.  A CTA converts its weights once for all tokens of its tile, which takes sixteen warps about 860
    // cycles per 64 columns; up to 256 tokens hide behind that (MXFP4, 192 tokens: the tensor cores are busy 43 % of the time).  Wider
    // tiles convert less often, and what then counts is shared memory: about 10 / 3 cycles per token (384 tokens: 1270).
    static constexpr int CONVERT = 860;
    Tiling tiling(const mk_stage_desc& d) const {
        const int blocks = (d.i[MKS_I_TILES] + 7) / 8, kbs = d.i[MKS_I_KC] * d.i[MKS_I_SPLITS] / 64, fmt = format(d);
        Tiling best = tile[0];
        double cost = 0.;
        for (int i = 0; i < (fmt == W_FP8_PIECES2 || fmt == W_FP8_PIECES3 ? 1 : 2); i++) {
            Tiling t = tile[i];
            t.ksplit = pick_ksplit(blocks * t.n, kbs, sms);
            const int per = (kbs + t.ksplit - 1) / t.ksplit + 6;
            const double c = (double)((blocks * t.n * t.ksplit + sms - 1) / sms) * per * (10 * t.nt > 3 * CONVERT ? 10. * t.nt / 3 : (double)CONVERT);
            if (!i || c < cost) {
                best = t;
                cost = c;
            }
        }
        return best;
    }

    void layout() {
        for (int s = 0; s < n_stages; s++) {
            const mk_stage_desc& d = prog[s];
            if (d.op == MKS_OP_EMBED) add(d.p[MKS_P_H], d.i[MKS_I_HIDDEN]);
            else if (d.op == MKS_OP_GEMV && d.i[MKS_I_EPILOGUE] != MKS_E_LOGITS && d.i[MKS_I_EPILOGUE] != MKS_E_GLU) add(d.p[MKS_P_OUT], d.i[MKS_I_OUT_STRIDE]);
            else if (d.op == MKS_OP_VEC && d.i[MKS_I_VEC_N]) add(d.p[MKS_P_VEC_OUT], d.i[MKS_I_VEC_N]);
        }
        for (auto& b : bufs) b.rows = arena.take<float>((size_t)rows * b.width);
        int kmax = 0, experts = 0, topk = 0;
        bool fp8 = true, scaled = false;      // the experts' weights
        size_t conv = 0, heads = 0, vals = 0, q_w = 0, ex_k = 0, ex_n = 0, ex_f = 0, sh = 0;
        for (int s = 0; s < n_stages; s++) {
            const mk_stage_desc& d = prog[s];
            auto up = [](size_t& a, size_t b) { if (b > a) a = b; };
            if (d.op == MKS_OP_GEMV && d.i[MKS_I_EPILOGUE] != MKS_E_LOGITS) {
                const int K = d.i[MKS_I_KC] * d.i[MKS_I_SPLITS];
                const bool routed = d.i[MKS_I_GROUPS] < 0;
                if (routed) {
                    fp8 &= d.i[MKS_I_FMT] == MKS_FMT_FP8;
                    scaled |= d.i[MKS_I_BLOCK_SCALES] != 0;
                }
                if (d.i[MKS_I_EPILOGUE] == MKS_E_GLU) {
                    if (routed) {
                        up(ex_k, K);
                        up(ex_f, d.i[MKS_I_N_VALID]);
                        sh |= d.p[MKS_P_W_SHARED] != 0;
                    } else need_slab(d.p[MKS_P_OUT], d.i[MKS_I_N_VALID]);
                }
                if (routed && d.i[MKS_I_EPILOGUE] != MKS_E_GLU) up(ex_n, d.i[MKS_I_N_VALID]);
                if (K > kmax) kmax = K;
                if (!routed) {
                    const int z = tiling(d).ksplit;
                    if (z > 1) up(part_floats, (size_t)z * rows * (d.i[MKS_I_EPILOGUE] == MKS_E_GLU ? d.i[MKS_I_TILES] * 16 : d.i[MKS_I_N_VALID]));
                }
            } else if (d.op == MKS_OP_GDN) {
                up(conv, d.i[MKS_I_CONV_DIM]);
                up(heads, d.i[MKS_I_NVH]);
                need_slab(d.p[MKS_P_Y2], d.i[MKS_I_NVH] * 128);
            } else if (d.op == MKS_OP_ATTN) {
                up(q_w, (size_t)d.i[MKS_I_NQ] * d.i[MKS_I_HD]);
                need_slab(d.p[MKS_P_A_Y2], d.i[MKS_I_NQ] * d.i[MKS_I_HD]);
            } else if (d.op == MKS_OP_ROUTE) {
                experts = d.i[MKS_I_EXPERTS];
                topk = d.i[MKS_I_TOPK];
            }
        }
        for (auto& s : slabs) s.x = arena.take<uint8_t>((size_t)(s.width + 63) / 64 * xrows * 128);
        vals = heads * 128;
        x_scratch = arena.take<uint8_t>((size_t)kmax / 64 * xrows * 128);
        if (part_floats) part = arena.take<float>(part_floats);
        if (conv) {
            qkv = arena.take<float>((size_t)rows * conv);
            scal = arena.take<float4>((size_t)rows * heads);
            o = arena.take<float>((size_t)rows * vals);
            gram = arena.take<float>((size_t)M * ((L + SCAN - 1) / SCAN) * heads * GRAM);
        }
        if (q_w) q = arena.take<__nv_bfloat16>((size_t)rows * q_w);
        if (experts) {
            // tile width of the routed products: about twice the mean load, so that most experts are one tile
            // (by estimate: narrower tiles leave fewer columns of padding, wider ones convert an expert's weights fewer times)
            const int mean = (int)((long long)rows * topk / experts);
            memset(&route, 0, sizeof route);
            // Few rows per expert go straight from the packed tiles.  Passes through the operand against these, ms, at a mean load of
            // block scales (256 experts): 40 9.37 / 7.62, 64 11.77 / 11.00, 78 13.71 / 13.21, 93 15.38 / 15.14; beyond, the operand's
            // tiles are 256 tokens wide.  Row scales (128 experts): 20 3.52 / 3.42, 24 3.57 / 3.58, 32 3.79 / 4.07.
            few = fp8 && mean <= (scaled ? 96 : 20);
            if (few) route.nt = 32;
            else route.nt = mean > 96 ? 256 : (mean > 40 ? 128 : (mean > 16 ? 64 : 32));
            slot_rows = (rows * topk + experts * 15 + route.nt + 15) / 16 * 16;
            max_items = experts + rows * topk / route.nt + 1;
            if (max_items > rows * topk) max_items = rows * topk;
            route.items = arena.take<int4>(max_items);
            route.counts = arena.take<int>(3 * experts + 1);
            route.n_items = route.counts ? route.counts + 3 * experts : nullptr;
            route.slot = arena.take<int>((size_t)rows * 8);
            route.weight = arena.take<float>((size_t)rows * 8);
            route.gate = arena.take<float>(rows);
            xg = arena.take<uint8_t>(ex_k / 64 * slot_rows * 128);
            act_g = arena.take<uint8_t>((ex_f + 63) / 64 * slot_rows * 128);
            yg = arena.take<float>((size_t)slot_rows * ex_n);
            if (sh) {
                act_s = arena.take<uint8_t>((ex_f + 63) / 64 * xrows * 128);
                ys = arena.take<float>((size_t)rows * ex_n);
            }
        }
    }

    int gemm(const mk_stage_desc& d, GemmArgs& A, int out, int items) {
        const int blocks = (d.i[MKS_I_TILES] + 7) / 8, ntiles = (A.rows + A.nt - 1) / A.nt;
        const int fmt = format(d);
        if ((fmt == W_FP8_PIECES2 || fmt == W_FP8_PIECES3) && A.ksplit == 1 && A.nt * (A.kbs / 2) <= 512 && A.kbs % 2 == 0)
            return launch_gemm<W_FP8_BLOCK, 1>(A, out, blocks, ntiles, items, st);
        switch (fmt) {
            case W_MXFP4: return launch_gemm<W_MXFP4, 1>(A, out, blocks, ntiles, items, st);
            case W_FP8: return launch_gemm<W_FP8, 1>(A, out, blocks, ntiles, items, st);
            case W_FP8_PIECES2: return launch_gemm<W_FP8_PIECES2, 1>(A, out, blocks, ntiles, items, st);
            case W_FP8_PIECES3: return launch_gemm<W_FP8_PIECES3, 1>(A, out, blocks, ntiles, items, st);
            default: return launch_gemm<W_BF16, 1>(A, out, blocks, ntiles, items, st);
        }
    }
    GemmArgs args(const mk_stage_desc& d) {
        GemmArgs A;
        memset(&A, 0, sizeof A);
        A.w = reinterpret_cast<const uint8_t*>(d.p[MKS_P_W]);
        A.tiles = d.i[MKS_I_TILES];
        A.unit_steps = d.i[MKS_I_UNIT_STEPS];
        A.chunk_steps = d.i[MKS_I_CHUNK_STEPS];
        A.chunk_bytes = d.i[MKS_I_CHUNK_BYTES];
        A.kc = d.i[MKS_I_KC];
        A.row_scale = reinterpret_cast<const float*>(d.p[MKS_P_ROW_SCALE]);
        A.kbs = d.i[MKS_I_KC] * d.i[MKS_I_SPLITS] / 64;
        A.ksplit = 1;
        A.rows = rows;
        A.nt = tile[0].nt;
        A.gelu = d.i[MKS_I_ACT] == MKS_ACT_GELU_TANH;
        A.n_valid = d.i[MKS_I_EPILOGUE] == MKS_E_GLU ? d.i[MKS_I_TILES] * 16 : d.i[MKS_I_N_VALID];
        A.act_cols = d.i[MKS_I_N_VALID];
        A.status = status;
        A.spin_limit_ns = spin;
        return A;
    }

    // The token operand of a stage: what its producer left as slabs, or its fp32 rows brought into that form.
    int operand(const mk_stage_desc& d, const uint8_t** x, int* x_rows) {
        if (Slab* s = slab(d.p[MKS_P_X])) {
            *x = s->x;
            *x_rows = s->rows;
            return MK_OK;
        }
        const bool norm = d.i[MKS_I_PROLOGUE] == MKS_P_NORM;
        const void* nw = norm ? reinterpret_cast<const void*>(d.p[MKS_P_NORM_W]) : nullptr;
        const float in_scale = d.f[MKS_F_IN_SCALE] != 0.f ? d.f[MKS_F_IN_SCALE] : 1.f;
        const Have want = {d.p[MKS_P_X], nw, in_scale, d.f[MKS_F_EPS], d.f[MKS_F_NORM_OFF], d.i[MKS_I_KC] * d.i[MKS_I_SPLITS]};
        const bool same = x_have.key == want.key && x_have.norm == nw && x_have.K == want.K && (!norm || (x_have.in_scale == in_scale && x_have.eps == want.eps && x_have.off == want.off));
        if (!same) {
            const int splits = left.key == want.key ? left.ksplit : 0;
            const RowsIn R = {at(d.p[MKS_P_X]), d.i[MKS_I_X_STRIDE], want.K, splits, rows, part, reinterpret_cast<const float*>(nw), d.f[MKS_F_NORM_OFF], d.f[MKS_F_EPS], in_scale, x_scratch, 0, xrows};
            MKP_CUDA(launch(splits ? rows_in<1, true> : rows_in<1, false>, dim3(rows), 256, 0, st, R));
            left = {};
            x_have = want;
        }
        *x = x_scratch;
        *x_rows = xrows;
        return MK_OK;
    }

    int dense(const mk_stage_desc& d) {
        GemmArgs A = args(d);
        int rc = operand(d, &A.x, &A.x_rows);
        if (rc != MK_OK) return rc;
        const Tiling t = tiling(d);
        A.nt = t.nt;
        A.ksplit = t.ksplit;
        A.part = part;
        A.part_rows = rows;
        int out;
        if (d.i[MKS_I_EPILOGUE] == MKS_E_GLU) {
            out = OUT_GLU;
            Slab* s = slab(d.p[MKS_P_OUT]);
            A.act = s->x;
            A.act_rows = s->rows;
        } else {
            out = d.i[MKS_I_EPILOGUE] == MKS_E_RESID ? OUT_ADD : OUT_STORE;
            A.out = at(d.p[MKS_P_OUT]);
            A.out_stride = d.i[MKS_I_OUT_STRIDE];
            written(d.p[MKS_P_OUT]);
            // the next record norms this residual: it adds the K splits' partials on the way
            const mk_stage_desc* n = &d + 1;
            A.leave = out == OUT_ADD && A.ksplit > 1 && n < prog + n_stages && n->op == MKS_OP_GEMV && n->i[MKS_I_EPILOGUE] != MKS_E_LOGITS && n->i[MKS_I_PROLOGUE] == MKS_P_NORM &&
                      n->p[MKS_P_X] == d.p[MKS_P_OUT] && n->i[MKS_I_KC] * n->i[MKS_I_SPLITS] == A.n_valid && n->i[MKS_I_X_STRIDE] == A.out_stride &&
                      (n->i[MKS_I_GROUPS] == 1 || n->i[MKS_I_EPILOGUE] == MKS_E_GLU);
            if (A.leave) left = {d.p[MKS_P_OUT], A.ksplit};
        }
        return gemm(d, A, out, 0);
    }

    int routed(const mk_stage_desc& d) {
        const bool shared = d.p[MKS_P_W_SHARED] != 0, up = d.i[MKS_I_EPILOGUE] == MKS_E_GLU;
        GemmArgs A = args(d);
        int rc;
        if (up) {
            rc = operand(d, &A.x, &A.x_rows);
            if (rc != MK_OK) return rc;
            if (shared) {                // the shared expert: a dense product on the rows as they are
                GemmArgs S = A;
                S.w = reinterpret_cast<const uint8_t*>(d.p[MKS_P_W_SHARED]);
                S.row_scale = reinterpret_cast<const float*>(d.p[MKS_P_RS_SHARED]);
                S.act = act_s;
                S.act_rows = xrows;
                rc = gemm(d, S, OUT_GLU, 0);
                if (rc != MK_OK) return rc;
            }
            auto gather = few ? gather_rows<true> : gather_rows<false>;
            MKP_CUDA(launch(gather, dim3(rows), 256, 0, st, A.x, A.x_rows, route.slot, route.topk, A.kbs, xg, slot_rows));
            MKP_CUDA(cudaGetLastError());
            A.x = xg;
            A.act = act_g;
            A.act_rows = slot_rows;
        } else {
            if (shared) {
                GemmArgs S = A;
                S.w = reinterpret_cast<const uint8_t*>(d.p[MKS_P_W_SHARED]);
                S.row_scale = reinterpret_cast<const float*>(d.p[MKS_P_RS_SHARED]);
                S.x = act_s;
                S.x_rows = xrows;
                S.out = ys;
                S.out_stride = d.i[MKS_I_N_VALID];
                rc = gemm(d, S, OUT_STORE, 0);
                if (rc != MK_OK) return rc;
            }
            A.x = act_g;
            A.out = yg;
            A.out_stride = d.i[MKS_I_N_VALID];
        }
        A.x_rows = slot_rows;
        A.w_gstride = d.p[MKS_P_W_GSTRIDE];
        A.rs_gstride = d.p[MKS_P_RS_GSTRIDE];
        A.nt = route.nt;
        A.items = route.items;
        A.n_items = route.n_items;
        const int out = up ? OUT_GLU : OUT_STORE;
        A.blocks = (d.i[MKS_I_TILES] + 7) / 8;
        if (!few) rc = gemm(d, A, out, max_items);
        else rc = d.i[MKS_I_BLOCK_SCALES] ? launch_experts<true, 4>(A, out, max_items, sms, st) : launch_experts<false, 4>(A, out, max_items, sms, st);
        if (rc != MK_OK || up) return rc;
        MKP_CUDA(launch(combine_rows, dim3(rows), 256, 0, st, yg, d.i[MKS_I_N_VALID], route.slot, route.weight, route.topk, shared ? ys : nullptr, route.gate,
                                           d.i[MKS_I_EPILOGUE] == MKS_E_RESID, at(d.p[MKS_P_OUT]), d.i[MKS_I_OUT_STRIDE]));
        MKP_CUDA(cudaGetLastError());
        written(d.p[MKS_P_OUT]);
        return MK_OK;
    }

    int gdn(const mk_stage_desc& d) {
        GdnArgs G;
        memset(&G, 0, sizeof G);
        G.y = at(d.p[MKS_P_Y]);
        G.y_stride = d.i[MKS_I_Y_STRIDE];
        G.M = M; G.L = L;
        G.nkh = d.i[MKS_I_NKH]; G.nvh = d.i[MKS_I_NVH]; G.conv_dim = d.i[MKS_I_CONV_DIM];
        G.q_off = d.i[MKS_I_Q_OFF]; G.k_off = d.i[MKS_I_K_OFF]; G.v_off = d.i[MKS_I_V_OFF]; G.z_off = d.i[MKS_I_Z_OFF];
        G.b_off = d.i[MKS_I_B_OFF]; G.a_off = d.i[MKS_I_A_OFF];
        G.conv_w = reinterpret_cast<const float*>(d.p[MKS_P_CONV_W]);
        G.A_log = reinterpret_cast<const float*>(d.p[MKS_P_A_LOG]);
        G.dt_bias = reinterpret_cast<const float*>(d.p[MKS_P_DT_BIAS]);
        G.norm_w = reinterpret_cast<const float*>(d.p[MKS_P_GDN_NORM]);
        G.conv_state = reinterpret_cast<float*>(d.p[MKS_P_CONV_STATE]);
        G.ring = 4;
        G.ssm = reinterpret_cast<float*>(d.p[MKS_P_SSM_STATE]);
        G.pos = pos;
        G.conv_bf16 = d.i[MKS_I_CONV_BF16];
        G.l2_clamp = d.i[MKS_I_L2_CLAMP];
        G.eps = G.norm_eps = d.f[MKS_F_EPS];
        G.qkv = qkv; G.scal = scal; G.o = o;
        Slab* s = slab(d.p[MKS_P_Y2]);
        G.out = s->x;
        G.out_rows = s->rows;
        G.gram = gram;
        return launch_gdn(G, gdn_gate<1>, sms, st);
    }

    template <int HD>
    int attn_hd(const AttnArgs& T) {
        const int bq = AT_ROWS / (T.nq / T.nkv);
        MKP_CUDA(launch((attn_prepare<HD, false, false>), dim3((T.nq + 2 * T.nkv + 7) / 8, rows), 256, 0, st, T));
        MKP_CUDA(cudaFuncSetAttribute(attn_rows<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_smem<HD>()));
        MKP_CUDA(launch(attn_rows<HD>, dim3((L + bq - 1) / bq, T.nkv, M), 256, attn_smem<HD>(), st, T));
        MKP_CUDA(cudaGetLastError());
        return MK_OK;
    }
    int attn(const mk_stage_desc& d) {
        AttnArgs T;
        memset(&T, 0, sizeof T);
        const int HD = d.i[MKS_I_HD];
        T.y = at(d.p[MKS_P_A_Y]);
        T.y_stride = d.i[MKS_I_A_Y_STRIDE];
        T.M = M; T.L = L; T.nq = d.i[MKS_I_NQ]; T.nkv = d.i[MKS_I_NKV];
        T.q_off = d.i[MKS_I_A_Q_OFF]; T.q_hs = d.i[MKS_I_A_Q_HSTRIDE]; T.gate_off = d.i[MKS_I_A_GATE_OFF];
        T.k_off = d.i[MKS_I_A_K_OFF]; T.v_off = d.i[MKS_I_A_V_OFF];
        T.rot = d.i[MKS_I_ROT]; T.pairs = d.i[MKS_I_ROPE_PAIRS]; T.window = d.i[MKS_I_WINDOW];
        T.norm_plain = d.i[MKS_I_NORM_PLAIN]; T.v_norm = d.i[MKS_I_V_NORM];
        T.eps = d.f[MKS_F_EPS]; T.scale = d.f[MKS_F_SCALE];
        T.q_norm = reinterpret_cast<const float*>(d.p[MKS_P_Q_NORM]);
        T.k_norm = reinterpret_cast<const float*>(d.p[MKS_P_K_NORM]);
        T.cos = reinterpret_cast<const float*>(d.p[MKS_P_ROPE_COS]);
        T.sin = reinterpret_cast<const float*>(d.p[MKS_P_ROPE_SIN]);
        T.k_cache = reinterpret_cast<void*>(d.p[MKS_P_K_CACHE]);
        T.v_cache = reinterpret_cast<void*>(d.p[MKS_P_V_CACHE]);
        T.bt = reinterpret_cast<const int*>(d.p[MKS_P_BLOCK_TABLE]);
        T.max_pages = d.i[MKS_I_MAX_PAGES];
        const int kvb = d.i[MKS_I_KV_BLOCK] > 0 ? d.i[MKS_I_KV_BLOCK] : 64;
        T.kv_shift = 31 - __builtin_clz(kvb);
        const bool own = d.i[MKS_I_KV_S_PAGE] == 0;
        T.s_page = own ? (uint32_t)(T.nkv * kvb * HD) : (uint32_t)d.i[MKS_I_KV_S_PAGE];
        T.s_head = own ? (uint32_t)(kvb * HD) : (uint32_t)d.i[MKS_I_KV_S_HEAD];
        T.s_pos = own ? (uint32_t)HD : (uint32_t)d.i[MKS_I_KV_S_POS];
        T.pos = pos;
        T.q = q;
        Slab* s = slab(d.p[MKS_P_A_Y2]);
        T.out = s->x;
        T.out_rows = s->rows;
        return HD == 512 ? attn_hd<512>(T) : attn_hd<256>(T);
    }

    int routing(const mk_stage_desc& d) {
        route.logits = at(d.p[MKS_P_LOGITS]);
        route.rows = rows;
        route.stride = d.i[MKS_I_LOGIT_STRIDE];
        route.experts = d.i[MKS_I_EXPERTS];
        route.topk = d.i[MKS_I_TOPK];
        route.kind = d.i[MKS_I_ROUTE_KIND];
        route.expert_scale = reinterpret_cast<const float*>(d.p[MKS_P_EXPERT_SCALE]);
        MKP_CUDA(cudaMemsetAsync(route.counts, 0, (3 * route.experts + 1) * sizeof(int), st));
        route.ids_out = h_last ? reinterpret_cast<int*>(d.p[MKS_P_ROUTE_OUT]) : nullptr;
        route.L = L;
        MKP_CUDA(launch(route_rows, dim3((rows + 7) / 8), 256, 0, st, route));
        MKP_CUDA(launch(route_plan, dim3(1), 256, 0, st, route));
        MKP_CUDA(launch(route_slots, dim3((rows * 8 + 255) / 256), 256, 0, st, route));
        MKP_CUDA(cudaGetLastError());
        return MK_OK;
    }

    int vec(const mk_stage_desc& d) {
        if (!d.i[MKS_I_VEC_N]) return MK_OK;
        MKP_CUDA(launch(vec_rows, dim3(rows), 256, 0, st, d.i[MKS_I_VEC_N], at(d.p[MKS_P_VEC_BASE]), at(d.p[MKS_P_VEC_A]), reinterpret_cast<const float*>(d.p[MKS_P_VEC_A_W]),
                                       at(d.p[MKS_P_VEC_B]), reinterpret_cast<const float*>(d.p[MKS_P_VEC_B_W]), d.f[MKS_F_NORM_OFF], d.f[MKS_F_EPS],
                                       d.f[MKS_F_SCALE] != 0.f ? d.f[MKS_F_SCALE] : 1.f, at(d.p[MKS_P_VEC_OUT])));
        MKP_CUDA(cudaGetLastError());
        written(d.p[MKS_P_VEC_OUT]);
        return MK_OK;
    }

    int run() {
        for (int s = 0; s < n_stages; s++) {
            const mk_stage_desc& d = prog[s];
            int rc = MK_OK;
            switch (d.op) {
                case MKS_OP_EMBED:
                    MKP_CUDA(launch(embed_rows, dim3(rows), 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(d.p[MKS_P_TABLE]), tokens, M, L, d.i[MKS_I_HIDDEN], d.i[MKS_I_VOCAB],
                                                     d.f[MKS_F_SCALE], at(d.p[MKS_P_H])));
                    MKP_CUDA(cudaGetLastError());
                    written(d.p[MKS_P_H]);
                    break;
                case MKS_OP_GEMV:
                    if (d.i[MKS_I_EPILOGUE] == MKS_E_LOGITS) break;            // the last token's step computes logits
                    rc = d.i[MKS_I_GROUPS] < 0 ? routed(d) : dense(d);
                    break;
                case MKS_OP_GDN: rc = gdn(d); break;
                case MKS_OP_ATTN: rc = attn(d); break;
                case MKS_OP_ROUTE: rc = routing(d); break;
                case MKS_OP_VEC: rc = vec(d); break;
                default: return pfail(MK_ERR_BADARG, "prefill: unknown op %d", d.op);
            }
            if (rc != MK_OK) return rc;
        }
        if (h_last) {
            const mk_stage_desc& d = prog[0];
            MKP_CUDA(launch(last_rows, dim3(M), 256, 0, st, at(d.p[MKS_P_H]), L, d.i[MKS_I_HIDDEN], reinterpret_cast<float*>(d.p[MKS_P_H]), reinterpret_cast<float*>(d.p[MKS_P_H_SSQ])));
        }
        MKP_CUDA(launch(advance_pos, dim3(1), 32, 0, st, pos, M, h_last ? L - 1 : L));
        MKP_CUDA(cudaGetLastError());
        return MK_OK;
    }
};

int prepare(Exec& E, const mk_stage_desc* prog, int n_stages, int batch, int positions, int device, void* workspace) {
    E.prog = prog;
    E.n_stages = n_stages;
    E.M = batch;
    E.L = positions;
    E.rows = batch * positions;
    token_tiles(E.rows, 256, &E.tile[0].n, &E.tile[0].nt);
    token_tiles(E.rows, 384, &E.tile[1].n, &E.tile[1].nt);
    for (auto& t : E.tile) E.xrows = E.xrows > t.n * t.nt ? E.xrows : t.n * t.nt;
    const int rc = mk_stage_validate(prog, n_stages, batch);
    if (rc != MK_OK) return rc;
    if (const char* why = refuse(prog, n_stages, batch)) return pfail(MK_ERR_UNSUPPORTED, "prefill: %s", why);
    if (cudaDeviceGetAttribute(&E.sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return pfail(MK_ERR_CUDA, "prefill: no device %d", device);
    E.arena.base = static_cast<uint8_t*>(workspace);
    E.layout();
    return MK_OK;
}

}  // namespace

extern "C" int64_t mk_stage_prefill_bytes(const mk_stage_desc* program, int n_stages, int batch, int positions, int device) {
    if (!program || n_stages < 1 || batch < 1 || batch > MKS_MAX_BATCH || positions < 1 || positions > MAX_ROWS / batch) return pfail(MK_ERR_BADARG, "mk_stage_prefill_bytes: bad argument");
    Exec E;
    const int rc = prepare(E, program, n_stages, batch, positions, device, nullptr);
    return rc == MK_OK ? (int64_t)E.arena.off + 1024 : rc;
}

extern "C" int mk_stage_prefill(const mk_stage_prefill_args* a, void* stream) {
    if (!a || !a->program || a->n_stages < 1) return pfail(MK_ERR_BADARG, "mk_stage_prefill: no program");
    if (a->batch < 1 || a->batch > MKS_MAX_BATCH || a->positions < 1 || a->positions > MAX_ROWS / a->batch)
        return pfail(MK_ERR_BADARG, "mk_stage_prefill: batch %d, positions %d (at most %d rows a call)", a->batch, a->positions, MAX_ROWS);
    if (!a->tokens || !a->pos || !a->status || !a->workspace) return pfail(MK_ERR_BADARG, "mk_stage_prefill: tokens / pos / status / workspace missing");
    MKP_CUDA(cudaSetDevice(a->device));
    Exec E;
    uint8_t* ws = reinterpret_cast<uint8_t*>((a->workspace + 1023) & ~(uint64_t)1023);
    const int rc = prepare(E, reinterpret_cast<const mk_stage_desc*>(a->program), a->n_stages, a->batch, a->positions, a->device, ws);
    if (rc != MK_OK) return rc;
    if ((int64_t)E.arena.off + 1024 > a->workspace_bytes) return pfail(MK_ERR_BADARG, "mk_stage_prefill: workspace of %lld bytes, %lld needed", (long long)a->workspace_bytes, (long long)E.arena.off + 1024);
    E.tokens = reinterpret_cast<const int*>(a->tokens);
    E.pos = reinterpret_cast<int*>(a->pos);
    E.status = reinterpret_cast<int*>(a->status);
    E.h_last = a->last != 0;
    E.spin = a->spin_limit_ns > 0 ? a->spin_limit_ns : 2000000000ll;
    E.st = static_cast<cudaStream_t>(stream);
    return E.run();
}
