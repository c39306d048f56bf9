// How a model is split over the thread-block clusters of decode_cluster.cu: host arithmetic only, no CUDA headers, so that it
// is tested without a GPU (tests/test_decode_plan_host.py).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace tb {

constexpr int DC_WARPS = 16;                              // compute warps
constexpr int DC_COMPUTE = DC_WARPS * 32;
constexpr int DC_THREADS = DC_COMPUTE + 64;               // + producer warp + tensor-core warp
constexpr int DC_SLOTS = 32;                              // chunks in flight (barrier pairs of the ring)
constexpr int DC_GROUP = 2;                               // attention: warps that share a chunk of cache rows
constexpr int DC_KV_ROWS = 64;                            // cache rows per chunk
constexpr int DC_KV_BYTES = 2 * DC_KV_ROWS * 128;         // keys + values of a chunk (128-byte rows, 128B swizzle)
constexpr int DC_STAGE_LD = 17;                           // floats per staged accumulator row (16 sequences + 1)
constexpr int DC_MAX_PAIRS = 8;                           // (sequence, head) pairs per CTA
constexpr int DC_TMEM_COLS = 256;
// accumulator columns: QKV (two tiles of 16), out-projection (64), gate|up (16), down-projection (64)
constexpr int DC_COL_Q = 0, DC_COL_O = 32, DC_COL_G = 96, DC_COL_D = 128;
constexpr int DC_OVERRUN = 16384;                         // a 128-row operand read of a shorter tile stays within this

// A projection as a CTA sees it: `tiles` operand tiles of `rows` weight rows (rows = slices * n for the sliced form);
// K in blocks of 64, kblocks of them per slice, `chunk` of them per copy.  umma_n: columns of one tensor-core instruction, which
// at M = 128 come in steps of 16 only -- three slices of one group of 8 sequences are 24, the instruction takes 32; what it
// reads behind the operand buffer is this CTA's own shared memory, and nobody reads the columns it makes of it.
struct DcProj { int n, rows, tiles, slices, kblocks, chunk, umma_n; uint32_t bytes; };

struct DcPlan {
    int S, D, H, F, R, P, C;                              // R sequences per cluster, P pairs per CTA, C CTAs per cluster
    int rg;                                               // groups of 8 sequences (1 or 2)
    uint32_t p_magic, h_magic, g8_magic;                  // ceil(2^16 / P), / H, / (g.n / 8): i / d = i * magic >> 16 for the few i here
    DcProj q, o, g, d;                                    // g.n = hidden units per CTA (rows = 2 n)
    uint32_t rank_bytes;
    int vec_floats;
    uint32_t ring_bytes;
    // shared-memory offsets
    uint32_t o_x, o_ax, o_att, o_ah, o_qkv, o_rot, o_stage, o_send, o_tab, o_vec, o_bars;
};

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// The split of the model over a cluster of C CTAs with R sequences; false if it does not fit.
inline bool dc_plan(DcPlan* p, size_t* smem_bytes, int S, int D, int H, int F, int C, int R) {
    const int hd = D / H;
    p->S = S; p->D = D; p->H = H; p->F = F; p->C = C; p->R = R;
    p->rg = ceil_div(R, 8);
    p->P = ceil_div(R * H, C);
    if (R > 16 || p->P > DC_MAX_PAIRS) return false;
    auto sliced = [&](int K) {
        DcProj q;
        q.n = 8 * ceil_div(ceil_div(D, C), 8);
        q.tiles = 1;
        q.slices = 1;
        for (int s = 4; s > 1; --s)
            if (K % 64 == 0 && (K / 64) % s == 0 && s * q.n <= 128) { q.slices = s; break; }
        q.rows = q.slices * q.n; q.kblocks = ceil_div(K, 64) / q.slices;
        return q;
    };
    p->q.n = 8 * ceil_div(ceil_div(3 * D, C), 8);
    p->q.tiles = ceil_div(p->q.n, 128);
    if (p->q.tiles == 2) p->q.n = 16 * ceil_div(p->q.n, 16);
    p->q.rows = p->q.n / p->q.tiles; p->q.slices = 1; p->q.kblocks = ceil_div(D, 64);
    p->o = sliced(D);
    p->d = sliced(F);
    p->g.n = 8 * ceil_div(ceil_div(F, C), 8);
    p->g.rows = 2 * p->g.n; p->g.tiles = 1; p->g.slices = 1; p->g.kblocks = ceil_div(D, 64);
    if (p->q.tiles > 2 || p->q.rows > 128 || p->o.n > 128 || p->g.rows > 128) return false;
    auto magic = [](int d) { return (uint32_t)((65536 + d - 1) / d); };
    p->p_magic = magic(p->P); p->h_magic = magic(H); p->g8_magic = magic(p->g.n / 8);
    if (R * p->o.n > 2 * DC_COMPUTE || R * p->g.n > 2 * DC_COMPUTE) return false;
    p->rank_bytes = 0;
    for (DcProj* pr : {&p->q, &p->o, &p->g, &p->d}) pr->umma_n = 16 * ceil_div(pr->slices * p->rg * 8, 16);
    int biggest = DC_KV_BYTES;
    for (DcProj* pr : {&p->q, &p->o, &p->g, &p->d}) {
        pr->bytes = (uint32_t)(pr->tiles * pr->kblocks * pr->rows * 128);
        p->rank_bytes += pr->bytes;
        // copies of up to 32 KB: a wait less per 64 columns of K
        pr->chunk = 1;
        for (int c = 2; c <= pr->kblocks; ++c)
            if (pr->kblocks % c == 0 && c * pr->rows * 128 <= 32 * 1024) pr->chunk = c;
        biggest = std::max(biggest, (pr->chunk * pr->rows * 128 + 1023) / 1024 * 1024);
    }
    p->vec_floats = (p->q.n + 2 * p->g.n + 2 * p->o.n + 2 * D + 3) / 4 * 4;
    uint32_t at = 0;
    auto take = [&](size_t bytes, size_t align) { at = (uint32_t)((at + align - 1) / align * align); const uint32_t o = at; at += (uint32_t)bytes; return o; };
    const uint32_t act_d = (uint32_t)(p->rg * ceil_div(D, 64) * 1024), act_f = (uint32_t)(p->rg * ceil_div(F, 64) * 1024);
    p->o_ax = take(act_d, 1024); p->o_att = take(act_d, 1024);
    // (an instruction with an odd number of 8-sequence groups reads one group behind the buffer, at most as much again as it
    // holds: for the first two buffers that lies inside the one that follows)
    p->o_ah = take(std::max({act_d, act_f, (uint32_t)(p->d.umma_n / 8 * p->d.kblocks * 1024)}), 1024);
    p->o_qkv = take((size_t)p->P * 3 * hd * 4, 128);
    p->o_rot = take(((size_t)p->P * 2 * hd + p->P) * 4, 128);
    p->o_x = take((size_t)C * R * p->o.n * 4, 128);
    p->o_send = take((size_t)std::max({R * p->o.n * 4, R * p->g.n * 2, p->P * hd * 2}), 128);
    p->o_tab = take((size_t)D / 4 * 2, 128);
    p->o_stage = take(std::max<size_t>((size_t)128 * DC_STAGE_LD, (size_t)32 * (hd + 4)) * 4, 128);
    p->o_vec = take((size_t)2 * p->vec_floats * 4, 128);
    p->o_bars = take((2 * DC_SLOTS + 6) * 8 + 2 * DC_SLOTS * 4 + 16, 128);
    // the ring comes first in memory: what a 128-row operand read of a shorter tile touches behind it is ours
    const int64_t budget = 227 * 1024 - 1024 - (int64_t)at;
    const int64_t ring = budget / 1024 * 1024;
    if (ring < 3 * (int64_t)biggest || at < DC_OVERRUN) return false;
    p->ring_bytes = (uint32_t)ring;
    for (uint32_t* o : {&p->o_ax, &p->o_att, &p->o_ah, &p->o_qkv, &p->o_rot, &p->o_x, &p->o_stage, &p->o_send, &p->o_tab, &p->o_vec, &p->o_bars})
        *o += p->ring_bytes;
    *smem_bytes = 1024 + (size_t)p->ring_bytes + at;
    return true;
}

// Whether the plan is better than the launch-per-kernel step, when `fit` clusters run at a time.  A wave of clusters takes a
// layer's chain of phases whatever it carries (14 us at width 64, 20 at 384, 27 - 35 at 1024), the other step grows slowly with
// the sequences, so the waves decide.  Cluster kernel : launch-per-kernel step, us per step at 128 cached rows:
//   one wave    width 384, 6 heads, 12 layers, 112 sequences 248 : 546, width 1024, 16 heads, 4 layers, 32 sequences 118 : 271
//   two         width 384, 200 sequences 483 : 662, width 1024, 64 heads, 28 sequences 218 : 281, width 768, 48 heads, 16 169 : 169
//   three       width 384, 336 sequences 721 : 802 (16 sequences per cluster), 12 heads, 200 681 : 687 (10);
//               width 768, 12 heads, 128 316 : 303 (8), width 1024, 64 heads, 32 322 : 287 (2), width 64, 256 84 : 60
//   four, five  width 384, 448 sequences 958 : 918, width 1024, 64 heads, 64 sequences 530 : 344
inline bool dc_pays(const DcPlan& p, int fit) {
    const int waves = ceil_div(ceil_div(p.S, p.R), fit);
    return waves <= 2 || (waves == 3 && p.R >= 10 && p.D >= 256);
}

}  // namespace tb
