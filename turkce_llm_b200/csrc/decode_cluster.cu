// One decode step of all layers, sequences spread over thread-block clusters.
//
// Sequences are independent of each other, so a decode step needs no grid-wide meeting point: a cluster of up to 16 CTAs
// (one per SM) takes up to 16 sequences through ALL layers, and different clusters never exchange anything.  Inside a
// cluster every CTA owns 1/16 of the output columns of each projection and 1/16 of the (sequence, head) pairs of the
// attention; what a phase produces is sent straight into the shared memory of all CTAs of the cluster (st.async, counted
// on an mbarrier of the receiver), so a phase ends with one remote store instead of a round trip through L2 and a barrier.
//
// What bounds it, and what follows from that:
//  * The chain of dependent phases (five per layer).  With a grid barrier and a re-load of the activations behind it a
//    phase cost ~6 us (366 us per step of 64 sequences); now all five take 10 us for one sequence per cluster and 15 for ten.
//  * Bytes: a CTA needs its slice of every weight matrix and the cache rows of its pairs.  None of them depends on the
//    step's own results (the new cache row is handled apart), so ONE producer warp streams them in the order of use
//    through a ring of ~130 KB that runs ahead of the chain, instead of in bursts behind each barrier.
//  * Products: weight columns are the M = 128 operand of tcgen05.mma, the sequences the N operand.  (mma.sync m16n8k16 runs
//    at one per ~18 clocks and SM on this part, measured; a layer's products would take 14,000 clocks with it.)  An
//    instruction costs ~40 clocks whatever N is, because it reads 128 rows of A from shared memory, so a tile of 24 columns
//    (out- and down-projection of a CTA at d_model 384) has its idle rows filled with further K slices: slice a of K
//    multiplies activation columns a, the off-diagonal blocks are ignored, the diagonal blocks added in a fixed order.
//  * Attention: one pass over the cache rows, a warp per 32 rows with a key per lane, float32 products of the float32 query and
//    probability with the bf16 cache rows; the partial results of a pair's warps are merged at the end.
// Measured, 12 layers of width 384, generate() with the LM head behind it: 64 sequences, cache 128 .. 256: 366 -> 207 us per step,
// 896 .. 1024: 719 -> 390; one sequence 267 -> 127 us.  What is left is latency: 64 sequences are 29,700 clocks per layer under
// ncu, with the tensor pipe active in 4 % of them, 27 % of the issue slots used and 1.1 TB/s from DRAM; most stalls are at the
// barriers between the steps of a phase.
//
// Replaces, for the decode step, the reference's re-run of lm_forward over the whole window per generated token
// (training/generate.c:186-212).
#include "common.h"
#include "decode_plan.h"
#include "ptx.cuh"
#include "step_kernels.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <vector>

namespace tb {

namespace {

struct DcLayer {
    bf16 *Kc, *Vc;                                        // [S, H, cap, hd]
    const CUtensorMap *mapK, *mapV;                       // (hd, cap, S*H) views, 64-row boxes
};

struct DcParams : DcPlan {
    int L, cap;
    const uint8_t* wt;                                    // [L][C][rank_bytes] operand images
    const float* vec;                                     // [L][C][vec_floats] biases and norm weights, see vec_layout_kernel
    float eps, inv_d, qscale;                             // qscale: log2(e) / sqrt(hd)
    const float *embed, *final_norm;
    const uint32_t* tok;
    const int* pos;
    const DcLayer* layers;
    const float *cos_t, *sin_t;
    bf16* out;                                            // [S, D] normalised hidden states for the LM head
    int* err;
};

__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// remote stores whose bytes are counted on an mbarrier of the same CTA as the destination
__device__ __forceinline__ void st_async_f32(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_16(uint32_t addr, const uint4& v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DC_COMPUTE) : "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr) : "memory");
}
// mbar_wait with the error word.  The waiting loop is a function of its own: inlined at every wait it cost registers and
// instructions on the way (4 - 8 % of the step).
__device__ __noinline__ bool dc_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err, int code) {
    if (mbar_wait(bar, parity, abort_flag)) return true;
    *abort_flag = 1;
    atomicCAS(err, 0, code);
    return false;
}
__device__ __forceinline__ bool dc_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err, int code) {
    return mbar_try_wait(bar, parity) || dc_wait_slow(bar, parity, abort_flag, err, code);
}

__device__ __forceinline__ float2 bf2_to_f2(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// byte offset of activation columns k .. k + 7 (k a multiple of 8) of sequence `row` in an operand buffer of kb K blocks:
// [8-sequence group][K block of 64][8 rows of 128 bytes, 128B swizzle]
__device__ __forceinline__ uint32_t act_offset(int row, int k, int kb) {
    return (uint32_t)(((row >> 3) * kb + (k >> 6)) * 1024 + (row & 7) * 128 + ((((k >> 3) ^ row) & 7) << 4));
}

template <int HD>
__global__ void __launch_bounds__(DC_THREADS, 1) decode_cluster_kernel(const __grid_constant__ DcParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);     // the same offset in every CTA
    uint8_t* ring = smem;
    const uint32_t s0 = smem_u32(smem);
    float* xbuf = reinterpret_cast<float*>(smem + p.o_x);              // [C][rows][o.n] residual stream, gathered from all CTAs
    uint16_t* tab = reinterpret_cast<uint16_t*>(smem + p.o_tab);       // [D / 4] place of columns 4 i .. 4 i + 3 of row 0 in it
    float* qkv_in = reinterpret_cast<float*>(smem + p.o_qkv);          // [P][3][HD] this CTA's pairs
    float* rq = reinterpret_cast<float*>(smem + p.o_rot);              // new q [P][HD] | new v [P][HD] | score of the new key [P]
    float* stage = reinterpret_cast<float*>(smem + p.o_stage);         // [128][17], or the attention's partial results
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.o_bars);
    uint64_t* empty = full + DC_SLOTS;
    uint64_t* acc_bar = empty + DC_SLOTS;
    uint64_t* x_bar = acc_bar + 1;                                     // x, then x2, of every layer
    uint64_t* n_bar = acc_bar + 2;                                     // their normalised form, by this CTA's warps
    uint64_t* qkv_bar = acc_bar + 3;
    uint64_t* att_bar = acc_bar + 4;
    uint64_t* h_bar = acc_bar + 5;
    volatile uint32_t* chunk_off = reinterpret_cast<volatile uint32_t*>(acc_bar + 6);      // [DC_SLOTS] place in the ring
    volatile uint32_t* chunk_end = chunk_off + DC_SLOTS;                                     // [DC_SLOTS] running end position
    uint32_t* tmem_slot = const_cast<uint32_t*>(chunk_end) + DC_SLOTS;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int C = p.C, D = p.D, H = p.H, F = p.F;
    const int rank = (int)cluster_ctarank();
    const int row0 = ((int)blockIdx.x / C) * p.R;
    const int rows = min(p.R, p.S - row0);                              // sequences of this cluster
    const int pair0 = rank * p.P;
    const int pairs = max(0, min(p.P, rows * H - pair0));               // pairs of this CTA

    const uint32_t x_bytes = (uint32_t)(C * rows * p.o.n * 4);
    if (tid == 0) {
#pragma unroll 1
        for (int i = 0; i < DC_SLOTS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], DC_GROUP); }
#pragma unroll 1
        for (int i = 0; i < 6; ++i) mbar_init(acc_bar + i, i == 2 ? DC_WARPS : 1);
        *abort_flag = 0;
        fence_mbar_init();
        // armed before any CTA can send (the cluster barrier below); re-armed by whoever waits on them
        mbar_expect_tx(x_bar, x_bytes);
        mbar_expect_tx(att_bar, (uint32_t)(rows * D * 2));
        mbar_expect_tx(h_bar, (uint32_t)(rows * F * 2));
        if (pairs > 0) mbar_expect_tx(qkv_bar, (uint32_t)(pairs * 3 * HD * 4));
    }
    // operand buffers start from zero: columns that pad K to a multiple of 64 meet zero weights
#pragma unroll 1
    for (uint32_t i = p.o_ax + tid * 16; i < p.o_qkv; i += DC_THREADS * 16) *reinterpret_cast<uint4*>(smem + i) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
    for (int i = tid; i < D / 4; i += DC_THREADS) tab[i] = (uint16_t)((4 * i / p.o.n) * rows * p.o.n + 4 * i % p.o.n);
    if (warp == DC_WARPS + 1) { tmem_alloc(tmem_slot, DC_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents_now();
    const int t = *p.pos;                                               // position of the new token = cached rows
    const int nblk = (t + DC_KV_ROWS - 1) / DC_KV_ROWS;
    const int q_chunks = p.q.tiles * (p.q.kblocks / p.q.chunk);
    const int layer_chunks = q_chunks + pairs * nblk + p.o.kblocks / p.o.chunk + p.g.kblocks / p.g.chunk + p.d.kblocks / p.d.chunk;

    if (warp == DC_WARPS) {
        // ------------------------------------------------------------------ producer: the CTA's bytes in the order of use
        if (elect_one()) {
            uint32_t head = 0, head_at = 0, tail = 0, issued = 0, popped = 0;   // running positions; head_at = head in the ring
            bool ok = true;
            const uint32_t ring_bytes = p.ring_bytes;
            auto place = [&](uint32_t bytes) -> int {
                const uint32_t size = (bytes + 1023u) & ~1023u;
                if (head_at + size > ring_bytes) { head += ring_bytes - head_at; head_at = 0; }
                const uint32_t end = head + size;
                while (issued - popped >= DC_SLOTS || end - tail > ring_bytes) {
                    const int s = (int)(popped % DC_SLOTS);
                    if (!dc_wait(&empty[s], (popped / DC_SLOTS) & 1u, abort_flag, p.err, 44)) { ok = false; return 0; }
                    tail = chunk_end[s];
                    ++popped;
                }
                const int s = (int)(issued % DC_SLOTS);
                chunk_off[s] = head_at;
                chunk_end[s] = end;
                mbar_expect_tx(&full[s], bytes);
                head = end; head_at += size;
                ++issued;
                return s;
            };
#pragma unroll 1
            for (int l = 0; l < p.L && ok; ++l) {
                const uint8_t* w = p.wt + ((size_t)l * C + rank) * p.rank_bytes;
#pragma unroll 1
                for (int phase = 0; phase < 5 && ok; ++phase) {
                    if (phase == 1) {
                        const CUtensorMap *mk = p.layers[l].mapK, *mv = p.layers[l].mapV;
                        const int item0 = row0 * H + pair0;
                        int b = 0, i = 0;
#pragma unroll 1
                        while (b < nblk && pairs > 0) {
                            const int s = place(DC_KV_BYTES);
                            if (!ok) break;
                            uint8_t* dst = ring + chunk_off[s];
                            tma_load_3d(dst, mk, &full[s], 0, b * DC_KV_ROWS, item0 + i);
                            tma_load_3d(dst + DC_KV_BYTES / 2, mv, &full[s], 0, b * DC_KV_ROWS, item0 + i);
                            if (++i == pairs) { i = 0; ++b; }
                        }
                        continue;
                    }
                    const DcProj pr = phase == 0 ? p.q : phase == 2 ? p.o : phase == 3 ? p.g : p.d;
                    const int n = pr.tiles * (pr.kblocks / pr.chunk);
                    const uint32_t bytes = (uint32_t)(pr.chunk * pr.rows * 128);
#pragma unroll 1
                    for (int i = 0; i < n; ++i) {
                        const int s = place(bytes);
                        if (!ok) break;
                        bulk_load(ring + chunk_off[s], w, bytes, &full[s]);
                        w += bytes;
                    }
                }
            }
        }
    } else if (warp == DC_WARPS + 1) {
        // ------------------------------------------------------------------ tensor core
        if (elect_one()) {
            bool ok = true;
            uint32_t ci = 0, at = 0;                                          // chunks seen, place of the next one in the ring
            const uint32_t ring_bytes = p.ring_bytes;
            auto take = [&](uint32_t size) {                                  // (the producer's placement over again)
                if (at + size > ring_bytes) at = 0;
                const uint32_t here = at;
                at += size;
                ++ci;
                return here;
            };
#pragma unroll 1
            for (int l = 0; l < p.L && ok; ++l) {
#pragma unroll 1
                for (int phase = 0; phase < 4 && ok; ++phase) {
                    // what the product reads, and the barrier that says it is there
                    const DcProj pr = phase == 0 ? p.q : phase == 1 ? p.o : phase == 2 ? p.g : p.d;
                    const uint32_t act = s0 + (phase == 1 ? p.o_att : phase == 3 ? p.o_ah : p.o_ax);
                    uint32_t dcol = tmem + (uint32_t)(phase == 0 ? DC_COL_Q : phase == 1 ? DC_COL_O : phase == 2 ? DC_COL_G : DC_COL_D);
                    uint64_t* bar = phase == 1 ? att_bar : phase == 3 ? h_bar : n_bar;
                    const uint32_t parity = (phase & 1) ? (uint32_t)l & 1u : (uint32_t)(phase >> 1);
                    if (phase == 1)
#pragma unroll 1
                        for (int i = pairs * nblk; i > 0; --i) take(DC_KV_BYTES);
                    const uint32_t idesc = umma_idesc(1u, 0u, 0u, 128, (uint32_t)pr.umma_n);
                    uint64_t b = umma_desc_sw128(act, 16, (uint32_t)(pr.kblocks * 1024));
                    const int nch = pr.kblocks / pr.chunk;
                    const uint32_t size = ((uint32_t)(pr.chunk * pr.rows * 128) + 1023u) & ~1023u;
                    const uint64_t astep = (uint64_t)(pr.rows * 8);
                    if (!dc_wait(bar, parity, abort_flag, p.err, 45)) { ok = false; break; }
                    // (written by ordinary and remote stores: fence before the tensor core reads them)
                    fence_proxy_async();
#pragma unroll 1
                    for (int tile = 0; tile < pr.tiles && ok; ++tile, dcol += 16, b -= (uint64_t)(64 * pr.kblocks)) {
                        uint32_t acc = 0;
#pragma unroll 1
                        for (int c = 0; c < nch; ++c) {
                            const int s = (int)(ci % DC_SLOTS);
                            const uint32_t par = (ci / DC_SLOTS) & 1u;
                            uint64_t a = umma_desc_sw128(s0 + take(size), 16, 1024);
                            if (!dc_wait(&full[s], par, abort_flag, p.err, 45)) { ok = false; break; }
                            tc_fence_after();
#pragma unroll 1
                            for (int kb = 0; kb < pr.chunk; ++kb, a += astep, b += 64) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) { umma_bf16(dcol, a + 2 * k, b + 2 * k, idesc, acc); acc = 1; }
                            }
                            umma_commit(&empty[s]);
                            mbar_arrive(&empty[s]);                        // (the second arrival; a cache chunk gets one from each of its warps)
                        }
                    }
                    if (ok) umma_commit(acc_bar);
                    if (phase & 1) mbar_expect_tx(bar, (uint32_t)(rows * (phase == 1 ? D : F) * 2));
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ compute warps
        // A wait that gives up sets the abort flag and the thread carries on (every later wait then returns at once), so
        // that all threads meet at the same barriers.
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            dc_wait(bar, parity, abort_flag, p.err, 46);
        };
        uint32_t acc_phase = 0, x_phase = 0;
        const int on = p.o.n, gn = p.g.n, qn = p.q.n;
        const int oc0 = rank * on, gc0 = rank * gn, qc0 = rank * qn;            // first columns this CTA owns
        // what a phase produces is first gathered in shared memory; warp w then sends all of it to CTA w: the 32 remote stores
        // of an instruction go to one CTA and, as far as the layout allows, to adjacent addresses.  (Lanes that send to
        // 8 or 16 different CTAs took three times as long for the same bytes: 2,900 against ~1,000 clocks for 960 bytes from
        // each of 16 CTAs to each.)
        uint8_t* send = smem + p.o_send;
        const uint32_t peer = mapa_u32(s0, (uint32_t)min(warp, C - 1));
        // items of the epilogues, two per thread: (sequence r, own column c)
        float x[2];                                                             // this thread's values of the residual stream
        int x_src[2], h_src[2];                                                 // where their accumulators are staged (-1: none)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = tid + u * DC_COMPUTE;
            int r = i / on, c = i % on;
            x_src[u] = r < rows ? c * DC_STAGE_LD + r : -1;
            x[u] = r < rows && oc0 + c < D ? __ldg(p.embed + (long long)p.tok[row0 + r] * D + oc0 + c) : 0.0f;
            r = i / gn; c = i % gn;
            h_src[u] = r < rows ? c * DC_STAGE_LD + r : -1;
        }
        const int sl_mine = (tid & 127) / on, sl_first = (warp & 3) * 32 / on, sl_last = ((warp & 3) * 32 + 31) / on;   // K slices of an accumulator row
        // attention: two warps take a block of 64 cached rows of a pair, 32 rows each; with fewer than eight pairs the blocks
        // of a pair go round several such groups.  Partial results of a pair: one per warp that has had rows.
        constexpr int PART_LD = HD + 4;
        const int gpp_shift = pairs <= 1 ? 3 : pairs <= 2 ? 2 : pairs <= 4 ? 1 : 0, gpp = 1 << gpp_shift;
        const int pr = warp >> (1 + gpp_shift), sub = (warp >> 1) & (gpp - 1);
        const int nparts = 2 * min(gpp, nblk);
        // one thread per rotated pair of the new row, HP threads per (sequence, head): a power of two, so that their sums are shuffles
        constexpr int HALF = HD / 2, HP = HD == 48 ? 32 : HALF;
        const size_t kv_at = ((size_t)(row0 * H + pair0 + tid / HP) * p.cap + t) * HD + 2 * (tid % HP);              // new cache row
        // RMSNorm: places of this lane's columns 4 (lane + 32 k), k < 4, in a row of xbuf
        uint32_t x_at[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x_at[k] = 4 * (lane + 32 * k) < D ? tab[lane + 32 * k] : 0u;
        // biases and norm weights of a layer, double-buffered: bq [qn] | bg [2 gn] | bo [on] | bd [on] | attention norm [D] | FFN norm [D]
        const float* vec_src = p.vec + (size_t)rank * p.vec_floats + tid * 4;
        auto fetch_vec = [&](int l) {
            float* dst = reinterpret_cast<float*>(smem + p.o_vec) + (l & 1) * p.vec_floats;
#pragma unroll 1
            for (int i = tid * 4; i < p.vec_floats; i += DC_COMPUTE * 4) cp_async_16(dst + i, vec_src + (i - tid * 4));
            vec_src += (size_t)C * p.vec_floats;
        };
        // this CTA's columns of the residual stream to all CTAs
        auto publish = [&]() {
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (x_src[u] >= 0) reinterpret_cast<float*>(send)[tid + u * DC_COMPUTE] = x[u];
            compute_sync();
            if (warp < C) {
                const uint32_t bar = peer + (smem_u32(x_bar) - s0), dst = peer + p.o_x + (uint32_t)(rank * rows * on) * 4;
#pragma unroll 1
                for (int i = lane * 16; i < rows * on * 4; i += 512) st_async_16(dst + (uint32_t)i, *reinterpret_cast<const uint4*>(send + i), bar);
            }
        };
        // RMSNorm of the gathered rows, a warp per row -> bf16 operand; lane owns columns 4 (lane + 32 k).
        auto row_at = [&](int c0, int k) { return c0 < 128 ? x_at[k] : (uint32_t)tab[(c0 >> 2) + 32 * k]; };
        auto row_rms = [&](int r) {
            const float* row = xbuf + r * on;
            float ss = 0.0f;
#pragma unroll 1
            for (int c0 = 4 * lane; c0 < D; c0 += 512) {
                float4 v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    v[k] = c0 + 128 * k < D ? *reinterpret_cast<const float4*>(row + row_at(c0, k)) : make_float4(0.f, 0.f, 0.f, 0.f);
                float part[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) part[k] = (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
                ss += (part[0] + part[1]) + (part[2] + part[3]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            return rsqrtf(ss * p.inv_d + p.eps);
        };
        auto scaled = [&](int r, uint32_t at, float rr, float4 wv) {
            const float4 v = *reinterpret_cast<const float4*>(xbuf + r * on + at);
            __nv_bfloat162 lo = __floats2bfloat162_rn(v.x * rr * wv.x, v.y * rr * wv.y);
            __nv_bfloat162 hi = __floats2bfloat162_rn(v.z * rr * wv.z, v.w * rr * wv.w);
            return make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
        };
        auto normalise = [&](const float* w) {
            if (warp < rows) {
                const float rr = row_rms(warp);
                uint8_t* dst = smem + p.o_ax + (warp >> 3) * p.q.kblocks * 1024 + (warp & 7) * 128 + (lane & 1) * 8;
#pragma unroll 1
                for (int c0 = 4 * lane; c0 < D; c0 += 512) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int c = c0 + 128 * k;
                        if (c < D)
                            *reinterpret_cast<uint2*>(dst + (c >> 6) * 1024 + ((((c >> 3) ^ warp) & 7) << 4)) =
                                scaled(warp, row_at(c0, k), rr, *reinterpret_cast<const float4*>(w + c));
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(n_bar);           // (the tensor-core thread fences before the operand is read)
        };
        auto wait_x = [&]() {
            wait(x_bar, x_phase);
            x_phase ^= 1u;
            if (tid == DC_COMPUTE - 1) mbar_expect_tx(x_bar, x_bytes);
        };
        auto acc_wait = [&]() {
            wait(acc_bar, acc_phase);
            acc_phase ^= 1u;
            tc_fence_after();
        };

        publish();
        fetch_vec(0);
        cp_async_wait();
        compute_sync();
#pragma unroll 1
        for (int l = 0; l < p.L; ++l) {
            const float* vec = reinterpret_cast<const float*>(smem + p.o_vec) + (l & 1) * p.vec_floats;
            const float *bg = vec + qn, *bo = bg + 2 * gn;
            bf16 *const Kc = p.layers[l].Kc, *const Vc = p.layers[l].Vc;         // (asked for long before they are needed)
#pragma unroll 1
            for (int phase = 0; phase < 4; ++phase) {
                if ((phase & 1) == 0) {
                    wait_x();
                    normalise(bo + 2 * on + (phase >> 1) * D);
                }
                // -------------------------------------------------------- accumulator -> stage[weight row][sequence]
                // (one place for the four products; the diagonal blocks of slices a and a + 1 at a time)
                const int slices = phase == 1 ? p.o.slices : phase == 3 ? p.d.slices : 1;
                if (phase == 0) {
                    // ------------------------------------------------------ QKV: every value to the CTA that owns its pair
                    if (warp < 4) {
                        acc_wait();
#pragma unroll 1
                        for (int tile = 0; tile < p.q.tiles; ++tile) {
                            const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(DC_COL_Q + 16 * tile);
                            const int lc = tile * p.q.rows + tid, c = qc0 + lc;
                            const int which = c >= 2 * D ? 2 : c >= D ? 1 : 0, cin = c - which * D, head = cin / HD;
                            int dest = (int)((uint32_t)head * p.p_magic >> 16), slot = head - dest * p.P;   // pair = sequence * H + head
                            const int dstep = (int)((uint32_t)H * p.p_magic >> 16), sstep = H - dstep * p.P;
                            const uint32_t base = s0 + p.o_qkv + (uint32_t)(which * HD + cin % HD) * 4, bar = smem_u32(qkv_bar);
                            const bool mine = tid < p.q.rows && c < 3 * D;
                            const float bias = mine ? vec[lc] : 0.0f;
#pragma unroll 1
                            for (int r0 = 0; r0 < rows; r0 += 8) {
                                uint32_t v[8];
                                tmem_ld8(ta + (uint32_t)r0, v);
                                tmem_ld_wait();
#pragma unroll
                                for (int r = 0; r < 8; ++r) {
                                    if (mine && r0 + r < rows)
                                        st_async_f32(mapa_u32(base + (uint32_t)(slot * 3 * HD) * 4, (uint32_t)dest), __uint_as_float(v[r]) + bias,
                                                     mapa_u32(bar, (uint32_t)dest));
                                    dest += dstep; slot += sstep;
                                    if (slot >= p.P) { slot -= p.P; ++dest; }
                                }
                            }
                        }
                        tc_fence_before();
                    }
                } else {
                    // ------------------------------------------------------ accumulator -> stage[weight row][sequence]
                    // (one place for the other three products; the diagonal blocks of slices a and a + 1 at a time)
                    if (warp < 4) {
                        acc_wait();
                        const int row = warp * 32 + lane, mine = phase == 2 ? 0 : sl_mine, last = phase == 2 ? 0 : min(slices - 1, sl_last);
                        const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(phase == 1 ? DC_COL_O : phase == 2 ? DC_COL_G : DC_COL_D);
#pragma unroll 1
                        for (int a = phase == 2 ? 0 : sl_first; a <= last; a += 2) {
                            uint32_t v[4][8];
                            const int hi = rows > 8 ? slices : 0, nx = a < last ? 1 : 0;
                            tmem_ld8(ta + (uint32_t)(a * 8), v[0]);
                            tmem_ld8(ta + (uint32_t)((a + nx) * 8), v[1]);
                            tmem_ld8(ta + (uint32_t)((a + hi) * 8), v[2]);
                            tmem_ld8(ta + (uint32_t)((a + nx + hi) * 8), v[3]);
                            tmem_ld_wait();
                            if (mine == a || mine == a + 1) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) stage[row * DC_STAGE_LD + i] = __uint_as_float(mine == a ? v[0][i] : v[1][i]);
                                if (rows > 8)
#pragma unroll
                                    for (int i = 0; i < 8; ++i) stage[row * DC_STAGE_LD + 8 + i] = __uint_as_float(mine == a ? v[2][i] : v[3][i]);
                            }
                        }
                        tc_fence_before();
                    }
                    if (phase == 3) cp_async_wait();                             // the next layer's vectors, before the barrier
                    compute_sync();
                }
                if (phase == 0) {
                    // ------------------------------------------------------ rotary embedding, cache append
                    float* rv = rq + p.P * HD;
                    float* snew = rv + p.P * HD;
                    if (pairs > 0) {
                        const int i = tid / HP, k = tid % HP;
                        const bool mine = i < pairs && k < HALF;
                        float c = 0.f, sn = 0.f;
                        if (mine) { c = __ldg(p.cos_t + t * HALF + k); sn = __ldg(p.sin_t + t * HALF + k); }
                        wait(qkv_bar, (uint32_t)l & 1u);
                        if (tid == DC_COMPUTE - 1) mbar_expect_tx(qkv_bar, (uint32_t)(pairs * 3 * HD * 4));
                        float dot = 0.0f;                                        // score of the new key
                        if (mine) {
                            const float* in = qkv_in + i * 3 * HD + 2 * k;
                            const float q0 = in[0], q1 = in[1], k0 = in[HD], k1 = in[HD + 1], v0 = in[2 * HD], v1 = in[2 * HD + 1];
                            const float r0 = (q0 * c - q1 * sn) * p.qscale, r1 = (q0 * sn + q1 * c) * p.qscale;
                            *reinterpret_cast<float2*>(rq + i * HD + 2 * k) = make_float2(r0, r1);
                            const __nv_bfloat162 kn = __floats2bfloat162_rn(k0 * c - k1 * sn, k0 * sn + k1 * c);
                            const __nv_bfloat162 vn = __floats2bfloat162_rn(v0, v1);
                            const size_t o = kv_at;
                            *reinterpret_cast<__nv_bfloat162*>(Kc + o) = kn;
                            *reinterpret_cast<__nv_bfloat162*>(Vc + o) = vn;
                            // (the new row takes part as the cache holds it)
                            dot = r0 * __bfloat162float(kn.x) + r1 * __bfloat162float(kn.y);
                            *reinterpret_cast<float2*>(rv + i * HD + 2 * k) = make_float2(__bfloat162float(vn.x), __bfloat162float(vn.y));
                        }
                        if (warp * 32 < pairs * HP) {
#pragma unroll
                            for (int o = HP / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                            if (i < pairs && k == 0) snew[i] = dot;
                        }
                    }
                    compute_sync();
                    if (l + 1 < p.L) fetch_vec(l + 1);
                    // ------------------------------------------------------ attention over the cached rows
                    constexpr int VL = HD == 48 ? 8 : HD / 8;                    // lanes that cover a value row (of 48: two have its zero padding)
                    constexpr int VK = 32 / VL;                                  // value rows per pass of the warp
                    if (pr < pairs) {
                        const float* q = rq + pr * HD;
                        float m = -INFINITY, lsum = 0.0f;
                        float2 acc[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[i] = make_float2(0.f, 0.f);
                        uint32_t ci = (uint32_t)(l * layer_chunks + q_chunks + sub * pairs + pr);
#pragma unroll 1
                        for (int b = sub; b < nblk; b += gpp, ci += (uint32_t)(gpp * pairs)) {
                            const int s = (int)(ci % DC_SLOTS);
                            wait(&full[s], (ci / DC_SLOTS) & 1u);
                            const uint8_t* kt = ring + chunk_off[s] + (warp & 1) * 32 * 128;
                            const uint8_t* vt = kt + DC_KV_BYTES / 2;
                            const int first = b * DC_KV_ROWS + (warp & 1) * 32;  // this warp's 32 cached rows, a key per lane
                            if (first < t) {
                                float2 d2 = make_float2(0.f, 0.f), e2 = make_float2(0.f, 0.f);
#pragma unroll
                                for (int c = 0; c < HD / 8; ++c) {
                                    const uint4 kk = *reinterpret_cast<const uint4*>(kt + lane * 128 + ((c ^ (lane & 7)) << 4));
                                    const float4 q0 = *reinterpret_cast<const float4*>(q + 8 * c), q1 = *reinterpret_cast<const float4*>(q + 8 * c + 4);
                                    d2 = __ffma2_rn(bf2_to_f2(kk.x), make_float2(q0.x, q0.y), d2);
                                    e2 = __ffma2_rn(bf2_to_f2(kk.y), make_float2(q0.z, q0.w), e2);
                                    d2 = __ffma2_rn(bf2_to_f2(kk.z), make_float2(q1.x, q1.y), d2);
                                    e2 = __ffma2_rn(bf2_to_f2(kk.w), make_float2(q1.z, q1.w), e2);
                                }
                                float sc = (d2.x + e2.x) + (d2.y + e2.y);
                                if (first + lane >= t) sc = -INFINITY;
                                float mx = sc;
#pragma unroll
                                for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                                const float m_new = fmaxf(m, mx);                 // finite: row `first` exists
                                const float corr = ex2_approx(m - m_new);
                                const float e = ex2_approx(sc - m_new);
                                m = m_new;
                                lsum = lsum * corr + e;
                                const float2 c2 = make_float2(corr, corr);
#pragma unroll
                                for (int i = 0; i < 4; ++i) acc[i] = __fmul2_rn(acc[i], c2);
#pragma unroll
                                for (int i = 0; i < 32 / VK; ++i) {
                                    const int key = i * VK + lane / VL;
                                    const float pk = __shfl_sync(0xffffffffu, e, key);
                                    const uint4 vv = *reinterpret_cast<const uint4*>(vt + key * 128 + (((lane % VL) ^ (key & 7)) << 4));
                                    const float2 p2 = make_float2(pk, pk);
                                    acc[0] = __ffma2_rn(bf2_to_f2(vv.x), p2, acc[0]);
                                    acc[1] = __ffma2_rn(bf2_to_f2(vv.y), p2, acc[1]);
                                    acc[2] = __ffma2_rn(bf2_to_f2(vv.z), p2, acc[2]);
                                    acc[3] = __ffma2_rn(bf2_to_f2(vv.w), p2, acc[3]);
                                }
                            }
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&empty[s]);
                        }
#pragma unroll
                        for (int o = VL; o < 32; o <<= 1)
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                acc[i].x += __shfl_xor_sync(0xffffffffu, acc[i].x, o);
                                acc[i].y += __shfl_xor_sync(0xffffffffu, acc[i].y, o);
                            }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
                        float* part = stage + (pr * 2 * gpp + sub * 2 + (warp & 1)) * PART_LD;
                        if (lane < HD / 8) {
                            *reinterpret_cast<float4*>(part + lane * 8) = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
                            *reinterpret_cast<float4*>(part + lane * 8 + 4) = make_float4(acc[2].x, acc[2].y, acc[3].x, acc[3].y);
                        }
                        if (lane == 0) { part[HD] = m; part[HD + 1] = lsum; }
                    }
                    compute_sync();
                    // ------------------------------------------------------ partial results of a pair's warps merged
                    if (tid < ((pairs * HD + 31) & ~31)) {
                        const int pair = tid / HD, d = tid % HD;
                        const bool valid = pair < pairs;
                        const float* part = stage + (valid ? pair : 0) * 2 * gpp * PART_LD;
                        const float sn = snew[valid ? pair : 0];
                        float mm = sn;
#pragma unroll 4
                        for (int i = 0; i < nparts; ++i) mm = fmaxf(mm, part[i * PART_LD + HD]);
                        const float en = ex2_approx(sn - mm);
                        float num = en * rv[(valid ? pair : 0) * HD + d], den = en;
#pragma unroll 4
                        for (int i = 0; i < nparts; ++i) {
                            const float w = ex2_approx(part[i * PART_LD + HD] - mm);       // 0 for a warp without rows
                            num += w * part[i * PART_LD + d];
                            den += w * part[i * PART_LD + HD + 1];
                        }
                        if (valid) reinterpret_cast<bf16*>(send)[tid] = __float2bfloat16_rn(__fdividef(num, den));
                    }
                    compute_sync();
                    if (warp < C) {
                        const uint32_t bar = peer + (smem_u32(att_bar) - s0);
#pragma unroll 1
                        for (int i = lane; i < pairs * (HD / 8); i += 32) {
                            const int g = pair0 + i / (HD / 8), r = (int)((uint32_t)g * p.h_magic >> 16);
                            st_async_16(peer + p.o_att + act_offset(r, (g - r * H) * HD + (i % (HD / 8)) * 8, p.q.kblocks),
                                        *reinterpret_cast<const uint4*>(send + i * 16), bar);
                        }
                    }
                } else if (phase == 2) {
                    // ------------------------------------------------------ SwiGLU
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (h_src[u] >= 0) {
                            const int c = h_src[u] / DC_STAGE_LD;
                            const float gv = stage[h_src[u]] + bg[c], uv = stage[h_src[u] + gn * DC_STAGE_LD] + bg[gn + c];
                            reinterpret_cast<bf16*>(send)[tid + u * DC_COMPUTE] =
                                __float2bfloat16_rn(gv * __fdividef(1.0f, 1.0f + ex2_approx(-gv * 1.4426950408889634f)) * uv);
                        }
                    compute_sync();
                    if (warp < C) {
                        const uint32_t bar = peer + (smem_u32(h_bar) - s0);
                        const int g8 = gn >> 3, kb = p.d.kblocks * p.d.slices;
#pragma unroll 1
                        for (int i = lane; i < rows * g8; i += 32) {
                            const int r = (int)((uint32_t)i * p.g8_magic >> 16), k = gc0 + (i - r * g8) * 8;
                            if (k < F) st_async_16(peer + p.o_ah + act_offset(r, k, kb), *reinterpret_cast<const uint4*>(send + i * 16), bar);
                        }
                    }
                } else {
                    // ------------------------------------------------------ out- / down-projection + residual
                    const float* b = phase == 1 ? bo : bo + on;
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (x_src[u] >= 0) {
                            float part[4];
#pragma unroll
                            for (int a = 0; a < 4; ++a) part[a] = a < slices ? stage[x_src[u] + a * on * DC_STAGE_LD] : 0.0f;
                            x[u] = ((part[0] + part[1]) + (part[2] + part[3])) + b[x_src[u] / DC_STAGE_LD] + x[u];
                        }
                    }
                    publish();
                }
            }
        }
        // ------------------------------------------------------------------ final norm: sequence r by CTA r mod C
        wait_x();
        if (warp < 2) {
            const int r = rank + warp * C;
            if (r < rows) {
                const float rr = row_rms(r);
#pragma unroll 1
                for (int c = 4 * lane; c < D; c += 128)
                    *reinterpret_cast<uint2*>(p.out + (long long)(row0 + r) * D + c) =
                        scaled(r, tab[c >> 2], rr, __ldg(reinterpret_cast<const float4*>(p.final_norm + c)));
            }
        }
    }

    // ---------------------------------------------------------------------- teardown
    __syncwarp();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);      // copies in flight land before the shared memory is released
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                           // nobody sends into this CTA any more
    if (warp == DC_WARPS + 1) {
        tc_fence_after();
        tmem_dealloc(tmem, DC_TMEM_COLS);
    }
}

// W [K][N] (row-major bf16) -> the operand image of every CTA: [tile][K block of 64][rows of 128 bytes, 128B swizzle];
// weight row r of a tile is slice a = r / n, column r % n; with pair_off > 0 rows n .. 2n - 1 are columns pair_off + ..
// One thread per 16-byte piece.
__global__ void cluster_layout_kernel(const bf16* __restrict__ W, uint8_t* __restrict__ out, DcProj pr, int K, int N, uint32_t rank_bytes,
                                      int pair_off) {
    const int rank = blockIdx.y;
    const int pieces = pr.tiles * pr.kblocks * pr.rows * 8;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pieces; i += gridDim.x * blockDim.x) {
        const int j = i & 7, r = (i >> 3) % pr.rows, blk = (i >> 3) / pr.rows;
        const int tile = blk / pr.kblocks;
        int slice = 0, col;
        if (pair_off > 0) {
            const int u = rank * pr.n + (r < pr.n ? r : r - pr.n);
            col = u < pair_off ? (r < pr.n ? u : pair_off + u) : N;
        } else if (pr.slices > 1) {
            slice = r / pr.n;
            col = rank * pr.n + r % pr.n;
        } else {
            col = rank * pr.n + tile * pr.rows + r;
        }
        const int k0 = (slice * pr.kblocks + blk % pr.kblocks) * 64 + j * 8;
        __align__(16) bf16 v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            v[e] = (col < N && k0 + e < K) ? W[(long long)(k0 + e) * N + col] : __float2bfloat16_rn(0.0f);
        *reinterpret_cast<uint4*>(out + (size_t)rank * rank_bytes + (size_t)blk * pr.rows * 128 + r * 128 + ((j ^ (r & 7)) << 4)) =
            *reinterpret_cast<const uint4*>(v);
    }
}

// Value rows from .. to - 1 of every cache = 0.  The attention takes rows in groups of 32 and gives those behind the last one the
// weight 0; what an earlier sequence left there need not be finite.  Cleared where a prompt begins, by how far the earlier one
// went (64 sequences, 128 rows: 75 MB): a test of every row in the attention itself cost 1 - 3 % of a step.
__global__ void clear_values_kernel(const DcLayer* __restrict__ layers, int heads, int cap, int from, int to, int hd) {
    pdl_wait();
    pdl_launch_dependents();
    bf16* const V = layers[blockIdx.y].Vc;
    const int pieces = (to - from) * (hd / 8);                            // 16 bytes each
    for (int h = blockIdx.x; h < heads; h += gridDim.x) {
        uint4* row = reinterpret_cast<uint4*>(V + ((size_t)h * cap + from) * hd);
        for (int i = threadIdx.x; i < pieces; i += blockDim.x) row[i] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// [L][C][bq (q.n) | bg (2 g.n) | bo (o.n) | bd (o.n) | attention norm (D) | FFN norm (D)]: what a CTA's epilogues add
// and scale by, zeros where its columns end
__global__ void vec_layout_kernel(const float* __restrict__ bq, const float* __restrict__ bg, const float* __restrict__ bo,
                                  const float* __restrict__ bd, const float* __restrict__ w1, const float* __restrict__ w2,
                                  float* __restrict__ out, int D, int F, int qn, int gn, int on, int vec_floats) {
    const int rank = blockIdx.x;
    for (int i = threadIdx.x; i < vec_floats; i += blockDim.x) {
        int c = i;
        float v = 0.0f;
        if (c < qn) { if (rank * qn + c < 3 * D) v = bq[rank * qn + c]; }
        else if ((c -= qn) < 2 * gn) {
            const int u = rank * gn + (c < gn ? c : c - gn);
            if (u < F) v = bg[(c < gn ? 0 : F) + u];
        }
        else if ((c -= 2 * gn) < on) { if (rank * on + c < D) v = bo[rank * on + c]; }
        else if ((c -= on) < on) { if (rank * on + c < D) v = bd[rank * on + c]; }
        else if ((c -= on) < D) v = w1[c];
        else if ((c -= D) < D) v = w2[c];
        out[(size_t)rank * vec_floats + i] = v;
    }
}

typedef void (*DcKernel)(const DcParams);
DcKernel dc_kernel(int hd) {
    return hd == 64 ? decode_cluster_kernel<64> : hd == 48 ? decode_cluster_kernel<48> : hd == 32 ? decode_cluster_kernel<32> : decode_cluster_kernel<16>;
}

cudaLaunchConfig_t dc_config(const DcParams& p, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ceil_div(p.S, p.R) * p.C)); cfg.blockDim = dim3(DC_THREADS);
    cfg.dynamicSmemBytes = smem; cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.C; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_mode() != 0 ? 2 : 1;
    return cfg;
}

}  // namespace

struct DecodeCluster {
    DcParams p;
    size_t smem = 0;
    uint8_t* wt = nullptr;
    float* vec = nullptr;
    DcLayer* d_layers = nullptr;
    CUtensorMap* d_maps = nullptr;             // [L][2]: K and V cache views
};

bool decode_cluster_supported(int D, int H, int F) {
    const int hd = H > 0 ? D / H : 0;
    return D % 16 == 0 && F % 16 == 0 && D <= 1024 && F <= 1024 && hd % 16 == 0 && hd >= 16 && hd <= 64;
}

// *out stays NULL when the shape does not fit a cluster or takes too many of them (the caller keeps the launch-per-kernel step).
int decode_cluster_create(DeviceCtx* ctx, DecodeCluster** out, int S, int D, int H, int F, int L, int cap, float eps, float scale) {
    *out = nullptr;
    if (!decode_cluster_supported(D, H, F) || L < 1 || S < 1) return 0;
    DcParams p;
    std::memset(&p, 0, sizeof(p));
    size_t smem = 0;
    const DcKernel kernel = dc_kernel(D / H);
    TB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    TB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    // 16 CTAs per cluster: half the weight bytes per SM of a cluster of 8, at the price of fewer clusters at a time (7 on a
    // B200 whose processor clusters hold 20, 20, .. 8 SMs).  The sequences are spread over the clusters that fit at once.
    // (A hidden size of 1024 needs the 16: a CTA of eight would own 256 rows of gate|up.  Sizes between were not measured.)
    bool found = false;
    for (int C = 16; C >= 8 && !found; C /= 2) {
        if (!dc_plan(&p, &smem, S, D, H, F, C, 1)) continue;
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = dc_config(p, smem, nullptr, attr);
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1) { cudaGetLastError(); continue; }
        for (int R = std::min(16, ceil_div(S, fit)); R >= 1 && !found; --R) found = dc_plan(&p, &smem, S, D, H, F, C, R);
        if (found && !dc_pays(p, fit)) return 0;
    }
    if (!found) return 0;
    DecodeCluster* m = new DecodeCluster();
    m->p = p;
    m->smem = smem;
    m->p.L = L; m->p.cap = cap; m->p.eps = eps; m->p.inv_d = 1.0f / (float)D; m->p.qscale = scale * 1.4426950408889634f;
    m->p.err = ctx->d_err;
    TB_CUDA(cudaMalloc(&m->wt, (size_t)L * p.C * p.rank_bytes));
    TB_CUDA(cudaMalloc(&m->d_layers, sizeof(DcLayer) * (size_t)L));
    TB_CUDA(cudaMalloc(&m->d_maps, sizeof(CUtensorMap) * 2 * (size_t)L));
    TB_CUDA(cudaMalloc(&m->vec, (size_t)L * p.C * p.vec_floats * sizeof(float)));
    m->p.wt = m->wt; m->p.vec = m->vec;
    m->p.layers = m->d_layers;
    *out = m;
    return 0;
}

void decode_cluster_destroy(DecodeCluster* m) {
    if (!m) return;
    cudaFree(m->wt); cudaFree(m->vec); cudaFree(m->d_layers); cudaFree(m->d_maps);
    delete m;
}

// (Re)builds the operand images of the weights and the per-layer pointer table; call after every weight upload.
int decode_cluster_set_weights(DeviceCtx* ctx, DecodeCluster* m, const float* params, const bf16* params16, const long long* offsets,
                               bf16* const* Kc, bf16* const* Vc, cudaStream_t st) {
    const int D = m->p.D, F = m->p.F, L = m->p.L, H = m->p.H, hd = D / H;
    std::vector<DcLayer> hl((size_t)L);
    std::vector<CUtensorMap> maps(2 * (size_t)L);
    for (int l = 0; l < L; ++l) {
        const long long* o = offsets + 1 + 10LL * l;
        DcLayer& y = hl[l];
        y.Kc = Kc[l]; y.Vc = Vc[l];
        TB_TRY(make_operand_map(&maps[2 * l], Kc[l], hd, m->p.cap, hd, m->p.S * H, (long long)m->p.cap * hd, DC_KV_ROWS));
        TB_TRY(make_operand_map(&maps[2 * l + 1], Vc[l], hd, m->p.cap, hd, m->p.S * H, (long long)m->p.cap * hd, DC_KV_ROWS));
        y.mapK = m->d_maps + 2 * l; y.mapV = m->d_maps + 2 * l + 1;
        uint8_t* w = m->wt + (size_t)l * m->p.C * m->p.rank_bytes;
        auto relayout = [&](const bf16* src, const DcProj& pr, int K, int N, int pair_off) -> int {
            const int pieces = (int)(pr.bytes / 16);
            cluster_layout_kernel<<<dim3(ceil_div(pieces, 256), m->p.C), 256, 0, st>>>(src, w, pr, K, N, m->p.rank_bytes, pair_off);
            TB_CUDA(cudaGetLastError());
            w += pr.bytes;
            return 0;
        };
        TB_TRY(relayout(params16 + o[1], m->p.q, D, 3 * D, 0));
        TB_TRY(relayout(params16 + o[3], m->p.o, D, D, 0));
        TB_TRY(relayout(params16 + o[6], m->p.g, D, 2 * F, F));
        TB_TRY(relayout(params16 + o[8], m->p.d, F, D, 0));
        vec_layout_kernel<<<m->p.C, 256, 0, st>>>(params + o[2], params + o[7], params + o[4], params + o[9], params + o[0], params + o[5],
                                                  m->vec + (size_t)l * m->p.C * m->p.vec_floats, D, F, m->p.q.n, m->p.g.n, m->p.o.n,
                                                  m->p.vec_floats);
        TB_CUDA(cudaGetLastError());
    }
    TB_CUDA(cudaMemcpyAsync(m->d_maps, maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice, st));
    TB_CUDA(cudaMemcpyAsync(m->d_layers, hl.data(), sizeof(DcLayer) * hl.size(), cudaMemcpyHostToDevice, st));
    TB_CUDA(cudaStreamSynchronize(st));              // the host copies go out of scope
    m->p.embed = params;
    m->p.final_norm = params + offsets[1 + 10LL * L];
    return 0;
}

int decode_cluster_clear_values(DeviceCtx* ctx, DecodeCluster* m, int from, int to, cudaStream_t st) {
    if (m->p.embed == nullptr) return 0;       // no weights yet: no step has run
    const DcPlan& p = m->p;
    prof_mark(ctx, "clear_values", 0.0, 2.0 * m->p.L * p.S * p.D * (to - from), st);
    TB_CUDA(launch_kernel(clear_values_kernel, dim3((unsigned)std::min(p.S * p.H, 4 * ctx->sm_count), (unsigned)m->p.L), dim3(128), 0, st,
                          (const DcLayer*)m->d_layers, p.S * p.H, m->p.cap, from, to, p.D / p.H));
    ctx->launches++;
    prof_close(ctx, st);
    return 0;
}

// tok [S] at position *pos -> out [S, D]: the final-norm output of the step, bf16; K and V rows appended to the caches.
int launch_decode_cluster(DeviceCtx* ctx, DecodeCluster* m, const uint32_t* tok, const int* pos, const float* cos_t, const float* sin_t,
                          bf16* out, cudaStream_t st) {
    TB_CHECK(m->p.embed != nullptr, "the decoder has no weights: call tb_decoder_upload first");      // (nor the kernel its tables)
    DcParams p = m->p;
    p.tok = tok; p.pos = pos; p.cos_t = cos_t; p.sin_t = sin_t; p.out = out;
    const DcKernel kernel = dc_kernel(p.D / p.H);
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = dc_config(p, m->smem, st, attr);
    prof_mark(ctx, "decode_layers", 0.0, 0.0, st);
    TB_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    ctx->launches++;
    prof_close(ctx, st);
    return 0;
}

}  // namespace tb
