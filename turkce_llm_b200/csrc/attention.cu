// Fused causal attention for sm_100a: S = Q K^T and O = P V on tcgen05 tensor cores with the
// score tile kept in TMEM, the softmax done in registers and P handed to the second product
// through shared memory -- the [T, T] score and probability matrices never exist in HBM.
//
// Replaces the reference's chain k_bf16_gemm_nt (QK^T) -> k_attn_softmax_fwd -> k_bf16_gemm_nn
// (P V) -> k_heads_merge and its backward counterpart (model/gpu_train.c:346-358, :435-455;
// cuda/train_kernels.cu:631-692), which stores P [B,H,T,T] in float32 per layer.
//
// Semantics are the reference's (model/attention.c:32-60): scores * 1/sqrt(hd), keys after the
// query excluded, softmax over the row, times V.  The reference adds -1e9 to the excluded scores;
// after exp in float32 that is exactly 0, so excluding them is the same function.  The softmax is
// evaluated block-wise with a running maximum (the result is the same softmax; rounding of P to
// bf16 happens against the running maximum instead of the final one).
//
// Layouts: Q, K, V bf16 [B*H, T, hd] (RoPE already applied), hd <= 64 and a multiple of 8 (rows
// are padded to 64 columns with zeros by the TMA loads).  Output bf16 [B*T, H*hd] (heads merged)
// plus the row-wise log-sum-exp, which is all the backward pass needs to rebuild P.
#include "common.h"
#include "ptx.cuh"

#include <algorithm>

#include <cstdlib>

namespace tb {

constexpr int ATT_BM = 128;       // queries per CTA
constexpr int ATT_BN = 128;       // keys per step
constexpr int ATT_HD = 64;        // padded head dimension
constexpr int TILE_BYTES = 128 * 64 * 2;   // one [128, 64] bf16 tile, 128-byte rows

// Shared-memory descriptors are built once per tile, outside the issue loops (one thread issues every
// UMMA of the CTA, so each instruction it spends per UMMA delays the tensor pipe); the loops only add
// to the start-address field (low 14 bits, 16-byte units; never carries below 256 KB).
// K-major operand tile [rows, 64] (128-byte rows, 128B swizzle): advance 32 bytes per K=16
__device__ __forceinline__ uint64_t kmajor_tile(uint32_t tile_addr) { return umma_desc_sw128(tile_addr, 16, 1024); }
// the same tile read as an MN-major operand (64 MN elements contiguous, K = rows): 16 rows per K=16;
// lbo = bytes between consecutive 64-wide MN blocks
__device__ __forceinline__ uint64_t mnmajor_tile(uint32_t tile_addr, uint32_t lbo) {
    return umma_desc_sw128(tile_addr, lbo, 1024);
}
constexpr uint64_t KSTEP = 32 >> 4;          // descriptor units per K=16 step of a K-major tile
constexpr uint64_t MNSTEP = 2048 >> 4;       // ... of an MN-major tile (16 rows of 128 bytes)
constexpr uint64_t TILESTEP = (128 * 64 * 2) >> 4;   // one [128, 64] bf16 tile

// 2^x on the special-function unit (one instruction; 2^-inf = 0)
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two float32 results per issue slot (fma.rn.f32x2 and friends, sm_100): the softmax warps of these kernels are
// bound by instruction issue (about 2,000 cycles per 128 x 128 block for 64 scores per thread), not by a unit.
__device__ __forceinline__ float2 pair_of(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }


struct AttFwdParams {
    int T, H, hd, D;
    int nq;                 // query blocks per head
    float scale_log2;       // 1/sqrt(hd) * log2(e)
    bf16* att;              // [B*T, D]
    float* lse;             // [B*H, T]
    int* err;
};

// ------------------------------------------------------------------------------------ forward
// CTA = 10 warps: TMA producer, MMA issuer (owns TMEM), and two groups of four softmax warps (thread = query row).  Keys are
// taken in half blocks of 64: group b takes the half blocks of parity b, with a score buffer, a probability buffer, a running
// maximum, a sum and an output accumulator of its own; the two are put together at the end.  While a group works on its half
// block, the tensor core forms the scores of its next one (the buffer is free as soon as the scores are in registers) and
// adds P V of its last one.  Two CTAs fit per SM on top of that.
// A half block is a chain of score load, maximum, exponentials, stores and a round trip through the tensor core, ~2,500 clocks
// for 512 of the 2^x unit, so what counts is the number of chains side by side: with one group per CTA (two warps per
// scheduler) and the output sums in registers 16 x 6 heads x 1024 took 36.2 us, 5 x 6 x 777 16.2; now 31.2 and 14.0.
// The running output stays in tensor memory and is read, rescaled and written back where the maximum of one of a warp's rows has
// grown.  The exponentials are always taken against the maximum so far, so that the largest probability of a row is 1 and exact
// in bf16: taken against an older maximum (rescaling only at a growth of 2^8) that one is rounded like the others, and where a
// row has one or a few keys that matter the output is further off (2-norm against float64, 16 x 6 heads x 1024: 1.99e-3 instead
// of 1.71e-3 with q four times as large, 2.02e-3 instead of 1.98e-3 as it is; 29.6 us instead of 31.2).

constexpr int ATT_FWD_THREADS = 320;
__global__ void __launch_bounds__(ATT_FWD_THREADS, 2)
attention_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                     const AttFwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    uint8_t* sQ = smem;                          // 16 KB
    uint8_t* sK = smem + TILE_BYTES;             // 2 x 16 KB
    uint8_t* sV = smem + 3 * TILE_BYTES;         // 2 x 16 KB
    uint8_t* sP = smem + 5 * TILE_BYTES;         // 2 x 16 KB: keys 0-63 | keys 64-127
    // the request is exactly 1 KB + 7 tiles (two CTAs per SM): the barriers go behind the tiles when
    // the alignment pad leaves room there (the usual case: pad 0), else into the pad itself
    const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    uint64_t* bars = reinterpret_cast<uint64_t*>(pad <= 768u ? smem + 7 * TILE_BYTES : smem_raw);
    uint64_t* q_full = bars;          // 1
    uint64_t* k_full = bars + 1;      // 2: K tile of 128 keys in stage s
    uint64_t* v_full = bars + 3;      // 2
    uint64_t* kv_empty = bars + 5;    // 2
    uint64_t* s_full = bars + 7;      // 2: score buffer b holds Q K^T of a 64-key half block
    uint64_t* s_free = bars + 9;      // 2
    uint64_t* p_full = bars + 11;     // 2: probability buffer b written
    uint64_t* o_full = bars + 13;     // 2: P V of a half block of parity b has been added to its accumulator
    uint64_t* out_full = bars + 18;   // 8 arrivals: the output tile is staged in shared memory
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // blocks are handed out x fastest: all heads' heaviest (last) query block first, the lightest last,
    // so the long CTAs start together and the short ones fill the tail
    const int qb = p.nq - 1 - (int)blockIdx.y;
    const int bh = blockIdx.x;
    const int q0 = qb * ATT_BM;
    const int nkv = qb + 1;                           // key blocks 0..qb

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&v_full[i], 1); mbar_init(&kv_empty[i], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1); mbar_init(&s_free[i], 4); mbar_init(&p_full[i], 4);
            mbar_init(&o_full[i], 1);
        }
        mbar_init(out_full, 8);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();                 // everything above is independent of earlier kernels' results
    // TMEM: two score buffers of 64 key columns, two output accumulators of 64 head-dim columns
    const uint32_t tS = tmem_base, tO = tmem_base + 128;
    const int nsub = 2 * nkv;                         // 64-key half blocks

    if (warp == 0) {
        if (elect_one()) {
            bool ok = true;
            mbar_expect_tx(q_full, TILE_BYTES);
            tma_load_3d(sQ, &tmQ, q_full, 0, q0, bh);
            for (int j = 0; j < nkv && ok; ++j) {
                const int s = j & 1;
                if (!mbar_wait(&kv_empty[s], (uint32_t)((j >> 1) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                mbar_expect_tx(&k_full[s], TILE_BYTES);
                tma_load_3d(sK + s * TILE_BYTES, &tmK, &k_full[s], 0, j * ATT_BN, bh);
                mbar_expect_tx(&v_full[s], TILE_BYTES);
                tma_load_3d(sV + s * TILE_BYTES, &tmV, &v_full[s], 0, j * ATT_BN, bh);
            }
            pdl_launch_dependents_now();     // all loads issued: the next kernel may start its prologue
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 11); }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // the scores of half block i+2 are issued as soon as its group has drained the buffer, while it works on i
            const uint32_t idesc_s = umma_idesc(1u, 0u, 0u, ATT_BM, 64);         // Q K^T: both K-major
            const uint32_t idesc_o = umma_idesc(1u, 0u, 1u, ATT_BM, ATT_HD);     // P V: V is MN-major
            const uint64_t dQ = kmajor_tile(smem_u32(sQ)), dK0 = kmajor_tile(smem_u32(sK)), dP0 = kmajor_tile(smem_u32(sP));
            const uint64_t dV0 = mnmajor_tile(smem_u32(sV), TILE_BYTES);
            bool ok = mbar_wait(q_full, 0, abort_flag);
            auto issue_scores = [&](int i) -> bool {
                const int j = i >> 1, st = j & 1, b = i & 1;
                if (b == 0 && !mbar_wait(&k_full[st], (uint32_t)((j >> 1) & 1), abort_flag)) return false;
                if (!mbar_wait(&s_free[b], (uint32_t)((i >> 1) & 1) ^ 1u, abort_flag)) return false;
                tc_fence_after();
                const uint64_t dK = dK0 + (uint64_t)st * TILESTEP + (uint64_t)b * (TILESTEP / 2);   // keys 64b.. of the tile
#pragma unroll
                for (int k = 0; k < ATT_HD / 16; ++k)
                    umma_bf16(tS + (uint32_t)(b * 64), dQ + k * KSTEP, dK + k * KSTEP, idesc_s, k > 0 ? 1u : 0u);
                umma_commit(&s_full[b]);
                return true;
            };
            if (ok) ok = issue_scores(0);
            if (ok && nsub > 1) ok = issue_scores(1);
            for (int i = 0; i < nsub && ok; ++i) {
                const int j = i >> 1, st = j & 1, b = i & 1;
                const uint32_t par = (uint32_t)((i >> 1) & 1);
                if (i + 2 < nsub && !issue_scores(i + 2)) { ok = false; break; }
                if (!mbar_wait(&p_full[b], par, abort_flag)) { ok = false; break; }
                if (b == 0 && !mbar_wait(&v_full[st], (uint32_t)((j >> 1) & 1), abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t dP = dP0 + (uint64_t)b * TILESTEP;
                const uint64_t dV = dV0 + (uint64_t)st * TILESTEP + (uint64_t)b * (4 * MNSTEP);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_bf16(tO + (uint32_t)(b * 64), dP + k * KSTEP, dV + k * MNSTEP, idesc_o, (i > 1 || k > 0) ? 1u : 0u);
                umma_commit(&o_full[b]);
                if (b == 1) umma_commit(&kv_empty[st]);          // both halves of the K/V tile are consumed
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 12); }
        }
    } else {
        const int q = warp & 3;
        const int b = (warp - 2) >> 2;               // this group's half blocks: i = b, b + 2, ..
        const int r = q * 32 + lane;                 // row of the tile = TMEM lane
        const int qi = q0 + r;                       // query position
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const uint32_t ts = tS + lane_base + (uint32_t)(b * 64), to = tO + lane_base + (uint32_t)(b * 64);
        float m = -INFINITY, l = 0.0f;               // the maximum the exponentials are taken against, and their sum
        bool ok = true;
        uint32_t v[2][32];                           // one half block's scores (or the accumulators) of this row
        for (int j = 0; j < nkv && ok; ++j) {
            if (!mbar_wait(&s_full[b], (uint32_t)(j & 1), abort_flag)) { ok = false; break; }
            tc_fence_after();
            // all 64 scores of the row in one TMEM round trip, then the buffer is free
            tmem_ld32(ts, v[0]);
            tmem_ld32(ts + 32, v[1]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[b]);
            const bool diag = j == qb;
            const int lim = diag ? r - b * 64 : 64;            // columns e <= lim are allowed
            float mx = -INFINITY;
            if (diag) {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    mx = fmaxf(mx, e <= lim ? __uint_as_float(v[0][e]) : -INFINITY);
                    mx = fmaxf(mx, e + 32 <= lim ? __uint_as_float(v[1][e]) : -INFINITY);
                }
            } else {
                // four chains instead of one of 32 dependent maxima
                float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
                for (int e = 0; e < 32; e += 4) {
                    m0 = fmaxf(m0, fmaxf(__uint_as_float(v[0][e]), __uint_as_float(v[1][e])));
                    m1 = fmaxf(m1, fmaxf(__uint_as_float(v[0][e + 1]), __uint_as_float(v[1][e + 1])));
                    m2 = fmaxf(m2, fmaxf(__uint_as_float(v[0][e + 2]), __uint_as_float(v[1][e + 2])));
                    m3 = fmaxf(m3, fmaxf(__uint_as_float(v[0][e + 3]), __uint_as_float(v[1][e + 3])));
                }
                mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
            }
            const float m_new = fmaxf(m, mx * p.scale_log2);
            float alpha = 1.0f;
            if (m_new > m) {                                 // (each row for itself: a row does not depend on its neighbours)
                alpha = fast_exp2(m - m_new);                // 0 on the first block (m = -inf)
                l *= alpha;
                m = m_new;
            }
            const bool move = __any_sync(0xffffffffu, alpha != 1.0f);
            // the group's last probabilities have been multiplied: their buffer is free and the accumulator is complete
            if (j > 0 && !mbar_wait(&o_full[b], (uint32_t)((j - 1) & 1), abort_flag)) { ok = false; break; }
            // p = 2^(s*c - m), row sum, bf16 P into shared memory (K-major, 128B swizzle)
            const float2 c2 = make_float2(p.scale_log2, p.scale_log2), nm2 = make_float2(-m, -m);
            float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            uint8_t* prow = sP + b * TILE_BYTES + r * 128;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    uint32_t w[4];
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const int e = 8 * g + 2 * h;
                        const float2 x = __ffma2_rn(pair_of(v[c][e], v[c][e + 1]), c2, nm2);
                        float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                        if (diag) {
                            pr.x = e + 32 * c <= lim ? pr.x : 0.0f;
                            pr.y = e + 1 + 32 * c <= lim ? pr.y : 0.0f;
                        }
                        ls[h & 1] = __fadd2_rn(ls[h & 1], pr);
                        __nv_bfloat162 hp = __floats2bfloat162_rn(pr.x, pr.y);
                        w[h] = *reinterpret_cast<uint32_t*>(&hp);
                    }
                    *reinterpret_cast<uint4*>(prow + (((4 * c + g) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            l += (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y);
            if (move && j > 0) {
                // P V so far, against the old maximum
                tc_fence_after();
#pragma unroll
                for (int h2 = 0; h2 < 2; ++h2) {
                    tmem_ld32(to + (uint32_t)(h2 * 32), v[0]);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[0][e] = __float_as_uint(__uint_as_float(v[0][e]) * alpha);
                    tmem_st32(to + (uint32_t)(h2 * 32), v[0]);
                }
                tmem_st_wait();
            }
            tc_fence_before();
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[b]);
        }
        // every product has completed (in this order: a group is at most one half block behind the other); the probability
        // tiles then hold the groups' maxima and sums
        if (ok) ok = mbar_wait(&o_full[0], (uint32_t)((nkv - 1) & 1), abort_flag) && mbar_wait(&o_full[1], (uint32_t)((nkv - 1) & 1), abort_flag);
        float2* stat = reinterpret_cast<float2*>(sP);
        if (ok) stat[b * ATT_BM + r] = make_float2(m, l);
        asm volatile("bar.sync 1, 256;" ::: "memory");       // (a thread whose wait gave up comes here as well)
        if (ok) {
            // head-dim columns 32 b .. of O = (O_0 2^(m_0 - M) + O_1 2^(m_1 - M)) / l.  (m_0 is finite: key 0 is allowed.)
            tc_fence_after();
            tmem_ld32(tO + lane_base + (uint32_t)(b * 32), v[0]);
            tmem_ld32(tO + lane_base + 64u + (uint32_t)(b * 32), v[1]);
            const float2 s0 = stat[r], s1 = stat[ATT_BM + r];
            const float M = fmaxf(s0.x, s1.x), e0 = fast_exp2(s0.x - M), e1 = fast_exp2(s1.x - M);
            const float lt = s0.y * e0 + s1.y * e1, inv = 1.0f / lt;
            const float w0 = e0 * inv, w1 = e1 * inv;
            tmem_ld_wait();
            // as bf16 into the Q tile, one TMA store for the 128 rows: a thread per row storing to global memory directly
            // touches 32 different rows per instruction
            if (qi < p.T) {
                uint8_t* row = sQ + r * 128;
#pragma unroll
                for (int d = 0; d < 32; d += 8) {
                    if (32 * b + d >= p.hd) break;
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int c = d + 2 * e;
                        __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(v[0][c]) * w0 + __uint_as_float(v[1][c]) * w1,
                                                                  __uint_as_float(v[0][c + 1]) * w0 + __uint_as_float(v[1][c + 1]) * w1);
                        w[e] = *reinterpret_cast<uint32_t*>(&h2);
                    }
                    *reinterpret_cast<uint4*>(row + (((4 * b + (d >> 3)) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                if (p.lse && b == 0) p.lse[(long long)bh * p.T + qi] = (M + log2f(lt)) * 0.6931471805599453f;
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(out_full);
            if (warp == 2 && lane == 0) {
                if (mbar_wait(out_full, 0, abort_flag)) {
                    tma_store_4d(&tmO, sQ, 0, q0, bh % p.H, bh / p.H);          // rows past T are clipped
                    tma_store_commit();
                    tma_store_wait_read<0>();
                } else ok = false;
            }
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 13); }
    }

    __syncwarp();
    if (*abort_flag) for (int i = 0; i < 64; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

// ----------------------------------------------------------------------------------- backward
// With P rebuilt from the saved log-sum-exp (P = exp(S*scale - lse)) the backward is, per head,
//   dV = P^T dO,  dP = dO V^T,  dS = P * (dP - delta) * scale,  dQ = dS K,  dK = dS^T Q,
// delta[i] = <dO_i, O_i>  (the reference's k_attn_softmax_bwd row dot <dP, P>, since O = P V).
// Two kernels keep every sum in a fixed order without atomics: one owns a key block and walks the
// query blocks below the diagonal (dK, dV), the other owns a query block and walks its key blocks (dQ).
// Sequences of one block take one kernel (attention_bwd_one_block_kernel).

// <a, b> of eight values from o on, and the sum over a group of eight lanes
__device__ __forceinline__ float dot8(const bf16* __restrict__ a, const bf16* __restrict__ b, long long o) {
    const uint4 av = *reinterpret_cast<const uint4*>(a + o), bv = *reinterpret_cast<const uint4*>(b + o);
    const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&av);
    const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&bv);
    float s = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 x = __bfloat1622float2(a2[e]), y = __bfloat1622float2(b2[e]);
        s += x.x * y.x;
        s += x.y * y.y;
    }
    return s;
}
__device__ __forceinline__ float sum8(float s) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// delta of row (b, h, t): eight lanes per row, 16 bytes each, so that a warp reads four adjacent heads' pieces of a token (a
// thread per row read 32 different 128-byte rows per instruction; 8 x 6 x 1024 under ncu, cold: 9.8 us, this 7.2).
__global__ void attention_delta_kernel(const bf16* __restrict__ att, const bf16* __restrict__ datt,
                                       float* __restrict__ delta, int B, int T, int H, int hd) {
    pdl_wait();
    pdl_launch_dependents();
    const long long total = (long long)B * T * H;
    const int D = H * hd, piece = threadIdx.x & 7;
    const bool mine = piece * 8 < hd;
    // (whole groups of eight lanes go round the loop together, and a warp's groups leave it together: the bound is rounded up)
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3; i < ((total + 3) & ~3LL); i += (gridDim.x * blockDim.x) >> 3) {
        const long long n = total < (1LL << 31) ? (long long)((unsigned)i / (unsigned)H) : i / H;
        const int h = (int)(i - n * H);
        float s = 0.0f;
        if (mine && i < total) {
            const long long o = n * D + h * hd + piece * 8;
            s = dot8(att, datt, o);
        }
        s = sum8(s);
        if (piece == 0 && i < total) {
            const long long b = total < (1LL << 31) ? (long long)((unsigned)n / (unsigned)T) : n / T;
            delta[(b * H + h) * T + (n - b * T)] = s;
        }
    }
}

// ---- work items of the two gradient kernels
// An item is one (key or query block, head); the grid has a CTA per item, heaviest first, all heads of a block adjacent.  A CTA
// that has started takes over items whose CTAs have not (cluster launch control), so that the next item's loads lie under
// this one's work, and SMs that another kernel still holds simply take no part.  The next item is asked for with the last
// block's loads: a CTA that asks at its start takes items from SMs that are still empty (5 x 6 heads x 777: 31 us against 26).
// One thread asks for the items and hands them to the roles of the CTA through a ring of four; -1 ends the CTA.
constexpr int ITEM_RING = 4;
struct ItemRing {
    uint64_t *full, *empty, *answered;      // [ITEM_RING], [ITEM_RING], 1
    volatile int* items;                    // [ITEM_RING]
    uint8_t* answer;                        // 16 bytes, 16-byte aligned
};
__device__ __forceinline__ ItemRing item_ring(uint8_t* mem) {       // 104 bytes
    ItemRing r;
    r.answer = mem;
    r.full = reinterpret_cast<uint64_t*>(mem + 16);
    r.empty = r.full + ITEM_RING;
    r.answered = r.empty + ITEM_RING;
    r.items = reinterpret_cast<volatile int*>(r.answered + 1);
    return r;
}
__device__ __forceinline__ void item_ring_init(const ItemRing& r, uint32_t takers) {
    for (int i = 0; i < ITEM_RING; ++i) { mbar_init(&r.full[i], 1); mbar_init(&r.empty[i], takers); }
    mbar_init(r.answered, 1);
}
// the asking thread: item k for everybody
__device__ __forceinline__ bool item_put(const ItemRing& r, int k, int item, volatile int* abort_flag) {
    const int s = k % ITEM_RING;
    if (!mbar_wait(&r.empty[s], (uint32_t)((k / ITEM_RING) & 1) ^ 1u, abort_flag)) return false;
    r.items[s] = item;
    mbar_arrive(&r.full[s]);
    return true;
}
// everybody else: item k, or -1 (also when a wait gave up: the abort flag is up then).  A warp takes it with all lanes.
__device__ __forceinline__ int item_get(const ItemRing& r, int k, bool one_thread, volatile int* abort_flag) {
    const int s = k % ITEM_RING;
    if (!mbar_wait(&r.full[s], (uint32_t)((k / ITEM_RING) & 1), abort_flag)) { *abort_flag = 1; return -1; }
    const int item = r.items[s];
    if (!one_thread) __syncwarp();
    if (one_thread || (threadIdx.x & 31) == 0) mbar_arrive(&r.empty[s]);
    return item;
}
// asks for a CTA that has not started ..
__device__ __forceinline__ void item_ask(const ItemRing& r) {
    fence_proxy_async();                                 // (the last answer was read by ordinary loads)
    mbar_expect_tx(r.answered, 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(smem_u32(r.answer)), "r"(smem_u32(r.answered)) : "memory");
}
// .. and the answer to request number k: its index, or -1 when all have started (nothing is asked after that)
__device__ __forceinline__ int item_answer(const ItemRing& r, int k, volatile int* abort_flag) {
    if (!mbar_wait(r.answered, (uint32_t)(k & 1), abort_flag)) { *abort_flag = 1; return -1; }
    uint32_t got, x;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
        "ld.shared.b128 h, [%2];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
        "selp.b32 %0, 1, 0, p;\n\tmov.b32 %1, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
        : "=r"(got), "=r"(x) : "r"(smem_u32(r.answer)) : "memory");
    return got ? (int)x : -1;
}
// items = rounds of BH heads: i / BH by multiplication with ceil(2^32 / BH) where that is exact (magic != 0; a division by a
// run-time value is ~150 clocks in front of an item's first load)
__device__ __forceinline__ int att_round(int i, int BH, unsigned magic) {
    return magic ? (int)__umulhi((unsigned)i, magic) : i / BH;
}
inline unsigned att_magic(long long BH, long long items) {
    return (BH > 1 && BH * items < (1LL << 32)) ? (unsigned)(((1ULL << 32) + BH - 1) / BH) : 0u;
}

struct AttBwdParams {
    int T, H, hd;
    int nq;
    int BH;                 // heads of all sequences; work items = BH * nq
    unsigned bh_magic;
    float scale, scale_log2;
    const float* lse;       // [B*H, T]
    float* delta;           // [B*H, T]
    const bf16 *att, *datt; // [B*T, H*hd]
    float* dQ; float* dK; float* dV;     // [B*H, T, hd]
    // merged output (optional, replaces dQ/dK/dV): dqkv bf16 [B*T, 3*H*hd] with the inverse rotation of
    // the position embedding applied to dQ and dK on the way out (the reference's k_qkv_rope_merge_bwd,
    // cuda/train_kernels.cu:600-626); cos_t/sin_t are the [T, hd/2] tables
    bf16* dqkv; const float* cos_t; const float* sin_t;
    // dS hand-off between the two kernels: the dK/dV kernel stores each [128 q x 128 keys] block of dS' = P * (dP - delta)
    // (bf16, the 32 KB shared-memory image it feeds its own tensor-core product with) at block index
    // bh * nq*(nq+1)/2 + qb*(qb+1)/2 + kb; the dQ kernel reads the blocks back and only forms dQ = sum_kb dS' K.
    // (Recomputing S, dP and the exponentials there instead cost a second pass over the 2^x unit, the busiest one.)
    bf16* ds;
    int* err;
};
constexpr int DS_BLOCK_BYTES = 2 * TILE_BYTES;

// The rotation tables of one row for 32 consecutive head-dim values (16 pairs) starting at d0: fetched before the
// wait for the accumulators, in one batch (loads placed between the stores of a row would each wait for the
// store before them, since the compiler cannot tell the tables from the output).
struct RopeRow { float4 c[4], s[4]; };
__device__ __forceinline__ void load_rope_row(RopeRow& t, const float* cs, const float* sn, int d0, int hd) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        if (d0 + 8 * g < hd) {
            t.c[g] = *reinterpret_cast<const float4*>(cs + ((d0 + 8 * g) >> 1));
            t.s[g] = *reinterpret_cast<const float4*>(sn + ((d0 + 8 * g) >> 1));
        } else {
            t.c[g] = make_float4(1.f, 1.f, 1.f, 1.f);
            t.s[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

// 32 consecutive head-dim values of one row (first index d0), times mul, optionally through the inverse rotation of
// the interleaved pairs (2k, 2k+1): out = (a*c + b*s, -a*s + b*c), as bf16 into row r of a [128 x 64] tile in shared
// memory (128-byte rows, 128B swizzle), from where one TMA store writes the whole tile: a thread per row storing to global memory directly touches 32 different
// rows per instruction (one 16-byte piece each), which took ~4,500 cycles per CTA.
__device__ __forceinline__ void stage_row_bf16(uint8_t* tile, int r, const uint32_t (&v)[32], int d0, int hd,
                                               const RopeRow* rot, float mul) {
    uint8_t* row = tile + r * 128;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const int e = 8 * g;
        if (d0 + e >= hd) break;
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(v[e + j]) * mul;
        if (rot != nullptr) {
            const float4 c4 = rot->c[g], s4 = rot->s[g];
            const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float a = o[2 * j], b = o[2 * j + 1];
                o[2 * j] = a * cc[j] + b * ss[j];
                o[2 * j + 1] = -a * ss[j] + b * cc[j];
            }
        }
        uint4 pk;
        __nv_bfloat162 h0 = __floats2bfloat162_rn(o[0], o[1]), h1 = __floats2bfloat162_rn(o[2], o[3]);
        __nv_bfloat162 h2 = __floats2bfloat162_rn(o[4], o[5]), h3 = __floats2bfloat162_rn(o[6], o[7]);
        pk.x = *reinterpret_cast<uint32_t*>(&h0); pk.y = *reinterpret_cast<uint32_t*>(&h1);
        pk.z = *reinterpret_cast<uint32_t*>(&h2); pk.w = *reinterpret_cast<uint32_t*>(&h3);
        const int chunk = (d0 >> 3) + g;
        *reinterpret_cast<uint4*>(row + ((chunk ^ (r & 7)) << 4)) = pk;
    }
}

// 32 float32 values times mul into row r of a [128 x 32] float32 tile (128-byte rows, 128B swizzle) for a TMA store
__device__ __forceinline__ void stage_row_f32(uint8_t* tile, int r, const uint32_t (&v)[32], float mul) {
    uint8_t* row = tile + r * 128;
#pragma unroll
    for (int g = 0; g < 8; ++g)
        *reinterpret_cast<float4*>(row + ((g ^ (r & 7)) << 4)) =
            make_float4(__uint_as_float(v[4 * g]) * mul, __uint_as_float(v[4 * g + 1]) * mul,
                        __uint_as_float(v[4 * g + 2]) * mul, __uint_as_float(v[4 * g + 3]) * mul);
}

// P = 2^(s*c - lse) and dS' = P * (dP - delta) of scores E0 .. E0 + 15 of one row, two per instruction, as 16 bf16 each.  The
// factor 1/sqrt(hd) of dS is applied to the accumulated dQ and dK instead (they are linear in dS).  lim: columns e <= lim are
// allowed.
template <int E0>
__device__ __forceinline__ void p_and_ds16(const uint32_t (&sv)[32], const uint32_t (&dv)[32], float scale_log2, float lse2,
                                           float dl, bool diag, int lim, uint4 (&pP)[2], uint4 (&pD)[2]) {
    const float2 c2 = make_float2(scale_log2, scale_log2), nl2 = make_float2(-lse2, -lse2), nd2 = make_float2(-dl, -dl);
    uint32_t wp[8], wd[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = E0 + 2 * i;
        const float2 x = __ffma2_rn(pair_of(sv[e], sv[e + 1]), c2, nl2);
        float p0 = fast_exp2(x.x), p1 = fast_exp2(x.y);
        if (diag) { p0 = e <= lim ? p0 : 0.0f; p1 = e + 1 <= lim ? p1 : 0.0f; }
        const float2 d = __fmul2_rn(make_float2(p0, p1), __fadd2_rn(pair_of(dv[e], dv[e + 1]), nd2));
        __nv_bfloat162 hp = __floats2bfloat162_rn(p0, p1), hd = __floats2bfloat162_rn(d.x, d.y);
        wp[i] = *reinterpret_cast<uint32_t*>(&hp);
        wd[i] = *reinterpret_cast<uint32_t*>(&hd);
    }
    pP[0] = make_uint4(wp[0], wp[1], wp[2], wp[3]); pP[1] = make_uint4(wp[4], wp[5], wp[6], wp[7]);
    pD[0] = make_uint4(wd[0], wd[1], wd[2], wd[3]); pD[1] = make_uint4(wd[4], wd[5], wd[6], wd[7]);
}

// 16 bf16 of row r, columns 32 c + 16 h .., into a [128 x 128] operand stored as two [128 x 64] tiles
__device__ __forceinline__ void store_half_chunk(uint8_t* tiles, int r, int c, int h, const uint4 (&v)[2]) {
    uint8_t* row = tiles + (c >> 1) * TILE_BYTES + r * 128;
#pragma unroll
    for (int i = 0; i < 2; ++i) *reinterpret_cast<uint4*>(row + ((((c & 1) * 4 + h * 2 + i) ^ (r & 7)) << 4)) = v[i];
}

constexpr int ATT_BWD_STAGES = 3;       // stages of the (Q, dO) pair in the dK/dV kernel
constexpr int ATT_BWD_CW = 16;          // compute warps
// Barriers that say "the dK products of block g have read dS'", in turn.  The store thread lets block g + 1 go on (w_free)
// before it waits for block g, so at an item's boundary two more blocks can end before it has looked, and with one barrier it
// would take the second one's phase for its own and wait until its limit.  It holds up the third block, so two are enough.
constexpr int ATT_DS_FREE = 2;
constexpr int ATT_BWD_THREADS = 128 + 32 * ATT_BWD_CW;      // + TMA warp, score-MMA warp, gradient-MMA warp, store warp
// (two issuing threads on different schedulers: one thread cannot issue a block's 24 UMMAs as fast as the
//  tensor pipe retires them while the compute warps compete for the same issue slots)

// dK, dV of key blocks: an item is one key block of one head, walking the query blocks qb = kb .. nq-1; a CTA works through
// several items (early key blocks, which have the most query blocks, first).
// What bounds it (16 x 6 heads x 1024, a block = 128 queries x 128 keys): 1,024 clocks of 2^x per block (16,384 at 16 a clock),
// 512 of shared-memory writes of P and dS' (64 KB at 128 bytes a clock), ~1,100 from the signal that P is written to the end
// of the gradient products, and what an item costs outside its loop.  (The clocks that are not counts are from stamps of a
// throw-away build.)  Hence
//  * sixteen compute warps of 32 key columns (with eight of 64 the chain of one warp took 2,240 clocks a block);
//  * P is free again after the dV products, which come first, and half of a block's exponentials come behind the stores of
//    the first half;
//  * dS' blocks leave through a thread of their own (reading 32 KB out takes 1,400 clocks, a third of a block's time when the
//    gradient thread waited for it), three stages of Q and dO cover the loads (2,000 clocks under load);
//  * with a CTA per item the set-up, the first loads and the epilogue took 4.3 us against 1.2 per block; now the next
//    item's K, V, Q and dO come in, and its first scores are formed, under the last block and the epilogue of the one before.
__global__ void __launch_bounds__(ATT_BWD_THREADS, 1)
attention_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                          const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                          const __grid_constant__ CUtensorMap tmoK, const __grid_constant__ CUtensorMap tmoV,
                          const AttBwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    uint8_t* sK = smem;
    uint8_t* sV = smem + TILE_BYTES;
    uint8_t* sQ = smem + 2 * TILE_BYTES;                              // ATT_BWD_STAGES stages
    uint8_t* sdO = smem + (2 + ATT_BWD_STAGES) * TILE_BYTES;          // ATT_BWD_STAGES stages
    uint8_t* sP = smem + (2 + 2 * ATT_BWD_STAGES) * TILE_BYTES;       // [128 q, 128 keys] as two tiles
    uint8_t* sdS = smem + (4 + 2 * ATT_BWD_STAGES) * TILE_BYTES;      // same, two buffers (one is being stored)
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (8 + 2 * ATT_BWD_STAGES) * TILE_BYTES);
    uint64_t* kv_full = bars;
    uint64_t* kv_empty = bars + 1;
    uint64_t* qdo_full = bars + 2;     // ATT_BWD_STAGES
    uint64_t* qdo_empty = bars + 6;    // ATT_BWD_STAGES
    uint64_t* sdp_full = bars + 10;
    uint64_t* sdp_free = bars + 11;    // one arrival per compute warp
    uint64_t* pds_full = bars + 12;    // one arrival per compute warp
    uint64_t* w_free = bars + 13;      // 2 arrivals: block g's dV products have read P, block g - 1's dS buffer has been read out
    uint64_t* ds_free = bars + 14;     // ATT_DS_FREE
    uint64_t* acc_full = bars + 14 + ATT_DS_FREE;    // an item's last products are done
    uint64_t* out_full = bars + 17;    // one arrival per compute warp: an item's output tiles are staged
    uint64_t* out_done = bars + 18;    // the store has read them
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const ItemRing ring = item_ring(reinterpret_cast<uint8_t*>(bars + 20));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Blocks are counted through all items of the CTA (g); item k has nq - kb of them.

    if (threadIdx.x == 0) {
        for (int i = 0; i < 19; ++i) mbar_init(&bars[i], (i == 11 || i == 12 || i == 17) ? ATT_BWD_CW : i == 13 ? 2 : 1);
        item_ring_init(ring, 3 + ATT_BWD_CW);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();                 // everything above is independent of earlier kernels' results
    const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 320;

    if (warp == 0) {
        if (elect_one()) {
            bool ok = true;
            int g = 0;
            for (int k = 0, item = (int)blockIdx.x; ok; ++k) {
                if (!item_put(ring, k, item, abort_flag)) { ok = false; break; }
                if (item < 0) break;
                const int kb = att_round(item, p.BH, p.bh_magic), bh = item - kb * p.BH, b = bh / p.H, h = bh % p.H;
                for (int qb = kb; qb < p.nq; ++qb, ++g) {
                    const int s = g % ATT_BWD_STAGES;
                    if (qb == p.nq - 1) item_ask(ring);
                    if (!mbar_wait(&qdo_empty[s], (uint32_t)((g / ATT_BWD_STAGES) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                    mbar_expect_tx(&qdo_full[s], 2 * TILE_BYTES);
                    tma_load_3d(sQ + s * TILE_BYTES, &tmQ, &qdo_full[s], 0, qb * ATT_BM, bh);
                    tma_load_4d(sdO + s * TILE_BYTES, &tmdO, &qdo_full[s], 0, qb * ATT_BM, h, b);
                    if (qb == kb) {             // (behind the first Q and dO, for which there may be room earlier)
                        if (!mbar_wait(kv_empty, (uint32_t)(k & 1) ^ 1u, abort_flag)) { ok = false; break; }
                        mbar_expect_tx(kv_full, 2 * TILE_BYTES);
                        tma_load_3d(sK, &tmK, kv_full, 0, kb * ATT_BN, bh);
                        tma_load_3d(sV, &tmV, kv_full, 0, kb * ATT_BN, bh);
                    }
                }
                if (ok) item = item_answer(ring, k, abort_flag);
            }
            pdl_launch_dependents_now();     // all loads issued: the next kernel may start its prologue
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 21); }
        }
    } else if (warp == 1) {
        // S = Q K^T and dP = dO V^T of every block; may run ahead of the gradient products because the compute warps free
        // the two score tiles as soon as they hold them in registers
        if (elect_one()) {
            const uint32_t id_s = umma_idesc(1u, 0u, 0u, 128, 128);
            const uint64_t dKk = kmajor_tile(smem_u32(sK)), dVk = kmajor_tile(smem_u32(sV));
            const uint64_t dQk0 = kmajor_tile(smem_u32(sQ)), ddOk0 = kmajor_tile(smem_u32(sdO));
            bool ok = true;
            int g = 0;
            for (int k = 0, item; ok && (item = item_get(ring, k, true, abort_flag)) >= 0; ++k) {
                const int n = p.nq - att_round(item, p.BH, p.bh_magic);
                if (!mbar_wait(kv_full, (uint32_t)(k & 1), abort_flag)) { ok = false; break; }
                for (int it = 0; it < n; ++it, ++g) {
                    const int s = g % ATT_BWD_STAGES;
                    const uint64_t dQk = dQk0 + (uint64_t)s * TILESTEP, ddOk = ddOk0 + (uint64_t)s * TILESTEP;
                    if (!mbar_wait(&qdo_full[s], (uint32_t)((g / ATT_BWD_STAGES) & 1), abort_flag)) { ok = false; break; }
                    if (!mbar_wait(sdp_free, (uint32_t)(g & 1) ^ 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_bf16(tS, dQk + j * KSTEP, dKk + j * KSTEP, id_s, j > 0 ? 1u : 0u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_bf16(tdP, ddOk + j * KSTEP, dVk + j * KSTEP, id_s, j > 0 ? 1u : 0u);
                    umma_commit(sdp_full);
                }
                if (ok) umma_commit(kv_empty);
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 22); }
        }
    } else if (warp == 2 + ATT_BWD_CW) {
        // second issuer: dV += P^T dO and dK += dS^T Q once the compute warps have written P and dS
        if (elect_one()) {
            const uint32_t id_t = umma_idesc(1u, 1u, 1u, 128, 64);       // both operands MN-major
            const uint64_t dPm = mnmajor_tile(smem_u32(sP), TILE_BYTES), ddSm0 = mnmajor_tile(smem_u32(sdS), TILE_BYTES);
            const uint64_t dQm0 = mnmajor_tile(smem_u32(sQ), TILE_BYTES), ddOm0 = mnmajor_tile(smem_u32(sdO), TILE_BYTES);
            bool ok = true;
            int g = 0;
            for (int k = 0, item; ok && (item = item_get(ring, k, true, abort_flag)) >= 0; ++k) {
                const int n = p.nq - att_round(item, p.BH, p.bh_magic);
                for (int it = 0; it < n; ++it, ++g) {
                    const int s = g % ATT_BWD_STAGES;
                    const uint64_t dQm = dQm0 + (uint64_t)s * TILESTEP, ddOm = ddOm0 + (uint64_t)s * TILESTEP;
                    const uint64_t ddSm = ddSm0 + (uint64_t)(g & 1) * (2 * TILESTEP);
                    if (!mbar_wait(&qdo_full[s], (uint32_t)((g / ATT_BWD_STAGES) & 1), abort_flag)) { ok = false; break; }
                    if (!mbar_wait(pds_full, (uint32_t)(g & 1), abort_flag)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        umma_bf16(tdV, dPm + j * MNSTEP, ddOm + j * MNSTEP, id_t, (it > 0 || j > 0) ? 1u : 0u);
                    umma_commit(w_free);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        umma_bf16(tdK, ddSm + j * MNSTEP, dQm + j * MNSTEP, id_t, (it > 0 || j > 0) ? 1u : 0u);
                    umma_commit(&ds_free[g % ATT_DS_FREE]);
                    // S and dP of this block (the other issuer's) completed before the compute warps could sign
                    // pds_full, so this commit covers every read of the stage
                    umma_commit(&qdo_empty[s]);
                }
                if (ok) umma_commit(acc_full);
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 24); }
        }
    } else if (warp == 3 + ATT_BWD_CW) {
        // the dS blocks leave for the dQ kernel as they lie in shared memory.  Not before the products that read them have
        // completed: a 32 KB read of shared memory beside those would delay them.  An item's output tiles leave here too:
        // no compute warp waits for them to be read out.
        if (elect_one()) {
            const long long nblk = (long long)p.nq * (p.nq + 1) / 2;
            bool ok = true;
            int g = 0;
            mbar_arrive(w_free);                      // in front of block 0: no buffer to be read out
            for (int k = 0, item; ok && (item = item_get(ring, k, true, abort_flag)) >= 0; ++k) {
                const int kb = att_round(item, p.BH, p.bh_magic), bh = item - kb * p.BH, b = bh / p.H, h = bh % p.H;
                for (int qb = kb; qb < p.nq; ++qb, ++g) {
                    if (!mbar_wait(&ds_free[g % ATT_DS_FREE], (uint32_t)((g / ATT_DS_FREE) & 1), abort_flag)) { ok = false; break; }
                    bulk_store(reinterpret_cast<uint8_t*>(p.ds) + ((long long)bh * nblk + (long long)qb * (qb + 1) / 2 + kb) * DS_BLOCK_BYTES,
                               sdS + (g & 1) * DS_BLOCK_BYTES, DS_BLOCK_BYTES);
                    tma_store_commit();
                    tma_store_wait_read<0>();
                    mbar_arrive(w_free);
                }
                if (!ok || !mbar_wait(out_full, (uint32_t)(k & 1), abort_flag)) { ok = false; break; }
                if (p.dqkv != nullptr) {
                    tma_store_4d(&tmoK, sP, 0, kb * ATT_BN, h, b);              // rows past T are clipped
                    tma_store_4d(&tmoV, sP + TILE_BYTES, 0, kb * ATT_BN, h, b);
                } else {
                    uint8_t* spare = sdS + (g & 1) * DS_BLOCK_BYTES;
                    for (int c = 0; c * 32 < p.hd; ++c) {
                        tma_store_3d(&tmoK, sP + c * TILE_BYTES, c * 32, kb * ATT_BN, bh);
                        tma_store_3d(&tmoV, spare + c * TILE_BYTES, c * 32, kb * ATT_BN, bh);
                    }
                }
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(out_done);
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 25); }
        }
    } else {
        const int q = warp & 3;
        const int cq = (warp - 2) >> 2;               // which 32 key columns this warp handles
        const int r = q * 32 + lane;                  // query row inside the block
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const int half = cq & 1;                      // epilogue: dV leaves by the first eight warps (two per lane quarter:
        const bool is_dk = cq >= 2;                   // head-dim columns 0-31 | 32-63), dK by the others
        bool ok = true;
        int g = 0;
        // the row's log-sum-exp and delta of the NEXT query block are asked for while this one is worked on
        float lse_next = INFINITY, dl_next = 0.0f;
        auto fetch_row = [&](int item, int qb) {
            const int qi = qb * ATT_BM + r;
            lse_next = INFINITY; dl_next = 0.0f;      // rows past T: P = 0
            if (qi < p.T) {
                const long long o = (long long)(item - att_round(item, p.BH, p.bh_magic) * p.BH) * p.T + qi;
                lse_next = p.lse[o]; dl_next = p.delta[o];
            }
        };
        int item = item_get(ring, 0, false, abort_flag);
        if (item >= 0) fetch_row(item, att_round(item, p.BH, p.bh_magic));
        for (int k = 0; ok && item >= 0; ++k) {
            const int kb = att_round(item, p.BH, p.bh_magic), k0 = kb * ATT_BN;
            int next_item = -1;
            for (int qb = kb; qb < p.nq; ++qb, ++g) {
                const uint32_t pi = (uint32_t)(g & 1);
                const bool diag = qb == kb;
                // (the factor is applied here and not where the value is asked for: there it would wait for the load)
                const float lse2 = lse_next * 1.4426950408889634f, dl = dl_next;
                if (!mbar_wait(sdp_full, pi, abort_flag)) { ok = false; break; }
                tc_fence_after();
                // this thread's 32 scores and 32 dP values in one TMEM round trip, then the tiles are free
                uint32_t sv[32], dv[32];
                tmem_ld32(tS + lane_base + cq * 32, sv);
                tmem_ld32(tdP + lane_base + cq * 32, dv);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(sdp_free);
                if (qb + 1 < p.nq) fetch_row(item, qb + 1);
                else if ((next_item = item_get(ring, k + 1, false, abort_flag)) >= 0)
                    fetch_row(next_item, att_round(next_item, p.BH, p.bh_magic));
                uint8_t* sdS_g = sdS + pi * DS_BLOCK_BYTES;
                // the diagonal block masks keys after the query: columns e <= lim are allowed
                const int lim = diag ? r - cq * 32 : 32;
                uint4 pP[2], pD[2];
                p_and_ds16<0>(sv, dv, p.scale_log2, lse2, dl, diag, lim, pP, pD);
                // the previous block's P has been read, the one before has left this dS buffer; at an item's start the staged
                // outputs have left both
                if (!mbar_wait(w_free, pi ^ 1u, abort_flag)) { ok = false; break; }
                if (diag && k > 0 && !mbar_wait(out_done, (uint32_t)(k & 1) ^ 1u, abort_flag)) { ok = false; break; }
                store_half_chunk(sP, r, cq, 0, pP);
                store_half_chunk(sdS_g, r, cq, 0, pD);
                p_and_ds16<16>(sv, dv, p.scale_log2, lse2, dl, diag, lim, pP, pD);
                store_half_chunk(sP, r, cq, 1, pP);
                store_half_chunk(sdS_g, r, cq, 1, pD);
                tc_fence_before();
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(pds_full);
            }
            const int kj = k0 + r;                        // key row of the accumulators
            RopeRow rot;                                  // fetched while the last products finish
            if (ok && is_dk && kj < p.T && p.dqkv != nullptr)
                load_rope_row(rot, p.cos_t + (long long)kj * (p.hd >> 1), p.sin_t + (long long)kj * (p.hd >> 1), half * 32, p.hd);
            if (ok && !mbar_wait(acc_full, (uint32_t)(k & 1), abort_flag)) ok = false;
            // the float32 dV tiles go into the dS buffer that the next item's first block will use (g is behind the last block)
            uint8_t* spare = sdS + (g & 1) * DS_BLOCK_BYTES;
            if (ok && p.dqkv == nullptr && !mbar_wait(w_free, (uint32_t)(g & 1) ^ 1u, abort_flag)) ok = false;
            if (ok) {
                tc_fence_after();
                uint32_t v[32];
                tmem_ld32((is_dk ? tdK : tdV) + lane_base + half * 32, v);
                tmem_ld_wait();
                tc_fence_before();
                if (p.dqkv != nullptr) {
                    // the P tiles are free (every product has completed): dK into the first, dV into the second
                    if (kj < p.T) stage_row_bf16(sP + (is_dk ? 0 : TILE_BYTES), r, v, half * 32, p.hd, is_dk ? &rot : nullptr, is_dk ? p.scale : 1.0f);
                } else {
                    // separate float32 outputs [B*H, T, hd]: dK into the two P tiles (head-dim columns 0-31 | 32-63), dV
                    // into the spare dS buffer; tmoK / tmoV are float32 maps here
                    if (kj < p.T && half * 32 < p.hd) stage_row_f32((is_dk ? sP : spare) + half * TILE_BYTES, r, v, is_dk ? p.scale : 1.0f);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(out_full);
            }
            item = next_item;
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 23); }
    }

    __syncwarp();
    if (*abort_flag) for (int i = 0; i < 64; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// dQ of one query block: dQ = scale * sum over its key blocks kb = 0 .. qb of dS'(qb, kb) K(kb), the dS' blocks read
// back as the dK/dV kernel stored them.  No exponentials and no compute warps in the loop: a loader, a tensor-core
// issuer and four epilogue warps (thread = query row).  A CTA works through several (query block, head) items with
// four stages of 48 KB running through all of them and two accumulators, so that an item's epilogue lies beside the next
// one's loop (two CTAs per SM with an item each and two stages took 31 us at 16 x 6 heads x 1024: the set-up, first loads
// and epilogue of an item are as long as its 4.5 blocks).  Sums are formed in key-block order: fixed, no atomics.
constexpr int ATT_DQ_THREADS = 192;
constexpr int ATT_DQ_STAGES = 4;
constexpr int ATT_DQ_STAGE_BYTES = DS_BLOCK_BYTES + TILE_BYTES;

__global__ void __launch_bounds__(ATT_DQ_THREADS, 1)
attention_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmoQ,
                        const AttBwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    // stage s: dS block (two [128 x 64] tiles) then the K tile; behind the stages two tiles for the output
    uint8_t* out = smem + ATT_DQ_STAGES * ATT_DQ_STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(out + 2 * TILE_BYTES);
    uint64_t* full = bars;             // ATT_DQ_STAGES
    uint64_t* empty = bars + 4;        // ATT_DQ_STAGES
    uint64_t* acc_full = bars + 8;     // 2
    uint64_t* acc_empty = bars + 10;   // 2, four arrivals
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const ItemRing ring = item_ring(reinterpret_cast<uint8_t*>(bars + 14));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto q_block = [&](int item) { return p.nq - 1 - att_round(item, p.BH, p.bh_magic); };       // heaviest query blocks of all heads first

    if (threadIdx.x == 0) {
        for (int i = 0; i < 12; ++i) mbar_init(&bars[i], i >= 10 ? 4 : 1);
        item_ring_init(ring, 5);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 128); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tdQ = *tmem_slot;
    pdl_wait();                 // everything above is independent of earlier kernels' results

    if (warp == 0) {
        if (elect_one()) {
            bool ok = true;
            const long long nblk = (long long)p.nq * (p.nq + 1) / 2;
            int g = 0;
            for (int k = 0, item = (int)blockIdx.x; ok; ++k) {
                if (!item_put(ring, k, item, abort_flag)) { ok = false; break; }
                if (item < 0) break;
                const int qb = q_block(item), bh = item - (p.nq - 1 - qb) * p.BH;
                const uint8_t* src = reinterpret_cast<const uint8_t*>(p.ds) +
                                     ((long long)bh * nblk + (long long)qb * (qb + 1) / 2) * DS_BLOCK_BYTES;
                for (int it = 0; it <= qb; ++it, ++g) {
                    const int s = g % ATT_DQ_STAGES;
                    if (it == qb) item_ask(ring);
                    if (!mbar_wait(&empty[s], (uint32_t)((g / ATT_DQ_STAGES) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                    uint8_t* st = smem + s * ATT_DQ_STAGE_BYTES;
                    mbar_expect_tx(&full[s], ATT_DQ_STAGE_BYTES);
                    bulk_load(st, src + (long long)it * DS_BLOCK_BYTES, DS_BLOCK_BYTES, &full[s]);
                    tma_load_3d(st + DS_BLOCK_BYTES, &tmK, &full[s], 0, it * ATT_BN, bh);
                }
                if (ok) item = item_answer(ring, k, abort_flag);
            }
            pdl_launch_dependents_now();     // all loads issued: the next kernel may start its prologue
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 31); }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t id_q = umma_idesc(1u, 0u, 1u, 128, 64);       // dS (K-major) x K block (MN-major)
            bool ok = true;
            int g = 0;
            for (int k = 0, item; ok && (item = item_get(ring, k, true, abort_flag)) >= 0; ++k) {
                const int qb = q_block(item);
                if (!mbar_wait(&acc_empty[k & 1], (uint32_t)((k >> 1) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after();
                for (int it = 0; it <= qb; ++it, ++g) {
                    const int s = g % ATT_DQ_STAGES;
                    const uint32_t st = smem_u32(smem + s * ATT_DQ_STAGE_BYTES);
                    const uint64_t ddSk = kmajor_tile(st);
                    const uint64_t dKm = mnmajor_tile(st + DS_BLOCK_BYTES, TILE_BYTES);
                    if (!mbar_wait(&full[s], (uint32_t)((g / ATT_DQ_STAGES) & 1), abort_flag)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        umma_bf16(tdQ + (uint32_t)((k & 1) * 64), ddSk + (uint64_t)(j >> 2) * TILESTEP + (uint64_t)(j & 3) * KSTEP,
                                  dKm + j * MNSTEP, id_q, (it > 0 || j > 0) ? 1u : 0u);
                    umma_commit(&empty[s]);
                }
                if (ok) umma_commit(&acc_full[k & 1]);
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 32); }
        }
    } else {
        const int q = warp & 3;
        const int r = q * 32 + lane;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        bool ok = true;
        for (int k = 0, item; (item = item_get(ring, k, false, abort_flag)) >= 0; ++k) {
            const int qb = q_block(item), bh = item - (p.nq - 1 - qb) * p.BH, q0 = qb * ATT_BM, qi = q0 + r;
            const bool valid = qi < p.T;
            RopeRow rot0, rot1;                           // fetched while the products run
            if (valid && p.dqkv != nullptr) {
                const float* cs = p.cos_t + (long long)qi * (p.hd >> 1);
                const float* sn = p.sin_t + (long long)qi * (p.hd >> 1);
                load_rope_row(rot0, cs, sn, 0, p.hd);
                load_rope_row(rot1, cs, sn, 32, p.hd);
            }
            // (a thread whose wait gave up goes on with the others to the barriers below; every later wait returns at once)
            if (!mbar_wait(&acc_full[k & 1], (uint32_t)((k >> 1) & 1), abort_flag)) { ok = false; *abort_flag = 1; }
            tc_fence_after();
            uint32_t v0[32], v1[32];
            tmem_ld32(tdQ + (uint32_t)((k & 1) * 64) + lane_base, v0);
            tmem_ld32(tdQ + (uint32_t)((k & 1) * 64) + lane_base + 32, v1);
            tmem_ld_wait();
            tc_fence_before();
            if (q == 0 && lane == 0) tma_store_wait_read<0>();       // the previous item's rows have left the output tiles
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (lane == 0) mbar_arrive(&acc_empty[k & 1]);
            if (p.dqkv != nullptr) {
                if (valid) {
                    stage_row_bf16(out, r, v0, 0, p.hd, &rot0, p.scale);
                    stage_row_bf16(out, r, v1, 32, p.hd, &rot1, p.scale);
                }
            } else if (valid) {                       // float32 dQ [B*H, T, hd]
                stage_row_f32(out, r, v0, p.scale);
                if (p.hd > 32) stage_row_f32(out + TILE_BYTES, r, v1, p.scale);
            }
            fence_proxy_async();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (q == 0 && lane == 0) {
                const int b = bh / p.H, h = bh % p.H;
                if (p.dqkv != nullptr) tma_store_4d(&tmoQ, out, 0, q0, h, b);          // rows past T are clipped
                else for (int c = 0; c * 32 < p.hd; ++c) tma_store_3d(&tmoQ, out + c * TILE_BYTES, c * 32, q0, bh);
                tma_store_commit();
            }
        }
        if (q == 0 && lane == 0) tma_store_wait_read<0>();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 33); }
    }

    __syncwarp();
    if (*abort_flag) for (int i = 0; i < 64; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tdQ, 128); }
}

// dQ, dK and dV of a head whose sequence is one block (T <= 128), in one kernel: no second pass, no dS' blocks in memory, no
// kernel for the row dots in front.  Nothing is long enough to be bound by a pipe here; the time is the chain load -> scores ->
// P and dS' -> products -> output (~4 us), so the three launches of the longer path cost more than their work, and two CTAs per
// SM put 296 heads under way at once.  Hence 113 KB (P takes V's tile, which is free once dP is formed, and one more; the outputs
// are staged over P, dS' and Q) and 256 tensor-memory columns (the products accumulate over S and dP, which are in registers by
// then); one thread does all loads, products and stores.  Rows of steps past T are left out of the products.
// Measured against the three kernels: 100 x 6 heads x 128, hd 64: 57 -> 37 us; training step of 28 x 128 tokens, 12 layers, TF32:
// 4384 -> 4210 us; of 4 x 64 tokens, 2 layers of width 64: 227 -> 217 us.
constexpr int ATT_BWD1_CW = 8;          // compute warps: row dots, then 64 key columns of a row per thread
constexpr int ATT_BWD1_THREADS = 32 + 32 * ATT_BWD1_CW;
constexpr int ATT_BWD1_SMEM = 7 * TILE_BYTES + 1024;

__global__ void __launch_bounds__(ATT_BWD1_THREADS, 2)
attention_bwd_one_block_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                               const __grid_constant__ CUtensorMap tmoQ, const __grid_constant__ CUtensorMap tmoK,
                               const __grid_constant__ CUtensorMap tmoV, const AttBwdParams p) {
    // (two CTAs fill the SM's shared memory to the byte, so there is no room to align the tiles by hand)
    extern __shared__ __align__(1024) uint8_t smem_tiles[];
    uint8_t* sP = smem_tiles;                              // 2 tiles, the first is V's
    uint8_t* sV = smem_tiles;
    uint8_t* sdS = smem_tiles + 2 * TILE_BYTES;            // 2 tiles
    uint8_t* sQ = smem_tiles + 4 * TILE_BYTES;
    uint8_t* sdO = smem_tiles + 5 * TILE_BYTES;
    uint8_t* sK = smem_tiles + 6 * TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_tiles + 7 * TILE_BYTES);
    uint64_t* qk_full = bars;
    uint64_t* ov_full = bars + 1;
    uint64_t* sdp_full = bars + 2;
    uint64_t* pds_full = bars + 3;     // one arrival per compute warp
    uint64_t* acc_full = bars + 4;
    uint64_t* out_full = bars + 5;     // one arrival per compute warp
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* s_delta = reinterpret_cast<float*>(bars + 8);   // [128]

    if (smem_u32(smem_tiles) & 1023u) {        // (the swizzled tiles need it; nothing in front of them moves them)
        if (threadIdx.x == 0) atomicExch(p.err, 28);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bh = (int)blockIdx.x, b = bh / p.H, h = bh - b * p.H;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 6; ++i) mbar_init(&bars[i], (i == 3 || i == 5) ? ATT_BWD1_CW : 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tdP = tmem_base + 128;
    const uint32_t tOut = tmem_base;                       // dK | dV | dQ, 64 columns each
    pdl_wait();                 // everything above is independent of earlier kernels' results

    if (warp == 0) {
        if (elect_one()) {
            const int steps = (p.T + 15) >> 4;
            bool ok = true;
            mbar_expect_tx(qk_full, 2 * TILE_BYTES);
            tma_load_3d(sQ, &tmQ, qk_full, 0, 0, bh);
            tma_load_3d(sK, &tmK, qk_full, 0, 0, bh);
            mbar_expect_tx(ov_full, 2 * TILE_BYTES);
            tma_load_4d(sdO, &tmdO, ov_full, 0, 0, h, b);
            tma_load_3d(sV, &tmV, ov_full, 0, 0, bh);
            pdl_launch_dependents_now();     // all loads issued: the next kernel may start its prologue
            const uint32_t id_s = umma_idesc(1u, 0u, 0u, 128, 128), id_t = umma_idesc(1u, 1u, 1u, 128, 64);
            const uint32_t id_q = umma_idesc(1u, 0u, 1u, 128, 64);
            ok = mbar_wait(qk_full, 0, abort_flag);
            if (ok) {
                const uint64_t dQk = kmajor_tile(smem_u32(sQ)), dKk = kmajor_tile(smem_u32(sK));
#pragma unroll
                for (int j = 0; j < 4; ++j) umma_bf16(tS, dQk + j * KSTEP, dKk + j * KSTEP, id_s, j > 0 ? 1u : 0u);
                ok = mbar_wait(ov_full, 0, abort_flag);
            }
            if (ok) {
                const uint64_t ddOk = kmajor_tile(smem_u32(sdO)), dVk = kmajor_tile(smem_u32(sV));
#pragma unroll
                for (int j = 0; j < 4; ++j) umma_bf16(tdP, ddOk + j * KSTEP, dVk + j * KSTEP, id_s, j > 0 ? 1u : 0u);
                umma_commit(sdp_full);
                ok = mbar_wait(pds_full, 0, abort_flag);
            }
            if (ok) {
                tc_fence_after();
                const uint64_t dPm = mnmajor_tile(smem_u32(sP), TILE_BYTES), ddSm = mnmajor_tile(smem_u32(sdS), TILE_BYTES);
                const uint64_t dQm = mnmajor_tile(smem_u32(sQ), TILE_BYTES), ddOm = mnmajor_tile(smem_u32(sdO), TILE_BYTES);
                const uint64_t ddSk = kmajor_tile(smem_u32(sdS)), dKm = mnmajor_tile(smem_u32(sK), TILE_BYTES);
                for (int j = 0; j < steps; ++j) umma_bf16(tOut, ddSm + j * MNSTEP, dQm + j * MNSTEP, id_t, j > 0 ? 1u : 0u);
                for (int j = 0; j < steps; ++j) umma_bf16(tOut + 64, dPm + j * MNSTEP, ddOm + j * MNSTEP, id_t, j > 0 ? 1u : 0u);
                for (int j = 0; j < steps; ++j)
                    umma_bf16(tOut + 128, ddSk + (uint64_t)(j >> 2) * TILESTEP + (uint64_t)(j & 3) * KSTEP, dKm + j * MNSTEP, id_q,
                              j > 0 ? 1u : 0u);
                umma_commit(acc_full);
                ok = mbar_wait(out_full, 0, abort_flag);
            }
            if (ok) {
                if (p.dqkv != nullptr) {
                    tma_store_4d(&tmoK, smem_tiles, 0, 0, h, b);              // rows past T are clipped
                    tma_store_4d(&tmoV, smem_tiles + TILE_BYTES, 0, 0, h, b);
                    tma_store_4d(&tmoQ, smem_tiles + 2 * TILE_BYTES, 0, 0, h, b);
                } else {
                    for (int c = 0; c * 32 < p.hd; ++c) {
                        tma_store_3d(&tmoK, smem_tiles + c * TILE_BYTES, c * 32, 0, bh);
                        tma_store_3d(&tmoV, smem_tiles + (2 + c) * TILE_BYTES, c * 32, 0, bh);
                        tma_store_3d(&tmoQ, smem_tiles + (4 + c) * TILE_BYTES, c * 32, 0, bh);
                    }
                }
                tma_store_commit();
                tma_store_wait_read<0>();
            }
            if (!ok) { *abort_flag = 1; atomicExch(p.err, 26); }
        }
    } else {
        const int w = warp - 1, q = warp & 3, half = w >> 2;      // TMEM lane quarter; 64 key columns, later 32 head-dim columns
        const int r = q * 32 + lane;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const float lse2 = r < p.T ? p.lse[(long long)bh * p.T + r] * 1.4426950408889634f : INFINITY;     // rows past T: P = 0
        // the row dots of 16 rows per warp, eight lanes a row
        {
            const int D = p.H * p.hd, piece = lane & 7;
            float s[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = w * 16 + i * 4 + (lane >> 3);
                s[i] = (t < p.T && piece * 8 < p.hd) ? dot8(p.att, p.datt, ((long long)b * p.T + t) * D + h * p.hd + piece * 8) : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = w * 16 + i * 4 + (lane >> 3);
                s[i] = sum8(s[i]);
                if (piece == 0) {
                    s_delta[t] = s[i];
                    if (t < p.T) p.delta[(long long)bh * p.T + t] = s[i];
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * ATT_BWD1_CW) : "memory");
        const float dl = s_delta[r];
        bool ok = mbar_wait(sdp_full, 0, abort_flag);
        if (ok) {
            tc_fence_after();
#pragma unroll 1
            for (int c = 2 * half; c < 2 * half + 2; ++c) {
                uint4 pP[2], pD[2];
                if (c <= q) {
                    uint32_t sv[32], dv[32];
                    tmem_ld32(tS + lane_base + c * 32, sv);
                    tmem_ld32(tdP + lane_base + c * 32, dv);
                    tmem_ld_wait();
                    const int lim = r - c * 32;           // keys after the query are masked
                    p_and_ds16<0>(sv, dv, p.scale_log2, lse2, dl, true, lim, pP, pD);
                    store_half_chunk(sP, r, c, 0, pP);
                    store_half_chunk(sdS, r, c, 0, pD);
                    p_and_ds16<16>(sv, dv, p.scale_log2, lse2, dl, true, lim, pP, pD);
                } else {                                  // all of them
                    pP[0] = pP[1] = pD[0] = pD[1] = make_uint4(0u, 0u, 0u, 0u);
                    store_half_chunk(sP, r, c, 0, pP);
                    store_half_chunk(sdS, r, c, 0, pD);
                }
                store_half_chunk(sP, r, c, 1, pP);
                store_half_chunk(sdS, r, c, 1, pD);
            }
            tc_fence_before();
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(pds_full);
            RopeRow rot;                                  // fetched while the products run; row r is query and key
            if (r < p.T && p.dqkv != nullptr)
                load_rope_row(rot, p.cos_t + (long long)r * (p.hd >> 1), p.sin_t + (long long)r * (p.hd >> 1), half * 32, p.hd);
            ok = mbar_wait(acc_full, 0, abort_flag);
            if (ok) {
                tc_fence_after();
#pragma unroll
                for (int o = 0; o < 3; ++o) {             // dK, dV, dQ
                    uint32_t v[32];
                    tmem_ld32(tOut + o * 64 + lane_base + half * 32, v);
                    tmem_ld_wait();
                    if (r < p.T && p.dqkv != nullptr)
                        stage_row_bf16(smem_tiles + o * TILE_BYTES, r, v, half * 32, p.hd, o != 1 ? &rot : nullptr, o != 1 ? p.scale : 1.0f);
                    else if (r < p.T && half * 32 < p.hd)
                        stage_row_f32(smem_tiles + (2 * o + half) * TILE_BYTES, r, v, o != 1 ? p.scale : 1.0f);
                }
                tc_fence_before();
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(out_full);
            }
        }
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 27); }
    }

    __syncwarp();
    if (*abort_flag) for (int i = 0; i < 64; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

constexpr int ATT_DKDV_SMEM = 1024 + (8 + 2 * ATT_BWD_STAGES) * TILE_BYTES + 384;
constexpr int ATT_DQ_SMEM = 1024 + ATT_DQ_STAGES * ATT_DQ_STAGE_BYTES + 2 * TILE_BYTES + 384;

size_t attention_bwd_ds_bytes(int B, int H, int T) {
    const long long nq = (T + ATT_BM - 1) / ATT_BM;
    return (size_t)((long long)B * H * (nq * (nq + 1) / 2) * DS_BLOCK_BYTES);
}

int launch_attention_bwd(DeviceCtx* ctx, const bf16* Q, const bf16* K, const bf16* V, const bf16* att,
                         const bf16* datt, const float* lse, float* delta, float* dQ, float* dK, float* dV, int B,
                         int H, int T, int hd, float scale, cudaStream_t stream, bf16* dqkv, const float* cos_t,
                         const float* sin_t, bf16* ds_blocks) {
    TB_CHECK(hd > 0 && hd <= ATT_HD && hd % 8 == 0, "fused attention needs head_dim <= 64 and a multiple of 8 (got %d)", hd);
    TB_CHECK(dqkv != nullptr ? (cos_t && sin_t && (reinterpret_cast<uintptr_t>(dqkv) & 15u) == 0) : (dQ && dK && dV),
             "attention backward needs either dQ, dK, dV or the merged output with the rotation tables");
    TB_CHECK(B > 0 && H > 0 && T > 0, "attention dims must be positive");
    const int BH = B * H, D = H * hd;
    CUtensorMap tmQ, tmK, tmV, tmdO;
    TB_TRY(make_operand_map(&tmQ, Q, hd, T, hd, BH, (long long)T * hd, 128));
    TB_TRY(make_operand_map(&tmK, K, hd, T, hd, BH, (long long)T * hd, 128));
    TB_TRY(make_operand_map(&tmV, V, hd, T, hd, BH, (long long)T * hd, 128));
    TB_TRY(make_operand_map4(&tmdO, datt, hd, T, D, H, hd, B, (long long)T * D, 128));
    // the merged output dqkv [B*T, 3D] as three (hd, T, H, B) views for the tile stores
    CUtensorMap tmoQ = tmdO, tmoK = tmdO, tmoV = tmdO;
    if (dqkv != nullptr) {
        TB_TRY(make_operand_map4(&tmoQ, dqkv, hd, T, 3LL * D, H, hd, B, (long long)T * 3 * D, 128));
        TB_TRY(make_operand_map4(&tmoK, dqkv + D, hd, T, 3LL * D, H, hd, B, (long long)T * 3 * D, 128));
        TB_TRY(make_operand_map4(&tmoV, dqkv + 2 * D, hd, T, 3LL * D, H, hd, B, (long long)T * 3 * D, 128));
    } else {
        TB_TRY(make_operand_map_f32(&tmoQ, dQ, hd, T, hd, BH, (long long)T * hd, 128));
        TB_TRY(make_operand_map_f32(&tmoK, dK, hd, T, hd, BH, (long long)T * hd, 128));
        TB_TRY(make_operand_map_f32(&tmoV, dV, hd, T, hd, BH, (long long)T * hd, 128));
    }
    AttBwdParams p;
    p.T = T; p.H = H; p.hd = hd; p.nq = (T + ATT_BM - 1) / ATT_BM;
    p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
    p.lse = lse; p.delta = delta; p.dQ = dQ; p.dK = dK; p.dV = dV; p.err = ctx->d_err;
    p.dqkv = dqkv; p.cos_t = cos_t; p.sin_t = sin_t;
    p.att = att; p.datt = datt; p.BH = BH;
    const double tri = (double)BH * T * (double)T * hd;      // one lower-triangular product = tri flops
    if (p.nq == 1) {        // one block per head: nothing to hand from kernel to kernel
        static bool attr_one[64] = {false};
        if (!attr_one[ctx->device & 63]) {
            TB_CUDA(cudaFuncSetAttribute(attention_bwd_one_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_BWD1_SMEM));
            attr_one[ctx->device & 63] = true;
        }
        prof_mark(ctx, "attention_bwd_one_block", 5.0 * tri, (double)BH * T * hd * (2.0 * 5 + 12.0), stream);
        TB_CUDA(launch_kernel(attention_bwd_one_block_kernel, dim3((unsigned)BH), dim3(ATT_BWD1_THREADS), ATT_BWD1_SMEM, stream, tmQ, tmK,
                              tmV, tmdO, tmoQ, tmoK, tmoV, p));
        TB_CUDA(cudaGetLastError());
        ctx->launches++;
        prof_close(ctx, stream);
        return 0;
    }
    if (ds_blocks == nullptr) {      // no caller-owned buffer for the dS blocks: the context's scratch
        TB_TRY(ensure_scratch(ctx, attention_bwd_ds_bytes(B, H, T)));
        ds_blocks = reinterpret_cast<bf16*>(ctx->scratch);
    }
    TB_CHECK((reinterpret_cast<uintptr_t>(ds_blocks) & 15u) == 0, "the dS block buffer must be 16-byte aligned");
    p.ds = ds_blocks;
    static bool attr_set[64] = {false};
    if (!attr_set[ctx->device & 63]) {
        TB_CUDA(cudaFuncSetAttribute(attention_bwd_dkdv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_DKDV_SMEM));
        TB_CUDA(cudaFuncSetAttribute(attention_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_DQ_SMEM));
        attr_set[ctx->device & 63] = true;
    }
    {
        const long long total = (long long)B * T * H;
        long long blocks = (total + 31) / 32;         // eight lanes per row
        if (blocks > 8LL * ctx->sm_count) blocks = 8LL * ctx->sm_count;
        prof_mark(ctx, "attention_delta", 0.0, 0.0, stream);
        TB_CUDA(launch_kernel(attention_delta_kernel, dim3((int)blocks), dim3(256), 0, stream, att, datt, delta, B, T, H, hd));
        TB_CUDA(cudaGetLastError());
        ctx->launches++;
        prof_close(ctx, stream);
    }
    p.bh_magic = att_magic(BH, (long long)BH * p.nq);
    const dim3 grid((unsigned)(BH * p.nq));
    prof_mark(ctx, "attention_bwd_dkdv", 4.0 * tri, (double)BH * T * hd * (2.0 * 4 + 8.0), stream);
    TB_CUDA(launch_kernel(attention_bwd_dkdv_kernel, grid, dim3(ATT_BWD_THREADS), ATT_DKDV_SMEM, stream, tmQ, tmK, tmV, tmdO, tmoK, tmoV, p));
    TB_CUDA(cudaGetLastError());
    ctx->launches++;
    prof_close(ctx, stream);
    prof_mark(ctx, "attention_bwd_dq", 1.0 * tri, (double)BH * T * hd * (2.0 * 4 + 4.0), stream);
    TB_CUDA(launch_kernel(attention_bwd_dq_kernel, grid, dim3(ATT_DQ_THREADS), ATT_DQ_SMEM, stream, tmK, tmoQ, p));
    TB_CUDA(cudaGetLastError());
    ctx->launches++;
    prof_close(ctx, stream);
    return 0;
}

constexpr int ATT_FWD_SMEM = 1024 + 7 * TILE_BYTES;

int launch_attention_fwd(DeviceCtx* ctx, const bf16* Q, const bf16* K, const bf16* V, bf16* att, float* lse, int B,
                         int H, int T, int hd, float scale, cudaStream_t stream, long long kv_rows_per_head) {
    TB_CHECK(hd > 0 && hd <= ATT_HD && hd % 8 == 0, "fused attention needs head_dim <= 64 and a multiple of 8 (got %d)", hd);
    TB_CHECK(B > 0 && H > 0 && T > 0, "attention dims must be positive");
    const int BH = B * H;
    CUtensorMap tmQ, tmK, tmV;
    TB_TRY(make_operand_map(&tmQ, Q, hd, T, hd, BH, (long long)T * hd, ATT_BM));
    const long long kv_rows = kv_rows_per_head > 0 ? kv_rows_per_head : T;      // a KV cache has room for more rows
    TB_TRY(make_operand_map(&tmK, K, hd, T, hd, BH, kv_rows * hd, ATT_BN));
    TB_TRY(make_operand_map(&tmV, V, hd, T, hd, BH, kv_rows * hd, ATT_BN));
    CUtensorMap tmO;        // att [B*T, D] as (hd, T, H, B) for the tile store
    TB_TRY(make_operand_map4(&tmO, att, hd, T, (long long)H * hd, H, hd, B, (long long)T * H * hd, ATT_BM));
    AttFwdParams p;
    p.T = T; p.H = H; p.hd = hd; p.D = H * hd;
    p.nq = (T + ATT_BM - 1) / ATT_BM;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.att = att; p.lse = lse; p.err = ctx->d_err;
    static bool attr_set[64] = {false};
    if (!attr_set[ctx->device & 63]) {
        TB_CUDA(cudaFuncSetAttribute(attention_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_FWD_SMEM));
        attr_set[ctx->device & 63] = true;
    }
    dim3 grid(BH, p.nq);
    // algorithmic work: the lower triangle of two products of 2*T*T*hd flops each
    prof_mark(ctx, "attention_fwd", 2.0 * (double)BH * T * (double)T * hd, (double)BH * T * hd * 2.0 * 4.0, stream);
    TB_CUDA(launch_kernel(attention_fwd_kernel, dim3(grid), dim3(ATT_FWD_THREADS), ATT_FWD_SMEM, stream, tmQ, tmK, tmV, tmO, p));
    TB_CUDA(cudaGetLastError());
    ctx->launches++;
    prof_close(ctx, stream);
    return 0;
}

}  // namespace tb

