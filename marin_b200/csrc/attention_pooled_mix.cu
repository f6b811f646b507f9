// bf16 attention over a window and pooled blocks with mixed head weights (attention_pooled.cu) over prompt portions, on the tensor cores
// (tcgen05; the mixing mma.sync), compiled for one head layout: -DHEAD_DIM, -DV_DIM (multiples of 16 up to 128), -DGROUP (2 or 4 query heads a kv head), -DKV_HEADS
// (with GROUP * KV_HEADS 16 or 32).
//
// out_h = sum_j (sum_g talk[h, g] p_g[j]) v_kv(h)[j]: the heads' weights of a (query, key) pair are mixed before they meet the values, so every
// head multiplies its own kv head's values once.  (attention_pooled_fast.cu sums every head over every kv head's values and mixes the sums: KV_HEADS
// times the products with V, and a float32 [tokens][H][KV_HEADS][V_DIM] that a second kernel reads.)  Mixing needs the weights already
// divided by their sums, so three kernels:
//   stats_kernel  (a CTA per kv head and 128 rows = queries x its heads, tcgen05): the logarithm of every row's sum of weights;
//   mix_kernel    (equal runs of the tiles' blocks a CTA, two heads a warp, 16 queries x 16 keys a step): the weights of all heads, mixed, to scratch memory in 16 bits;
//   value_kernel  (a CTA per 128 rows of a kv head, tcgen05): mixed weights x values.
// Exactness: the weights p are float32 and enter the mixing product as pairs of bf16 numbers (p = hi + lo), as does talk; the three larger of the four
// products are taken, so about 16 bits of each enter.  The mixed weights, bounded numbers, wait as halves under one power of two for all of them (11 bits) and
// meet the values as two bf16 numbers that hold the 11 bits exactly: they add next to nothing to the error that rounding the results
// makes, where weights rounded to bf16 (every head's, in the other kernel) made it 1.17 times as large.
// Scratch: [tile][block][kv head][query][8 keys][its head][key] halves, a tile of 16 queries of one request, its blocks of 32 pooled rows, then of 32 positions.
// Measured on B200, 2,048 tokens, 32 heads of 128 over 8, window 1,024, pools of 64: the other kernel and its mixing 1,189 us;
// these 55 + 166 + 63 us (95 + 216 + 141 with a CTA a tile in the mixing, three barriers a block and the sums and values on mma.sync).  mix_kernel is bound by issue: about a
// thousand instructions a warp and block (cap, exponential, two parts, their stores) behind which its products of 3,600 clocks a block hide.
#define MB_LIB "attention_pooled_mix"
#define MB_LIB_ID 25
#include <cuda_fp16.h>
#include "tc_common.cuh"
#include "launch.cuh"
#include "mma_helpers.cuh"

#ifndef HEAD_DIM
#define HEAD_DIM 128
#endif
#ifndef V_DIM
#define V_DIM HEAD_DIM
#endif
#ifndef GROUP
#define GROUP 4
#endif
#ifndef KV_HEADS
#define KV_HEADS 8
#endif
static_assert(HEAD_DIM % 16 == 0 && HEAD_DIM >= 16 && HEAD_DIM <= 128 && V_DIM % 16 == 0 && V_DIM >= 16 && V_DIM <= 128, "head sizes: multiples of 16 up to 128");
static_assert(GROUP == 2 || GROUP == 4, "two or four query heads a kv head");
static_assert(GROUP * KV_HEADS == 16 || GROUP * KV_HEADS == 32, "16 or 32 query heads");

#define D HEAD_DIM
#define DV V_DIM
#define G GROUP
#define KH KV_HEADS
#define NH (GROUP * KV_HEADS)
#define NQ 16                         // queries a tile
#define NK 32                         // keys a block
#define LDK (D + 8)                   // padded rows in shared memory (elements): ldmatrix without bank conflicts
#define LOG2E 1.4426950408889634f

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// tanh(x) = 1 - 2 / (1 + e^(2x)) from the fast exponential: its absolute error is a few 1e-7 (see attention_pooled_fast.cu)
__device__ __forceinline__ float tanh_approx(float x) { return 1.0f - __fdividef(2.0f, 1.0f + ex2_approx(x * (2.0f * LOG2E))); }
// Scores in the exp2 domain, capped where there is a cap: cap tanh(x) with x = s scale / cap.  Where every |x| of a warp's block is at most 0.5, tanh(x) = x P(x^2)
// with the cubic fitted there by least squares that attention_tc.cu uses (relative error 6e-7), which leaves the one exponential of the weight to the unit for
// functions; else from the fast exponential.
struct Cap {
    float to_cap, sl2, p0, p1, p2, p3;
    bool on;
    __device__ Cap(float scale, float cap) {
        on = cap > 0.0f;
        to_cap = on ? scale / cap : 0.0f;
        sl2 = (on ? cap : scale) * LOG2E;
        const float c2 = to_cap * to_cap;
        p0 = 0.999999464f * to_cap; p1 = -0.333264679f * to_cap * c2; p2 = 0.131918818f * to_cap * c2 * c2; p3 = -0.0444444381f * to_cap * c2 * c2 * c2;
    }
    // what sl2 multiplies
    __device__ float small(float s) const { const float t = s * s; return s * fmaf(t, fmaf(t, fmaf(t, p3, p2), p1), p0); }
    template <int N> __device__ void apply(float (*s)[4]) const {
        if (!on) return;
        float top = 0.0f;
#pragma unroll
        for (int j = 0; j < N; ++j) top = fmaxf(top, fmaxf(fmaxf(fabsf(s[j][0]), fabsf(s[j][1])), fmaxf(fabsf(s[j][2]), fabsf(s[j][3]))));
        if (__all_sync(0xffffffffu, top * fabsf(to_cap) <= 0.5f)) {
#pragma unroll
            for (int j = 0; j < N; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[j][e] = small(s[j][e]);
        } else {
#pragma unroll
            for (int j = 0; j < N; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[j][e] = tanh_approx(s[j][e] * to_cap);
        }
    }
};

// What a query at position p sees: pooled rows below nb, positions from lo on.
__device__ __forceinline__ int first_seen(int p, int window) { return window > 0 ? max(0, p - window + 1) : 0; }
__device__ __forceinline__ int pools_seen(int p, int window, int pool) { return pool > 0 && window > 0 ? max(0, (p - window + 1) / pool) : 0; }

// The tiles of 16 queries of request r start at this tile of the step's portions (room is left for a partial tile per request).
__device__ __forceinline__ int first_tile(const int* cu_tokens, int first_req, int r) { return (cu_tokens[r] - cu_tokens[first_req]) / NQ + (r - first_req); }

// Blocks of a tile whose queries are at positions q_first .. q_last: pooled ones first, then positions from the block of the first one seen.  Of a
// block only the rows from `begin` to `end` are read, what lies beside them counts as zero: a page that the window has passed may belong to another
// request, and a number there that is not finite would reach the sums through a weight of zero.
struct Blocks {
    int pooled, first, count, nb_most, seen, q_last;
    __device__ Blocks(int q_first, int q_last_, int window, int pool, int size) {
        q_last = q_last_;
        nb_most = pools_seen(q_last, window, pool);
        pooled = (nb_most + size - 1) / size;
        seen = first_seen(q_first, window);
        first = seen / size;
        count = pooled + q_last / size - first + 1;
    }
    __device__ bool is_pooled(int b) const { return b < pooled; }
    __device__ int begin(int b) const { return b < pooled ? 0 : seen; }
    __device__ int end(int b) const { return b < pooled ? nb_most - 1 : q_last; }
    __device__ int key0(int b, int size) const { return b < pooled ? b * size : (first + b - pooled) * size; }
};

// Where key n of kv head kh lies: a position's row, or (pooled) block n's row.
__device__ __forceinline__ size_t row_at(const int* table, int n, bool pooled, int kh, int page_shift, int pool, int pool_rows) {
    const int p = pooled ? n * pool + pool - 1 : n, mask = (1 << page_shift) - 1;
    const size_t page = (size_t)table[p >> page_shift];
    return pooled ? (page * KH + kh) * (size_t)pool_rows + (size_t)((p & mask) / pool) : (((page * KH + kh) << page_shift) + (size_t)(p & mask));
}

// The A operand of one 16 x 16 step straight from memory: rows r and r + 8 (null: not there) at column c.
__device__ __forceinline__ void q_fragment(uint32_t* a, const bf16* lo, const bf16* hi, int c) {
    a[0] = lo != nullptr ? *reinterpret_cast<const uint32_t*>(lo + c) : 0u;
    a[1] = hi != nullptr ? *reinterpret_cast<const uint32_t*>(hi + c) : 0u;
    a[2] = lo != nullptr ? *reinterpret_cast<const uint32_t*>(lo + c + 8) : 0u;
    a[3] = hi != nullptr ? *reinterpret_cast<const uint32_t*>(hi + c + 8) : 0u;
}

// ---- the logarithm (base 2) of every row's sum of weights ---------------------------------------------------------------------------------
// On tcgen05: 128 rows (queries x the heads of a kv head) x 64 keys a block into one of four buffers of tensor memory; a thread has a row, two warps of 32
// rows take the blocks in turn and add their sums at the end.  Four warps bring the keys, one issues the MMAs.  Bound by the rows' instructions (62% of the issue slots,
// tensor cores 13%); on mma.sync, where a warp also loaded fragments and shared its rows' maxima, 79 us, now 55 (2,048 tokens, 32 heads of 128, window 1,024).
#define SQ (128 / G)                  // queries a CTA
#define SN 64                         // keys a block
#define S_STAGES 4                    // blocks of keys, and buffers of scores
#define S_HALVES ((D + 63) / 64)
#define S_Q_HALF (128 * 128)
#define S_K_HALF (SN * 128)
#define S_K_BYTES (S_HALVES * S_K_HALF)
#define STATS_SMEM (S_HALVES * S_Q_HALF + S_STAGES * S_K_BYTES + 1024)
#define S_ROW_WARPS 8
#define S_LOAD_WARPS 4
#define STATS_THREADS (32 * (S_ROW_WARPS + S_LOAD_WARPS + 1))
#define S_ROW_BLOCKS 24               // blocks whose rows' places are kept in shared memory

__global__ void __launch_bounds__(STATS_THREADS, 2) stats_kernel(
    const bf16* __restrict__ q, const bf16* __restrict__ k_cache, const bf16* __restrict__ k_pool, float* __restrict__ lse,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens, int first_req,
    int page_shift, float scale, float cap, int window, int pool, int pool_rows, int* __restrict__ error_flag) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t k_full[S_STAGES], s_done[S_STAGES], s_free[S_STAGES];
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned s_row[S_ROW_BLOCKS * SN];
    __shared__ float2 s_other[128];
    uint8_t* sQ = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sK = sQ + S_HALVES * S_Q_HALF;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    PDL_ENTER_EARLY();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); k_pool = pdl_fresh(k_pool);
    const int r = first_req + blockIdx.y, kh = blockIdx.x, qt = gridDim.z - 1 - blockIdx.z;          // all heads' long tiles first
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    if (qt * SQ >= n) return;
    if (tid == 0) {
        for (int i = 0; i < S_STAGES; ++i) { mbar_init(&k_full[i], S_LOAD_WARPS); mbar_init(&s_done[i], 1); mbar_init(&s_free[i], 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc<false>(&tmem_slot, S_STAGES * SN);
    const int here = min(SQ, n - qt * SQ), pos0 = seq_lens[r] - n + qt * SQ;
    const int* table = block_table + (size_t)r * max_pages;
    const Blocks blocks(pos0, pos0 + here - 1, window, pool, SN);
    for (int idx = tid; idx < 128 * (D / 8); idx += STATS_THREADS) {
        const int row = idx / (D / 8), c = idx % (D / 8), ql = row / G;
        uint8_t* dst = sQ + c / 8 * S_Q_HALF + row * 128 + (((c ^ row) & 7) << 4);
        if (ql < here) cp_async16(dst, q + ((size_t)(tok0 + qt * SQ + ql) * NH + kh * G + row % G) * D + c * 8);
        else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    }
    cp_async_commit();
    auto row_of = [&](int b, int i) {
        const int key = blocks.key0(b, SN) + i;
        return key >= blocks.begin(b) && key <= blocks.end(b) ? (unsigned)row_at(table, key, blocks.is_pooled(b), kh, page_shift, pool, pool_rows) : ~0u;
    };
    for (int i = tid; i < min(blocks.count, S_ROW_BLOCKS) * SN; i += STATS_THREADS) s_row[i] = row_of(i / SN, i % SN);
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const int role = warp_same(warp), count = warp_same(blocks.count);
    bool ok = true;
    float m_run = -INFINITY, l_run = 0.0f;
    if (role == S_ROW_WARPS + S_LOAD_WARPS) {
        // ---- the MMAs: S(b) = Q K(b)^T once the keys have landed and the rows have read what lay in its buffer ----
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(SN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t elected = elect_one(), d = warp_same(tmem);
        for (int b = 0; b < count; ++b) {
            const int st = b % S_STAGES;
            if (ok && !mbar_wait_warp(&k_full[st], (b / S_STAGES) & 1)) { atomicExch(error_flag, 44); ok = false; }
            if (ok && b >= S_STAGES && !mbar_wait_warp(&s_free[st], (b / S_STAGES - 1) & 1)) { atomicExch(error_flag, 45); ok = false; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t da = umma_desc(smem_u32(sQ)), db = umma_desc(smem_u32(sK) + st * S_K_BYTES);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
                umma_bf16(d + (uint32_t)(st * SN), da + (uint32_t)(kk / 4 * (S_Q_HALF >> 4) + 2 * (kk % 4)), db + (uint32_t)(kk / 4 * (S_K_HALF >> 4) + 2 * (kk % 4)), idesc,
                          kk > 0 ? 1u : 0u, elected);
            umma_commit(&s_done[st], elected);
        }
    } else if (role >= S_ROW_WARPS) {
        // ---- the keys: a block's loads two blocks ahead of its arrival ----
        const int t = tid - 32 * S_ROW_WARPS;
        constexpr int PER = D / 8, THREADS = 32 * S_LOAD_WARPS;
        for (int b = 0; b < count + 2; ++b) {
            if (b < count) {
                const int st = b % S_STAGES;
                if (b >= S_STAGES && ok && !mbar_wait(&s_done[st], (b / S_STAGES - 1) & 1)) { atomicExch(error_flag, 46); ok = false; }
                uint8_t* to = sK + st * S_K_BYTES;
                const bf16* src = blocks.is_pooled(b) ? k_pool : k_cache;
#pragma unroll
                for (int i = 0; i < SN * PER; i += THREADS) {
                    const int idx = i + t, row = idx / PER, c = idx % PER;
                    const unsigned at = b < S_ROW_BLOCKS ? s_row[b * SN + row] : row_of(b, row);
                    uint8_t* dst = to + c / 8 * S_K_HALF + row * 128 + (((c ^ row) & 7) << 4);
                    if (at != ~0u) cp_async16(dst, src + (size_t)at * D + c * 8);
                    else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
                }
            }
            cp_async_commit();
            if (b < 2) continue;
            cp_async_wait<2>();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&k_full[(b - 2) % S_STAGES])) : "memory");
        }
    } else {
        // ---- the rows ----
        const int row = (warp & 3) * 32 + lane, qp = row / G < here ? pos0 + row / G : -1;       // (a query that is not there sees nothing)
        const int lo = first_seen(qp, window), nb = qp >= 0 ? pools_seen(qp, window, pool) : 0;
        const Cap c(scale, cap);
        for (int b = warp >> 2; b < count; b += 2) {
            const int st = b % S_STAGES;
            if (ok && !mbar_wait(&s_done[st], (b / S_STAGES) & 1)) { atomicExch(error_flag, 47); ok = false; }
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool pooled = blocks.is_pooled(b);
            const int key0 = blocks.key0(b, SN);
            const bool inside = __all_sync(0xffffffffu, pooled ? key0 + SN <= nb : key0 + SN - 1 <= qp && key0 >= lo);
#pragma unroll
            for (int half = 0; half < SN; half += 32) {
                float s[32];
                tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(st * SN + half), s);
                tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(st * SN + half + 16), s + 16);
                if (half + 32 == SN) {                         // the buffer may be written again
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&s_free[st])) : "memory");
                }
                c.apply<8>(reinterpret_cast<float(*)[4]>(s));
                if (!inside) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        const int kj = key0 + half + e;
                        if (!(pooled ? kj < nb : (kj <= qp && kj >= lo))) s[e] = -INFINITY;
                    }
                }
                float top[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
                for (int e = 4; e < 32; ++e) top[e & 3] = fmaxf(top[e & 3], s[e]);
                const float m_new = fmaxf(m_run, fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * c.sl2), base = m_new == -INFINITY ? 0.0f : m_new;
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int e = 0; e < 32; ++e) sum[e & 3] += ex2_approx(fmaf(s[e], c.sl2, -base));
                l_run = fmaf(l_run, ex2_approx(m_run - base), (sum[0] + sum[1]) + (sum[2] + sum[3]));
                m_run = m_new;
            }
        }
        if (warp >= 4) s_other[row] = make_float2(m_run, l_run);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tmem_free<false>(tmem, S_STAGES * SN);
    if (warp < 4) {
        const int row = tid, ql = row / G;
        const float2 o = s_other[row];
        const float m = fmaxf(m_run, o.x), base = m == -INFINITY ? 0.0f : m;
        if (ql < here) lse[(size_t)(tok0 + qt * SQ + ql) * NH + kh * G + row % G] = m + log2f(fmaf(l_run, ex2_approx(m_run - base), o.y * ex2_approx(o.x - base)));
    }
}

// ---- the weights of all heads, mixed -----------------------------------------------------------------------------------------------------
#define HW 2                          // heads a warp: their queries and scores then fit 128 registers, and 16 warps hide one another's waits
#define WK (G / HW)                   // warps a kv head
#define MIX_WARPS (KH * WK)
#define MIX_THREADS (32 * MIX_WARPS)
#define HK 16                         // keys a step: half a block
#define P_PITCH (2 * NH + 16)         // bytes of a pair's row of H weights
#define P_BYTES (NQ * HK * P_PITCH + NQ / 4 * 16)
#define TALK_FRAGS ((NH / 16) * (NH / 16))
#define MIX_SMEM (2 * KH * HK * LDK * 2 + 4 * P_BYTES + 2 * TALK_FRAGS * 4 * 512)
static_assert(MIX_SMEM <= 220 * 1024, "the mixing kernel's tiles do not fit shared memory");
// Where a query's row of pairs begins: a group of four queries 16 bytes further on, and a query's heads two by two turned by query % 4 within 16 bytes, so that the
// 32 rows a warp writes a word of lie in 32 banks (rows of whole 16 bytes alone: four of them a bank).  talk's columns are turned alike.
struct MixWhole { static constexpr bool value = false; };
struct MixMasked { static constexpr bool value = true; };
__device__ __forceinline__ int p_row(int query) { return query * HK * P_PITCH + (query >> 2) * 16; }

__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 back = __bfloat1622float2(h);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = pack_bf16(x - back.x, y - back.y);
}
__device__ __forceinline__ uint32_t pack_half(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// A mixed weight is at most NH times the largest |talk| (every weight is at most 1); this power of two brings it below 2^15, so that its 11 bits as a
// half are there down to 2^-29 of the bound (a bf16 has 8).  Found by every warp from all of talk: the largest of numbers does not depend on their order.
__device__ __forceinline__ int mixed_shift(const float* __restrict__ talk, int lane) {
    float top = 0.0f;
    for (int i = lane; i < NH * NH; i += 32) top = fmaxf(top, fabsf(talk[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    return min(100, max(-100, 14 - ilogbf(fmaxf(top, 1e-30f) * NH)));
}
__device__ __forceinline__ float two_to(int n) { return __int_as_float((127 + n) << 23); }

// The blocks of a step's tiles end to end, dealt out in equal runs over the CTAs: a tile ahead of a whole window has few blocks, and one CTA a tile left
// SMs idle for a third of the time.
__global__ void __launch_bounds__(MIX_THREADS, 1) mix_kernel(
    const bf16* __restrict__ q, const bf16* __restrict__ k_cache, const bf16* __restrict__ k_pool, const float* __restrict__ lse,
    const float* __restrict__ talk, __half* __restrict__ mixed, const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens,
    const int* __restrict__ seq_lens, int first_req, int reqs, int page_shift, float scale, float cap, int window, int pool, int pool_rows, int most_blocks) {
    PDL_ENTER();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); k_pool = pdl_fresh(k_pool); lse = pdl_fresh(lse);
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ int s_before[MIX_THREADS], s_warp[MIX_WARPS];
    bf16* sK = reinterpret_cast<bf16*>(smem_raw);              // two of [KH][HK][LDK]: a kv head's keys are fetched and read by its own warps
    uint8_t* sP = smem_raw + 2 * KH * HK * LDK * 2;            // two of [2][NQ][HK] rows of H weights: the larger part and what it leaves
    uint4* sT = reinterpret_cast<uint4*>(sP + 4 * P_BYTES);    // talk as A operands: [turned by][2 parts][H / 16][H / 16][lane]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t2 = 2 * (lane & 3);
    const int last_req = first_req + reqs - 1, tiles_all = first_tile(cu_tokens, first_req, last_req + 1);
    // the tile of this number: its request, and how many of it there are before (-1: none has this number)
    auto request_of = [&](int tile) {
        int lo = first_req, hi = last_req;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first_tile(cu_tokens, first_req, mid) <= tile) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    };
    auto blocks_of = [&](int tile) {
        if (tile >= tiles_all) return 0;
        const int r = request_of(tile), q0 = (tile - first_tile(cu_tokens, first_req, r)) * NQ, n = cu_tokens[r + 1] - cu_tokens[r];
        if (q0 >= n) return 0;
        const int pos0 = seq_lens[r] - n + q0;
        return Blocks(pos0, pos0 + min(NQ, n - q0) - 1, window, pool, NK).count;
    };
    const int per = (tiles_all + MIX_THREADS - 1) / MIX_THREADS;
    int units;                                                 // blocks of all tiles
    {
        int mine = 0;
        for (int i = 0; i < per; ++i) mine += blocks_of(tid * per + i);
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        if (lane == 31) s_warp[warp] = sum;
        __syncthreads();
        int before = 0;
        units = 0;
        for (int w = 0; w < MIX_WARPS; ++w) {
            if (w < warp) before += s_warp[w];
            units += s_warp[w];
        }
        s_before[tid] = before + sum - mine;
    }
    int unit = (int)((long long)units * blockIdx.x / gridDim.x);
    const int unit_end = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);
    if (unit >= unit_end) return;
    constexpr int MT = NH / 16;                                // 16 mixed heads at a time: a warp keeps to one of the MT
    const int mt = warp % MT, turned = (warp / MT) & 3;        // and to queries that are turned alike
    for (int idx = tid; idx < 4 * TALK_FRAGS * 32; idx += MIX_THREADS) {
        const int turn = idx / (TALK_FRAGS * 32), frag = idx / 32 % TALK_FRAGS, l = idx % 32, row = frag / MT * 16 + (l >> 2);
        const int col = frag % MT * 16 + 2 * ((l - turn) & 3);
        uint4 hi, lo;
        split_bf16(talk[row * NH + col], talk[row * NH + col + 1], hi.x, lo.x);
        split_bf16(talk[(row + 8) * NH + col], talk[(row + 8) * NH + col + 1], hi.y, lo.y);
        split_bf16(talk[row * NH + col + 8], talk[row * NH + col + 9], hi.z, lo.z);
        split_bf16(talk[(row + 8) * NH + col + 8], talk[(row + 8) * NH + col + 9], hi.w, lo.w);
        sT[(turn * 2) * TALK_FRAGS * 32 + frag * 32 + l] = hi;
        sT[(turn * 2 + 1) * TALK_FRAGS * 32 + frag * 32 + l] = lo;
    }
    const float up = two_to(mixed_shift(talk, lane));
    const Cap c(scale, cap);
    const int kv = warp / WK;
    bf16* myK = sK + kv * HK * LDK;
    const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(myK + ((lane & 7) + (lane >> 4) * 8) * LDK + ((lane >> 3) & 1) * 8);
    // a pair's row read as a B operand: eight keys of one query, 8 weights a matrix, up to 32 weights at a time
    const uint32_t p_addr = (uint32_t)__cvta_generic_to_shared(sP + (lane & 7) * P_PITCH + (lane >> 3) * 16);
    const int p_at = p_row(g8) + t2 * P_PITCH + ((warp * HW / 2) & ~3) * 4 + ((warp * HW / 2 + g8) & 3) * 4;   // where this warp's pair of heads lies in query g8's rows
    __syncthreads();                                           // s_before and talk are there
    int tile;                                                  // the tile this CTA begins in
    {
        int lo = 0, hi = MIX_THREADS - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_before[mid] <= unit) lo = mid;
            else hi = mid - 1;
        }
        tile = lo * per;
        int before = s_before[lo];
        for (int n; before + (n = blocks_of(tile)) <= unit; ++tile) before += n;
        unit -= before;                                        // (from here on: the first block of the tile; unit_end counts down with it)
        lo = before;
        hi = unit_end - before;
        for (int left = hi; left > 0; ++tile, unit = 0) {
            const int count = blocks_of(tile);
            if (count == 0) continue;
            const int b_end = min(count, left);
            left -= count;
            const int r = request_of(tile), qt = tile - first_tile(cu_tokens, first_req, r), tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
            const int here = min(NQ, n - qt * NQ), pos0 = seq_lens[r] - n + qt * NQ;
            const int* table = block_table + (size_t)r * max_pages;
            const Blocks blocks(pos0, pos0 + here - 1, window, pool, NK);
            __half* dst = mixed + (size_t)tile * most_blocks * (NH * NQ * NK);
            const int steps = 2 * (b_end - unit), b0 = unit;
            auto fetch = [&](int step) {                       // this warp's part of its kv head's keys: 16 bytes a lane
                if (step < steps) {
                    const int b = b0 + (step >> 1);
                    const bool pooled = blocks.is_pooled(b);
                    const int key0 = blocks.key0(b, NK) + (step & 1) * HK, begin = blocks.begin(b), end = blocks.end(b);
                    const bf16* src = pooled ? k_pool : k_cache;
                    bf16* to = myK + (step & 1) * KH * HK * LDK;
                    constexpr int PER = D / 8;
                    if (!pooled && page_shift >= 4 && key0 >= begin && key0 + HK - 1 <= end) {          // rows of one page, one behind the other
                        const bf16* from = src + row_at(table, key0, false, kv, page_shift, pool, pool_rows) * D;
#pragma unroll
                        for (int i = 0; i < HK * PER; i += 32 * WK) {
                            const int idx = i + warp % WK * 32 + lane;
                            if (HK * PER % (32 * WK) == 0 || idx < HK * PER) cp_async16(to + idx / PER * LDK + idx % PER * 8, from + idx * 8);
                        }
                    } else {
#pragma unroll 1
                        for (int idx = warp % WK * 32 + lane; idx < HK * PER; idx += 32 * WK) {
                            const int row = idx / PER, c8 = idx % PER, key = key0 + row;
                            if (key >= begin && key <= end) cp_async16(to + row * LDK + c8 * 8, src + row_at(table, key, pooled, kv, page_shift, pool, pool_rows) * D + c8 * 8);
                            else *reinterpret_cast<uint4*>(to + row * LDK + c8 * 8) = make_uint4(0, 0, 0, 0);
                        }
                    }
                }
                cp_async_commit();
            };
            fetch(0);
            fetch(1);
            // the queries of this warp's heads stay in registers; a thread's rows are queries g8 and g8 + 8
            uint32_t qa[HW][D / 16][4];
            float base[HW][2];
            int qp[2], seen[2], nb[2];
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                qp[rr] = g8 + 8 * rr < here ? pos0 + g8 + 8 * rr : -1;          // (a query that is not there sees nothing)
                seen[rr] = first_seen(qp[rr], window);
                nb[rr] = qp[rr] >= 0 ? pools_seen(qp[rr], window, pool) : 0;
            }
#pragma unroll
            for (int h = 0; h < HW; ++h) {
                const size_t a0 = (size_t)(tok0 + qt * NQ + g8) * NH + warp * HW + h, a1 = a0 + (size_t)8 * NH;
                const bf16 *r0 = qp[0] >= 0 ? q + a0 * D : nullptr, *r1 = qp[1] >= 0 ? q + a1 * D : nullptr;
                base[h][0] = qp[0] >= 0 ? lse[a0] : 0.0f;
                base[h][1] = qp[1] >= 0 ? lse[a1] : 0.0f;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) q_fragment(qa[h][kk], r0, r1, kk * 16 + t2);
            }
            float s[HW][HK / 8][4];
            auto scores = [&](int step) {
                const uint32_t at = k_addr + (uint32_t)((step & 1) * KH * HK * LDK * 2);
#pragma unroll
                for (int h = 0; h < HW; ++h)
#pragma unroll
                    for (int j = 0; j < HK / 8; ++j) s[h][j][0] = s[h][j][1] = s[h][j][2] = s[h][j][3] = 0.0f;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    uint32_t b0, b1, b2, b3;
                    ldsm_x4(at + (uint32_t)(kk * 32), b0, b1, b2, b3);
#pragma unroll
                    for (int h = 0; h < HW; ++h) {
                        mma_bf16_16816(s[h][0], qa[h][kk], b0, b1);
                        mma_bf16_16816(s[h][1], qa[h][kk], b2, b3);
                    }
                }
            };
            auto put = [&](uint8_t* to, int key0, bool pooled, auto masked) {     // in two parts, to the pairs' rows
#pragma unroll
                for (int j = 0; j < HK / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int rr = e >> 1, in = j * 8 + t2 + (e & 1), kj = key0 + in;
                        float w0 = ex2_approx(fmaf(s[0][j][e], c.sl2, -base[0][rr])), w1 = ex2_approx(fmaf(s[1][j][e], c.sl2, -base[1][rr]));
                        if (decltype(masked)::value && !(pooled ? kj < nb[rr] : (kj <= qp[rr] && kj >= seen[rr]))) w0 = w1 = 0.0f;
                        uint32_t hi, low;
                        split_bf16(w0, w1, hi, low);
                        const int at = (8 * rr * HK + j * 8 + (e & 1)) * P_PITCH + 2 * rr * 16;
                        *reinterpret_cast<uint32_t*>(to + at) = hi;
                        *reinterpret_cast<uint32_t*>(to + P_BYTES + at) = low;
                    }
            };
            auto weights = [&](int step) {
                const int b = b0 + (step >> 1);
                const bool pooled = blocks.is_pooled(b);
                const int key0 = blocks.key0(b, NK) + (step & 1) * HK;
                c.apply<HW * HK / 8>(&s[0][0]);
                const bool inside = pooled ? key0 + HK <= nb[0] && qp[1] >= 0 : key0 + HK - 1 <= qp[0] && key0 >= seen[1] && qp[1] >= 0;
                uint8_t* to = sP + (step & 1) * 2 * P_BYTES + p_at;
                if (__all_sync(0xffffffffu, inside)) put(to, key0, pooled, MixWhole());
                else put(to, key0, pooled, MixMasked());
            };
            // talk x weights: eight pairs (one query, eight keys) at a time, straight to memory: [kv head][query][8 keys][its head][key]
            auto mix = [&](int step) {
                const uint4* t = sT + turned * 2 * TALK_FRAGS * 32 + mt * MT * 32 + lane;
                uint4 th[MT], tl[MT];
#pragma unroll
                for (int ks = 0; ks < MT; ++ks) { th[ks] = t[ks * 32]; tl[ks] = t[(TALK_FRAGS + ks) * 32]; }
                __half* to = dst + (size_t)(b0 + (step >> 1)) * (NH * NQ * NK) + (mt * 16 + g8) / G * (NQ * NK * G) + ((step & 1) * (HK / 8) * G + g8 % G) * 8 + t2;
                constexpr int GROUPS = MIX_WARPS / MT;         // (eight or more: a warp's queries are turned alike)
                static_assert(GROUPS % 4 == 0, "queries that are turned alike");
#pragma unroll
                for (int query = warp / MT; query < NQ; query += GROUPS)
#pragma unroll
                    for (int k8 = 0; k8 < HK / 8; ++k8) {
                        uint32_t ph[4], pl[4];
                        const uint32_t row = p_addr + (uint32_t)((step & 1) * 2 * P_BYTES + p_row(query) + k8 * 8 * P_PITCH);
                        if (NH == 32) {
                            ldsm_x4(row, ph[0], ph[1], ph[2], ph[3]);
                            ldsm_x4(row + P_BYTES, pl[0], pl[1], pl[2], pl[3]);
                        } else {
                            // (16 heads: two matrices; the upper lanes' addresses are not used)
                            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(ph[0]), "=r"(ph[1]) : "r"(row));
                            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(pl[0]), "=r"(pl[1]) : "r"(row + P_BYTES));
                        }
                        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                        for (int ks = 0; ks < MT; ++ks) {
                            const uint32_t ah[4] = {th[ks].x, th[ks].y, th[ks].z, th[ks].w}, al[4] = {tl[ks].x, tl[ks].y, tl[ks].z, tl[ks].w};
                            mma_bf16_16816(acc, ah, ph[2 * ks], ph[2 * ks + 1]);
                            mma_bf16_16816(acc, al, ph[2 * ks], ph[2 * ks + 1]);
                            mma_bf16_16816(acc, ah, pl[2 * ks], pl[2 * ks + 1]);
                        }
                        __half* w = to + (query * (NK / 8) + k8) * G * 8;
                        *reinterpret_cast<uint32_t*>(w) = pack_half(acc[0] * up, acc[1] * up);
                        *reinterpret_cast<uint32_t*>(w + 8 / G * (NQ * NK * G)) = pack_half(acc[2] * up, acc[3] * up);
                    }
            };
            cp_async_wait<1>();
            __syncthreads();                                   // the first step's keys are there (and nobody mixes the tile before any more)
            scores(0);
            weights(0);
            cp_async_wait<0>();
            __syncthreads();
            // one barrier a step: behind it lie the step's weights and the next step's keys; the products of both and the next step's weights run side by side
            for (int step = 0; step < steps; ++step) {
                fetch(step + 2);
                if (step + 1 < steps) scores(step + 1);
                mix(step);
                if (step + 1 < steps) weights(step + 1);
                cp_async_wait<0>();
                __syncthreads();
            }
        }
    }
}

// ---- mixed weights x values -----------------------------------------------------------------------------------------------------------------
// On tcgen05: 128 rows (neighbouring tiles' queries x the heads of a kv head) x 32 keys a block, the weights' 11 bits as two bf16 numbers side by side in a row
// of 128 bytes (32 keys' larger parts, then what they leave), the values as the other operand for both.  Eight warps bring the weights (four blocks
// ahead, in registers) and the values (two ahead, by cp.async), one issues the MMAs.  Bound by the bytes of the mixed weights, most of which come back from HBM.
#define V_STAGES 4
#define VT (8 / G)                    // tiles of 16 queries a CTA: 128 rows
#define V_AHEAD 4                     // blocks of mixed weights on their way in registers
#define V_ROW_BLOCKS 48               // blocks whose rows' places are kept in shared memory (of those behind them they are looked up in the walk)
#define V_HALVES ((DV + 63) / 64)
#define V_A_BYTES (128 * 128)
#define V_B_HALF (NK * 128)           // 64 columns of 32 keys
#define V_STAGE_BYTES (V_A_BYTES + V_HALVES * V_B_HALF)
#define VALUE_SMEM (V_STAGES * V_STAGE_BYTES + 1024)
#define VALUE_WORKERS 256
#define V_CHUNKS (VT * G * NQ * (NK / 8) / VALUE_WORKERS)      // 16-byte pieces of a block's mixed weights a thread
static_assert(VT * G * NQ == 128 && V_CHUNKS == 2, "128 rows, two pieces a thread");
#define V_COLS (DV <= 32 ? 32 : DV <= 64 ? 64 : 128)

__global__ void __launch_bounds__(VALUE_WORKERS + 32, 2) value_kernel(
    const __half* __restrict__ mixed, const float* __restrict__ talk, const bf16* __restrict__ v_cache, const bf16* __restrict__ v_pool, bf16* __restrict__ out,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens, int first_req, int page_shift,
    int window, int pool, int pool_rows, int most_blocks, int* __restrict__ error_flag) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[V_STAGES], done[V_STAGES];
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned s_row[V_ROW_BLOCKS * NK];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    PDL_ENTER();
    mixed = pdl_fresh(mixed); v_cache = pdl_fresh(v_cache); v_pool = pdl_fresh(v_pool);
    const int r = first_req + blockIdx.y, kh = blockIdx.x, qt = (gridDim.z - 1 - blockIdx.z) * VT;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    if (qt * NQ >= n) return;
    if (tid == 0) {
        for (int i = 0; i < V_STAGES; ++i) { mbar_init(&full[i], VALUE_WORKERS / 32); mbar_init(&done[i], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc<false>(&tmem_slot, V_COLS);
    const int here = min(VT * NQ, n - qt * NQ), pos0 = seq_lens[r] - n + qt * NQ;
    const int* table = block_table + (size_t)r * max_pages;
    const Blocks all(pos0, pos0 + here - 1, window, pool, NK);
    // where the blocks' rows lie (~0: not there), looked up ahead of all else: in the walk it would be a third of its instructions
    auto row_of = [&](int b, int n) {
        const int key = all.key0(b, NK) + n;
        return key >= all.begin(b) && key <= all.end(b) ? (unsigned)row_at(table, key, all.is_pooled(b), kh, page_shift, pool, pool_rows) : ~0u;
    };
    for (int i = tid; i < min(all.count, V_ROW_BLOCKS) * NK; i += VALUE_WORKERS + 32) s_row[i] = row_of(i / NK, i % NK);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    if (warp_same(warp) == VALUE_WORKERS / 32) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(DV >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t elected = elect_one(), d = warp_same(tmem);
        const int blocks = warp_same(all.count);
        for (int b = 0; b < blocks; ++b) {
            const int st = b % V_STAGES;
            if (ok && !mbar_wait_warp(&full[st], (b / V_STAGES) & 1)) { atomicExch(error_flag, 41); ok = false; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(smem) + st * V_STAGE_BYTES;
            const uint64_t da = umma_desc(a), db = umma_desc_mn(a + V_A_BYTES, V_B_HALF);
#pragma unroll
            for (int part = 0; part < 2; ++part)
#pragma unroll
                for (int kk = 0; kk < NK / 16; ++kk)
                    umma_bf16(d, da + (uint32_t)(4 * part + 2 * kk), db + (uint32_t)(kk * (2048 >> 4)), idesc, (b > 0 || part > 0 || kk > 0) ? 1u : 0u, elected);
            umma_commit(&done[st], elected);
        }
    } else {
        // this thread's pieces of a block: (tile, 16 bytes of it); row = query of the CTA * G + head
        const __half* from[V_CHUNKS];
        uint32_t at[V_CHUNKS];
        int o_pooled[V_CHUNKS], shift_by[V_CHUNKS], last[V_CHUNKS];      // a tile's own blocks: its pooled ones, how far its positions' lie from the CTA's, its last
#pragma unroll
        for (int i = 0; i < V_CHUNKS; ++i) {
            const int piece = tid + VALUE_WORKERS * i, tile = piece / (G * NQ * (NK / 8)), idx = piece % (G * NQ * (NK / 8));
            const int head = idx % G, query = idx / G / (NK / 8), k8 = idx / G % (NK / 8), row = (tile * NQ + query) * G + head;
            from[i] = mixed + ((size_t)(first_tile(cu_tokens, first_req, r) + qt + tile) * most_blocks) * (NH * NQ * NK) + kh * (G * NQ * NK) + idx * 8;
            at[i] = (uint32_t)(row * 128 + ((k8 ^ (row & 7)) << 4));
            const int first = min(tile * NQ, here - 1), count = min(NQ, here - tile * NQ);
            const Blocks own(pos0 + first, pos0 + first + max(count, 1) - 1, window, pool, NK);
            o_pooled[i] = count > 0 ? own.pooled : 0;
            shift_by[i] = all.first - all.pooled - own.first + own.pooled;
            last[i] = count > 0 ? own.count : 0;
        }
        uint4 raw[V_AHEAD][V_CHUNKS];
        auto load = [&](int b, uint4* to) {
#pragma unroll
            for (int i = 0; i < V_CHUNKS; ++i) {
                const int mine = all.is_pooled(b) ? b : b + shift_by[i];
                const bool there = b < all.count && (all.is_pooled(b) ? b < o_pooled[i] : mine >= o_pooled[i] && mine < last[i]);
                to[i] = there ? *reinterpret_cast<const uint4*>(from[i] + (size_t)(unsigned)(mine * (NH * NQ * NK))) : make_uint4(0, 0, 0, 0);
            }
        };
        constexpr int PER = DV / 8, PASSES = (NK * PER + VALUE_WORKERS - 1) / VALUE_WORKERS;
        uint32_t v_at[PASSES];
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
            const int idx = tid + VALUE_WORKERS * i, row = idx / PER, c = idx % PER;
            v_at[i] = V_A_BYTES + c / 8 * V_B_HALF + row * 128 + (((c ^ row) & 7) << 4);
        }
        auto values = [&](int b) {
            if (b < all.count) {
                const uint32_t to = smem_u32(smem) + (b % V_STAGES) * V_STAGE_BYTES;
                const bf16* src = all.is_pooled(b) ? v_pool : v_cache;
#pragma unroll
                for (int i = 0; i < PASSES; ++i) {
                    const int row = (tid + VALUE_WORKERS * i) / PER;
                    if (NK * PER % VALUE_WORKERS != 0 && row >= NK) break;
                    const unsigned at_row = b < V_ROW_BLOCKS ? s_row[b * NK + row] : row_of(b, row);
                    if (at_row != ~0u) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + v_at[i]), "l"(src + (size_t)at_row * DV + (tid + VALUE_WORKERS * i) % PER * 8) : "memory");
                    else asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(to + v_at[i]), "r"(0) : "memory");
                }
            }
            cp_async_commit();
        };
#pragma unroll
        for (int i = 0; i < V_AHEAD; ++i) load(i, raw[i]);
        values(0);
        values(1);
        for (int b0 = 0; b0 < all.count; b0 += V_AHEAD) {
#pragma unroll
            for (int u = 0; u < V_AHEAD; ++u) {
                const int b = b0 + u, st = b % V_STAGES;
                if (b >= all.count) break;
                // (the stage of block b - 2 is the one that block b + 2's values go to; block b's was free before)
                if (b >= 2 && ok && !mbar_wait(&done[(b - 2) % V_STAGES], ((b - 2) / V_STAGES) & 1)) { atomicExch(error_flag, 42); ok = false; }
                values(b + 2);
                uint8_t* to = smem + st * V_STAGE_BYTES;
#pragma unroll
                for (int i = 0; i < V_CHUNKS; ++i) {
                    const uint32_t w[4] = {raw[u][i].x, raw[u][i].y, raw[u][i].z, raw[u][i].w};
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {              // 11 bits as two bf16 numbers, exactly (the power of two comes off the sums)
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                        split_bf16(f.x, f.y, hi[e], lo[e]);
                    }
                    *reinterpret_cast<uint4*>(to + at[i]) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4*>(to + (at[i] ^ 64)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
                load(b + V_AHEAD, raw[u]);
                cp_async_wait<2>();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[st])) : "memory");
            }
        }
        cp_async_wait<0>();
        const int end = all.count - 1;
        if (ok && !mbar_wait(&done[end % V_STAGES], (end / V_STAGES) & 1)) { atomicExch(error_flag, 43); ok = false; }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // two warps share 32 rows: each takes every other 16 columns
        const int row = (warp & 3) * 32 + lane, query = row / G;
        const float down = two_to(-mixed_shift(talk, lane));
        bf16* to = out + ((size_t)(tok0 + qt * NQ + query) * NH + kh * G + row % G) * DV;
#pragma unroll
        for (int c = 0; c < DV; c += 16) {
            if (((c >> 4) & 1) != (warp >> 2)) continue;
            float v[16];
            tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, v);
            if (query >= here) continue;
            uint32_t p[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) p[e] = pack_bf16(v[2 * e] * down, v[2 * e + 1] * down);
            *reinterpret_cast<uint4*>(to + c) = make_uint4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<uint4*>(to + c + 8) = make_uint4(p[4], p[5], p[6], p[7]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tmem_free<false>(tmem, V_COLS);
}

static int page_shift_of(int page_size) {
    for (int s = 0; s <= 6; ++s)
        if ((1 << s) == page_size) return s;
    return -1;
}

// Requests first_req .. first_req + count - 1 of the step; which: 0 the rows' sums (lse float32 [tokens][H]), 1 the mixed weights, 2 the results (in this
// order).  mixed: halves, (tokens / 16 + count) tiles of most_blocks blocks of H * 512; most_blocks: at least the blocks of 32 any tile of the step has.
// ctas: CTAs that the mixing deals the blocks out to (one per SM).  q, caches, out and mixed 16-byte aligned.
MB_API int mb_attn_pooled_mix(int which, const void* q, const void* k_cache, const void* v_cache, const void* k_pool, const void* v_pool, float* lse,
                              const float* talk, void* mixed, void* out, const int* block_table, int max_pages, const int* cu_tokens, const int* seq_lens,
                              int first_req, int count, int max_query_len, int page_size, float scale, float cap, int window, int pool, int pool_rows,
                              int most_blocks, int ctas, int* error_flag, cudaStream_t s) {
    if (count <= 0 || max_query_len <= 0) return 0;
    const int shift = page_shift_of(page_size);
    if (shift < 0 || window < 0 || pool < 0 || (pool > 0 && (k_pool == nullptr || v_pool == nullptr)) || most_blocks <= 0 || ctas <= 0) return MB_ERR_BAD_SIZE;
    if (pool > 0 && pool_rows != (page_size + pool - 1) / pool) return MB_ERR_BAD_SIZE;
    if ((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)mixed | (uintptr_t)out) & 15) != 0) return MB_ERR_BAD_SIZE;
    if (which == 0) {
        static LaunchSmem smem;
        const int rc = smem.allow(stats_kernel, STATS_SMEM);
        if (rc) return rc;
        return launch_kernel(stats_kernel, dim3(KH, count, (max_query_len + SQ - 1) / SQ), STATS_THREADS, STATS_SMEM, s, 0, (const bf16*)q, (const bf16*)k_cache,
                             (const bf16*)k_pool, lse, block_table, max_pages, cu_tokens, seq_lens, first_req, shift, scale, cap, window, pool, pool_rows, error_flag);
    }
    const int tiles_of = (max_query_len + NQ - 1) / NQ;
    if (which == 1) {
        static LaunchSmem smem;
        const int rc = smem.allow(mix_kernel, MIX_SMEM);
        if (rc) return rc;
        return launch_kernel(mix_kernel, dim3(ctas), MIX_THREADS, MIX_SMEM, s, 0, (const bf16*)q, (const bf16*)k_cache, (const bf16*)k_pool, (const float*)lse, talk,
                             (__half*)mixed, block_table, max_pages, cu_tokens, seq_lens, first_req, count, shift, scale, cap, window, pool, pool_rows, most_blocks);
    }
    static LaunchSmem smem;
    const int rc = smem.allow(value_kernel, VALUE_SMEM);
    if (rc) return rc;
    return launch_kernel(value_kernel, dim3(KH, count, (tiles_of + VT - 1) / VT), VALUE_WORKERS + 32, VALUE_SMEM, s, 0, (const __half*)mixed, talk, (const bf16*)v_cache, (const bf16*)v_pool, (bf16*)out, block_table,
                         max_pages, cu_tokens, seq_lens, first_req, shift, window, pool, pool_rows, most_blocks, error_flag);
}
