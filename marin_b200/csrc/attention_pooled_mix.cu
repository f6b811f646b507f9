// bf16 attention over a window and pooled blocks with mixed head weights (attention_pooled.cu) over prompt portions, on the tensor cores
// (mma.sync), compiled for one head layout: -DHEAD_DIM, -DV_DIM (multiples of 16 up to 128), -DGROUP (2 or 4 query heads a kv head), -DKV_HEADS
// (with GROUP * KV_HEADS 16 or 32).
//
// out_h = sum_j (sum_g talk[h, g] p_g[j]) v_kv(h)[j]: the heads' weights of a (query, key) pair are mixed before they meet the values, so every
// head multiplies its own kv head's values once.  (attention_pooled_fast.cu sums every head over every kv head's values and mixes the sums: KV_HEADS
// times the products with V, and a float32 [tokens][H][KV_HEADS][V_DIM] that a second kernel reads.)  Mixing needs the weights already
// divided by their sums, so three kernels:
//   stats_kernel  (a CTA per kv head and 128 rows = queries x its heads): the logarithm of every row's sum of weights;
//   mix_kernel    (a CTA per 16 queries, two heads a warp, 32 keys at a time): the weights of all heads, mixed, to scratch memory in 16 bits;
//   value_kernel  (a CTA per 32 queries and kv head, a warp per head and 16 queries): mixed weights x values.
// Exactness: the weights p are float32 and enter the mixing product as pairs of bf16 numbers (p = hi + lo), as does talk; the three larger of the four
// products are taken, so about 16 bits of each enter.  The mixed weights, bounded numbers, wait as halves under one power of two for all of them (11 bits) and
// meet the values as two bf16 numbers that hold the 11 bits exactly: they add next to nothing to the error that rounding the results
// makes, where weights rounded to bf16 (every head's, in the other kernel) made it 1.17 times as large.
// Scratch: [tile][block][H][16][32] halves, a tile of 16 queries of one request, its blocks of 32 pooled rows, then of 32 positions.
// Measured on B200, 2,048 tokens, 32 heads of 128 over 8, window 1,024, pools of 64: the other kernel and its mixing 1,189 us;
// these 95 + 216 + 141 us (the values 100 with weights rounded to bf16, one product a block instead of two).  mix_kernel is bound by the instructions that make a weight (about fourteen a score, with the cap) and its two mixing products.
#define MB_LIB "attention_pooled_mix"
#define MB_LIB_ID 25
#include <cuda_fp16.h>
#include "common.cuh"
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
#define LDV (DV + 8)
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
#define SQ (128 / G)                  // queries a CTA: 128 rows with the kv head's query heads
#define SN 64                         // keys a block
#define STATS_SMEM (2 * SN * LDK * 2)

__global__ void __launch_bounds__(256, 2) stats_kernel(
    const bf16* __restrict__ q, const bf16* __restrict__ k_cache, const bf16* __restrict__ k_pool, float* __restrict__ lse,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens, int first_req,
    int page_shift, float scale, float cap, int window, int pool, int pool_rows) {
    PDL_ENTER_EARLY();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); k_pool = pdl_fresh(k_pool);
    extern __shared__ __align__(16) uint8_t smem_raw[];
    bf16* sK = reinterpret_cast<bf16*>(smem_raw);
    const int r = first_req + blockIdx.z, kh = blockIdx.y, qt = gridDim.x - 1 - blockIdx.x;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    if (qt * SQ >= n) return;
    const int here = min(SQ, n - qt * SQ), pos0 = seq_lens[r] - n + qt * SQ;
    const int* table = block_table + (size_t)r * max_pages;
    const Blocks blocks(pos0, pos0 + here - 1, window, pool, SN);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    auto fetch = [&](int b) {
        const bool pooled = blocks.is_pooled(b);
        const int key0 = blocks.key0(b, SN);
        const bf16* src = pooled ? k_pool : k_cache;
        bf16* dst = sK + (b & 1) * SN * LDK;
        const int row = tid >> 2, key = key0 + row;            // four threads a row
        if (key >= blocks.begin(b) && key <= blocks.end(b)) {
            const bf16* from = src + row_at(table, key, pooled, kh, page_shift, pool, pool_rows) * D;
#pragma unroll
            for (int c = tid & 3; c < D / 8; c += 4) cp_async16(dst + row * LDK + c * 8, from + c * 8);
        } else {
#pragma unroll
            for (int c = tid & 3; c < D / 8; c += 4) *reinterpret_cast<uint4*>(dst + row * LDK + c * 8) = make_uint4(0, 0, 0, 0);
        }
        cp_async_commit();
    };
    fetch(0);
    // this thread's rows: warp * 16 + lane / 4 and 8 on; row = query * G + head of the group
    uint32_t qa[D / 16][4];
    int qp[2], lo[2], nb[2], at[2];
    {
        const bf16* rows[2];
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int row = warp * 16 + (lane >> 2) + 8 * rr, ql = row / G;
            const bool there = ql < here;
            at[rr] = there ? (tok0 + qt * SQ + ql) * NH + kh * G + row % G : -1;
            rows[rr] = there ? q + (size_t)at[rr] * D : nullptr;
            qp[rr] = pos0 + ql;
            lo[rr] = first_seen(qp[rr], window);
            nb[rr] = pools_seen(qp[rr], window, pool);
        }
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) q_fragment(qa[kk], rows[0], rows[1], kk * 16 + 2 * (lane & 3));
    }
    const Cap c(scale, cap);
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
    for (int b = 0; b < blocks.count; ++b) {
        const bool pooled = blocks.is_pooled(b);
        const int key0 = blocks.key0(b, SN);
        cp_async_wait<0>();
        __syncthreads();                                       // this block is there, and everyone is done with the other buffer
        if (b + 1 < blocks.count) fetch(b + 1);
        float s[SN / 8][4];
#pragma unroll
        for (int j = 0; j < SN / 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.0f;
        const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(sK + (b & 1) * SN * LDK + ((lane & 7) + (lane >> 4) * 8) * LDK + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
            for (int j = 0; j < SN / 8; j += 2) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4(k_addr + (uint32_t)(j * 8 * LDK * 2 + kk * 32), b0, b1, b2, b3);
                mma_bf16_16816(s[j], qa[kk], b0, b1);
                mma_bf16_16816(s[j + 1], qa[kk], b2, b3);
            }
        c.apply<SN / 8>(s);
        float mx[2] = {-INFINITY, -INFINITY};
        const bool inside = pooled ? key0 + SN <= nb[0] : key0 + SN - 1 <= qp[0] && key0 >= lo[1];      // (rows that are not there: positions beyond)
        if (!inside) {
#pragma unroll
            for (int j = 0; j < SN / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int rr = e >> 1, kj = key0 + j * 8 + 2 * (lane & 3) + (e & 1);
                    if (!(pooled ? kj < nb[rr] : (kj <= qp[rr] && kj >= lo[rr]))) s[j][e] = -INFINITY;
                }
        }
#pragma unroll
        for (int j = 0; j < SN / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
            }
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            mx[rr] = fmaxf(mx[rr], __shfl_xor_sync(0xffffffffu, mx[rr], 1));
            mx[rr] = fmaxf(mx[rr], __shfl_xor_sync(0xffffffffu, mx[rr], 2));
            const float m_new = fmaxf(m_run[rr], mx[rr] * c.sl2), base = m_new == -INFINITY ? 0.0f : m_new;
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < SN / 8; ++j) sum += ex2_approx(fmaf(s[j][2 * rr], c.sl2, -base)) + ex2_approx(fmaf(s[j][2 * rr + 1], c.sl2, -base));
            l_run[rr] = l_run[rr] * ex2_approx(m_run[rr] - base) + sum;
            m_run[rr] = m_new;
        }
    }
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        float l = l_run[rr];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if ((lane & 3) == 0 && at[rr] >= 0) lse[at[rr]] = m_run[rr] + log2f(l);
    }
}

// ---- the weights of all heads, mixed -----------------------------------------------------------------------------------------------------
#define HW 2                          // heads a warp: their queries and scores then fit 128 registers, and 16 warps hide one another's waits
#define WK (G / HW)                   // warps a kv head
#define MIX_WARPS (KH * WK)
#define MIX_THREADS (32 * MIX_WARPS)
#define P_PITCH (2 * NH + 16)         // bytes of a pair's row of H weights
#define P_QUERY (NK * P_PITCH + 16)   // bytes between queries (ldmatrix over a query's keys and the stores over queries both spread over the banks)
#define P_BYTES (NQ * P_QUERY)
#define W_PITCH (2 * NK + 16)         // bytes of a mixed row (one head and query)
#define W_HEAD (NQ * W_PITCH + 16)
#define TALK_FRAGS ((NH / 16) * (NH / 16))
#define MIX_SMEM (KH * NK * LDK * 2 + 2 * P_BYTES + NH * W_HEAD + 2 * TALK_FRAGS * 512)
static_assert(MIX_SMEM <= 227 * 1024, "the mixing kernel's tiles do not fit shared memory");

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

__global__ void __launch_bounds__(MIX_THREADS, 1) mix_kernel(
    const bf16* __restrict__ q, const bf16* __restrict__ k_cache, const bf16* __restrict__ k_pool, const float* __restrict__ lse,
    const float* __restrict__ talk, __half* __restrict__ mixed, const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens,
    const int* __restrict__ seq_lens, int first_req, int page_shift, float scale, float cap, int window, int pool, int pool_rows, int most_blocks) {
    PDL_ENTER();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); k_pool = pdl_fresh(k_pool); lse = pdl_fresh(lse);
    extern __shared__ __align__(16) uint8_t smem_raw[];
    bf16* sK = reinterpret_cast<bf16*>(smem_raw);              // [KH][NK][LDK]: a kv head's block is fetched and read by its own warps
    uint8_t* sPh = smem_raw + KH * NK * LDK * 2;               // [NQ][NK] rows of H weights: the larger part ...
    uint8_t* sPl = sPh + P_BYTES;                              // ... and what it leaves
    uint8_t* sW = sPl + P_BYTES;                               // [H][NQ] rows of NK mixed weights
    uint4* sT = reinterpret_cast<uint4*>(sW + NH * W_HEAD);    // talk as A operands: [2 parts][H / 16][H / 16][lane]
    const int r = first_req + blockIdx.z, qt = gridDim.x - 1 - blockIdx.x;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    if (qt * NQ >= n) return;
    const int here = min(NQ, n - qt * NQ), pos0 = seq_lens[r] - n + qt * NQ;
    const int* table = block_table + (size_t)r * max_pages;
    const Blocks blocks(pos0, pos0 + here - 1, window, pool, NK);
    __half* dst = mixed + (size_t)(first_tile(cu_tokens, first_req, r) + qt) * most_blocks * (NH * NQ * NK);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t2 = 2 * (lane & 3);
    const int kv = warp / WK;
    bf16* myK = sK + kv * NK * LDK;
    auto fetch = [&](int b) {                                  // this warp's part of its kv head's keys: 16 bytes a lane
        const bool pooled = blocks.is_pooled(b);
        const int key0 = blocks.key0(b, NK), begin = blocks.begin(b), end = blocks.end(b);
        const bf16* src = pooled ? k_pool : k_cache;
        constexpr int PER = D / 8;
#pragma unroll 4
        for (int idx = warp % WK * 32 + lane; idx < NK * PER; idx += 32 * WK) {
            const int row = idx / PER, c = idx % PER, key = key0 + row;
            if (key >= begin && key <= end) cp_async16(myK + row * LDK + c * 8, src + row_at(table, key, pooled, kv, page_shift, pool, pool_rows) * D + c * 8);
            else *reinterpret_cast<uint4*>(myK + row * LDK + c * 8) = make_uint4(0, 0, 0, 0);
        }
        cp_async_commit();
    };
    fetch(0);
    for (int idx = tid; idx < TALK_FRAGS * 32; idx += MIX_THREADS) {
        const int frag = idx / 32, l = idx % 32, row = frag / (NH / 16) * 16 + (l >> 2), col = frag % (NH / 16) * 16 + 2 * (l & 3);
        uint4 hi, lo;
        split_bf16(talk[row * NH + col], talk[row * NH + col + 1], hi.x, lo.x);
        split_bf16(talk[(row + 8) * NH + col], talk[(row + 8) * NH + col + 1], hi.y, lo.y);
        split_bf16(talk[row * NH + col + 8], talk[row * NH + col + 9], hi.z, lo.z);
        split_bf16(talk[(row + 8) * NH + col + 8], talk[(row + 8) * NH + col + 9], hi.w, lo.w);
        sT[idx] = hi;
        sT[TALK_FRAGS * 32 + idx] = lo;
    }
    // the queries of this warp's heads stay in registers; a thread's rows are queries g8 and g8 + 8
    uint32_t qa[HW][D / 16][4];
    float base[HW][2];
    int qp[2], lo[2], nb[2];
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        qp[rr] = g8 + 8 * rr < here ? pos0 + g8 + 8 * rr : -1;          // (a query that is not there sees nothing)
        lo[rr] = first_seen(qp[rr], window);
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
    const Cap c(scale, cap);
    const float up = two_to(mixed_shift(talk, lane));
    const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(myK + ((lane & 7) + (lane >> 4) * 8) * LDK + ((lane >> 3) & 1) * 8);
    // a pair's row read as a B operand: eight keys of one query, 8 weights a matrix, up to 32 weights at a time
    const uint32_t p_addr = (uint32_t)__cvta_generic_to_shared(sPh + (lane & 7) * P_PITCH + (lane >> 3) * 16);
    constexpr int MT = NH / 16;                                // 16 mixed heads at a time: a warp keeps to one of the MT, whose operands it loads once a block
    const int mt = warp % MT;
    cp_async_wait<0>();
    __syncthreads();                                           // the first block's keys and talk are there
    for (int b = 0; b < blocks.count; ++b) {
        const bool pooled = blocks.is_pooled(b);
        const int key0 = blocks.key0(b, NK);
        float s[HW][NK / 8][4];
#pragma unroll
        for (int h = 0; h < HW; ++h)
#pragma unroll
            for (int j = 0; j < NK / 8; ++j) s[h][j][0] = s[h][j][1] = s[h][j][2] = s[h][j][3] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
            for (int j = 0; j < NK / 8; j += 2) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4(k_addr + (uint32_t)(j * 8 * LDK * 2 + kk * 32), b0, b1, b2, b3);
#pragma unroll
                for (int h = 0; h < HW; ++h) {
                    mma_bf16_16816(s[h][j], qa[h][kk], b0, b1);
                    mma_bf16_16816(s[h][j + 1], qa[h][kk], b2, b3);
                }
            }
        c.apply<HW * NK / 8>(&s[0][0]);
        const bool inside = pooled ? key0 + NK <= nb[0] && qp[1] >= 0 : key0 + NK - 1 <= qp[0] && key0 >= lo[1] && qp[1] >= 0;
        // the weights, in two parts, to the pairs' rows
#pragma unroll
        for (int j = 0; j < NK / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int rr = e >> 1, in = j * 8 + t2 + (e & 1), kj = key0 + in;
                float w0 = ex2_approx(fmaf(s[0][j][e], c.sl2, -base[0][rr])), w1 = ex2_approx(fmaf(s[1][j][e], c.sl2, -base[1][rr]));
                if (!inside && !(pooled ? kj < nb[rr] : (kj <= qp[rr] && kj >= lo[rr]))) w0 = w1 = 0.0f;
                uint32_t hi, low;
                split_bf16(w0, w1, hi, low);
                const int at = (g8 + 8 * rr) * P_QUERY + in * P_PITCH + warp * HW * 2;
                *reinterpret_cast<uint32_t*>(sPh + at) = hi;
                *reinterpret_cast<uint32_t*>(sPl + at) = low;
            }
        __syncthreads();                                       // every head's weights of the block are there; its keys and the last mixed rows are done with
        if (b + 1 < blocks.count) fetch(b + 1);
        // talk x weights: eight pairs (one query, eight keys) at a time
        uint4 th[MT], tl[MT];
#pragma unroll
        for (int ks = 0; ks < MT; ++ks) { th[ks] = sT[(mt * MT + ks) * 32 + lane]; tl[ks] = sT[(TALK_FRAGS + mt * MT + ks) * 32 + lane]; }
#pragma unroll 4
        for (int job = warp / MT; job < NQ * (NK / 8); job += MIX_WARPS / MT) {
            const int query = job / (NK / 8), k8 = job % (NK / 8) * 8;
            uint32_t ph[4], pl[4];
            const uint32_t row = p_addr + (uint32_t)(query * P_QUERY + k8 * P_PITCH);
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
            uint8_t* w = sW + (mt * 16 + g8) * W_HEAD + query * W_PITCH + (k8 + t2) * 2;
            *reinterpret_cast<uint32_t*>(w) = pack_half(acc[0] * up, acc[1] * up);
            *reinterpret_cast<uint32_t*>(w + 8 * W_HEAD) = pack_half(acc[2] * up, acc[3] * up);
        }
        cp_async_wait<0>();
        __syncthreads();                                       // the mixed rows and the next block's keys are there; the pairs' rows may be written again
        for (int idx = tid; idx < NH * NQ * (NK / 8); idx += MIX_THREADS) {
            const int row = idx / (NK / 8), c8 = idx % (NK / 8);
            *reinterpret_cast<uint4*>(dst + (size_t)b * (NH * NQ * NK) + row * NK + c8 * 8) =
                *reinterpret_cast<const uint4*>(sW + (row / NQ) * W_HEAD + (row % NQ) * W_PITCH + c8 * 16);
        }
    }
}

// ---- mixed weights x values -----------------------------------------------------------------------------------------------------------------
// Bound by what a CTA fetches through L2: two neighbouring tiles share every block of values (their ranges of blocks differ by one at most at either end).
#define V_STAGES 4
#define VT 2                          // tiles of 16 queries a CTA
static_assert(VT == 2, "a tile's blocks are one of two");
#define A_PITCH (NK + 8)              // elements of a row of mixed weights in shared memory
#define A_TILE (G * NQ * A_PITCH)
#define V_STAGE_BYTES (VT * A_TILE * 2 + NK * LDV * 2)
#define VALUE_SMEM (V_STAGES * V_STAGE_BYTES)
#define VALUE_THREADS (32 * G * VT)

__global__ void __launch_bounds__(VALUE_THREADS, 2) value_kernel(
    const __half* __restrict__ mixed, const float* __restrict__ talk, const bf16* __restrict__ v_cache, const bf16* __restrict__ v_pool, bf16* __restrict__ out,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens, int first_req, int page_shift,
    int window, int pool, int pool_rows, int most_blocks) {
    PDL_ENTER();
    mixed = pdl_fresh(mixed); v_cache = pdl_fresh(v_cache); v_pool = pdl_fresh(v_pool);
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int r = first_req + blockIdx.z, kh = blockIdx.y, qt = (gridDim.x - 1 - blockIdx.x) * VT;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    if (qt * NQ >= n) return;
    const int here = min(VT * NQ, n - qt * NQ), pos0 = seq_lens[r] - n + qt * NQ;
    const int* table = block_table + (size_t)r * max_pages;
    const Blocks all(pos0, pos0 + here - 1, window, pool, NK);
    const Blocks own[VT] = {Blocks(pos0, pos0 + min(here, NQ) - 1, window, pool, NK), Blocks(pos0 + min(here - 1, NQ), pos0 + here - 1, window, pool, NK)};
    // block b of the CTA as a tile's own block (negative: the tile has no such block)
    auto block_of = [&](int b, int tile) {
        if (tile * NQ >= here) return -1;
        const int o_pooled = tile == 0 ? own[0].pooled : own[1].pooled, o_first = tile == 0 ? own[0].first : own[1].first;
        if (all.is_pooled(b)) return b < o_pooled ? b : -1;
        const int at = all.first + b - all.pooled - o_first, o_count = tile == 0 ? own[0].count : own[1].count;
        return at >= 0 && at < o_count - o_pooled ? o_pooled + at : -1;
    };
    const __half* src = mixed + (size_t)(first_tile(cu_tokens, first_req, r) + qt) * most_blocks * (NH * NQ * NK) + (size_t)kh * G * NQ * NK;
    const size_t per_tile = (size_t)most_blocks * (NH * NQ * NK);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tile = warp / G;
    auto fetch = [&](int b) {
        if (b < all.count) {
            __half* sA = reinterpret_cast<__half*>(smem_raw + (b % V_STAGES) * V_STAGE_BYTES);
            bf16* sV = reinterpret_cast<bf16*>(sA + VT * A_TILE);
            constexpr int PER_TILE = G * NQ * (NK / 8);
#pragma unroll
            for (int t = 0; t < VT; ++t) {
                const int mine = block_of(b, t);
                if (mine < 0) continue;
                for (int idx = tid; idx < PER_TILE; idx += VALUE_THREADS) {
                    const int row = idx / (NK / 8), c8 = idx % (NK / 8) * 8;
                    cp_async16(sA + t * A_TILE + row * A_PITCH + c8, src + t * per_tile + (size_t)mine * (NH * NQ * NK) + row * NK + c8);
                }
            }
            const bool pooled = all.is_pooled(b);
            const int key0 = all.key0(b, NK), begin = all.begin(b), end = all.end(b);
            const bf16* from = pooled ? v_pool : v_cache;
            constexpr int PER = DV / 8;
            for (int idx = tid; idx < NK * PER; idx += VALUE_THREADS) {
                const int row = idx / PER, c = idx % PER, key = key0 + row;
                if (key >= begin && key <= end) cp_async16(sV + row * LDV + c * 8, from + row_at(table, key, pooled, kh, page_shift, pool, pool_rows) * DV + c * 8);
                else *reinterpret_cast<uint4*>(sV + row * LDV + c * 8) = make_uint4(0, 0, 0, 0);
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int b = 0; b < V_STAGES - 1; ++b) fetch(b);
    const float down = two_to(-mixed_shift(talk, lane));
    float o[DV / 8][4];
#pragma unroll
    for (int i = 0; i < DV / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    for (int b = 0; b < all.count; ++b) {
        cp_async_wait<V_STAGES - 2>();
        __syncthreads();                                       // block b is there, and everyone is done with the stage that is filled next
        fetch(b + V_STAGES - 1);
        if (block_of(b, tile) < 0) continue;
        const __half* sA = reinterpret_cast<const __half*>(smem_raw + (b % V_STAGES) * V_STAGE_BYTES);
        const uint32_t a_addr = (uint32_t)__cvta_generic_to_shared(sA + (warp * NQ + (lane & 7) + ((lane >> 3) & 1) * 8) * A_PITCH + (lane >> 4) * 8);
        const uint32_t v_addr = (uint32_t)__cvta_generic_to_shared(sA + VT * A_TILE + ((lane & 7) + ((lane >> 3) & 1) * 8) * LDV + (lane >> 4) * 8);
#pragma unroll
        for (int ks = 0; ks < NK / 16; ++ks) {
            uint32_t a[4], hi[4], lo[4];
            ldsm_x4(a_addr + ks * 32, a[0], a[1], a[2], a[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {                      // 11 bits as two bf16 numbers, exactly
                const float2 w = __half22float2(*reinterpret_cast<const __half2*>(&a[i]));
                split_bf16(w.x * down, w.y * down, hi[i], lo[i]);
            }
#pragma unroll
            for (int dt = 0; dt < DV / 8; dt += 2) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4_trans(v_addr + (uint32_t)(ks * 16 * LDV * 2 + dt * 16), b0, b1, b2, b3);
                mma_bf16_16816(o[dt], hi, b0, b1);
                mma_bf16_16816(o[dt + 1], hi, b2, b3);
                mma_bf16_16816(o[dt], lo, b0, b1);
                mma_bf16_16816(o[dt + 1], lo, b2, b3);
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        const int row = tile * NQ + (lane >> 2) + 8 * rr;
        if (row >= here) continue;
        bf16* to = out + ((size_t)(tok0 + qt * NQ + row) * NH + kh * G + warp % G) * DV + 2 * (lane & 3);
#pragma unroll
        for (int i = 0; i < DV / 8; ++i) *reinterpret_cast<uint32_t*>(to + i * 8) = pack_bf16(o[i][2 * rr], o[i][2 * rr + 1]);
    }
}

static int page_shift_of(int page_size) {
    for (int s = 0; s <= 6; ++s)
        if ((1 << s) == page_size) return s;
    return -1;
}

// Requests first_req .. first_req + count - 1 of the step; which: 0 the rows' sums (lse float32 [tokens][H]), 1 the mixed weights, 2 the results (in this
// order).  mixed: halves, (tokens / 16 + count) tiles of most_blocks blocks of H * 512; most_blocks: at least the blocks of 32 any tile of the step has.
// q, caches, out and mixed 16-byte aligned.
MB_API int mb_attn_pooled_mix(int which, const void* q, const void* k_cache, const void* v_cache, const void* k_pool, const void* v_pool, float* lse,
                              const float* talk, void* mixed, void* out, const int* block_table, int max_pages, const int* cu_tokens, const int* seq_lens,
                              int first_req, int count, int max_query_len, int page_size, float scale, float cap, int window, int pool, int pool_rows,
                              int most_blocks, cudaStream_t s) {
    if (count <= 0 || max_query_len <= 0) return 0;
    const int shift = page_shift_of(page_size);
    if (shift < 0 || window < 0 || pool < 0 || (pool > 0 && (k_pool == nullptr || v_pool == nullptr)) || most_blocks <= 0) return MB_ERR_BAD_SIZE;
    if (pool > 0 && pool_rows != (page_size + pool - 1) / pool) return MB_ERR_BAD_SIZE;
    if ((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)mixed | (uintptr_t)out) & 15) != 0) return MB_ERR_BAD_SIZE;
    if (which == 0) {
        cudaFuncSetAttribute(stats_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, STATS_SMEM);
        return launch_kernel(stats_kernel, dim3((max_query_len + SQ - 1) / SQ, KH, count), 256, STATS_SMEM, s, 0, (const bf16*)q, (const bf16*)k_cache,
                             (const bf16*)k_pool, lse, block_table, max_pages, cu_tokens, seq_lens, first_req, shift, scale, cap, window, pool, pool_rows);
    }
    const int tiles_of = (max_query_len + NQ - 1) / NQ;
    if (which == 1) {
        cudaFuncSetAttribute(mix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MIX_SMEM);
        return launch_kernel(mix_kernel, dim3(tiles_of, 1, count), MIX_THREADS, MIX_SMEM, s, 0, (const bf16*)q, (const bf16*)k_cache, (const bf16*)k_pool, (const float*)lse, talk,
                             (__half*)mixed, block_table, max_pages, cu_tokens, seq_lens, first_req, shift, scale, cap, window, pool, pool_rows, most_blocks);
    }
    cudaFuncSetAttribute(value_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, VALUE_SMEM);
    return launch_kernel(value_kernel, dim3((tiles_of + VT - 1) / VT, KH, count), VALUE_THREADS, VALUE_SMEM, s, 0, (const __half*)mixed, talk, (const bf16*)v_cache, (const bf16*)v_pool, (bf16*)out, block_table,
                         max_pages, cu_tokens, seq_lens, first_req, shift, window, pool, pool_rows, most_blocks);
}
