// The 32-bit path's matrix product on the 5th-generation tensor cores: out[t, n] (+)= sum_k x[t, k] * w[n, k], all float32, with the error of
// float32 sums.
//
// A float32 number is three bf16 numbers (hi, mid, lo: 8 bits each, every one rounded to nearest, and their sum is the number itself), so a product
// is nine products of bf16 numbers, each exact in float32.  Six are taken; what is left out (mid lo, lo mid, lo lo) is below 2^-26 of the product, a quarter of
// what rounding it to float32 would do.  tcgen05.mma adds to its accumulator without rounding to nearest, so an accumulator takes 64 k only, the
// small products first; the tiles of 64 k are added in registers by ordinary float32 additions, in k's order within a group (a fixed part of K), the groups in
// order.  How K is cut into groups follows N and K alone and every column of a tile is worked out alike, so a row's result does not depend on how many
// other rows there are, nor on the tile's width or on how many CTAs share a tile.
// Error against 64 bits (2-norm, rows of normal numbers; in brackets the chains of float32 multiply-adds of gemm_simple.cu): K 64 0.74e-7 (0.85), 1,024
// 0.97e-7 (4.1; with few weight rows 1.05, 2.1), 3,072 1.1e-7 (3.6), 9,728 1.3e-7 (6.3).  With 128 k an accumulator the second stage's small
// products meet a large sum: 5.9e-7.
//
// Numbers that three bf16 numbers cannot hold (not finite, above bf16's range, or below 2^-110 with bits below its range) are noticed on the way:
// the outputs of a row of x or of w that has one are worked out by float32 multiply-adds instead (gf_dot).  So are a token's 128
// outputs of a tile where a sum is not finite: parts of huge numbers can multiply to infinities of both signs where the numbers' products give one, or a finite sum.
// 333 tokens by 4,096 rows of 1,024, 33 us: 58 with one such number in x, or in w; 697 with one in every row of x.  16 by 2,560 of 9,728, 54 us: 80, 95 and 265 (sums that
// overflow everywhere cost as much as bad rows everywhere).  (By a chain of K in one thread an output, and 128 weight rows for one of them: 110, 6,730, 6,750; 2,450, 10,700, 21,400.)
//
// A CTA has 128 weight rows (the MMA's M) and `width` tokens (N).  Its warps fetch the next 64 k of both operands (16-byte loads, in registers
// while the MMAs of the k ahead run), split them into the six planes of a stage in shared memory (128-byte swizzle), then add the accumulator of the
// stage that became free; one warp hands a stage's 24 MMAs over.  Few tokens: 16 or 32 a tile, one stage, two CTAs an SM, bound by a stage's chain of
// latencies (4,500 clocks for two CTAs' 64 KB of weights).  Many: up to 128 a tile, two stages, one CTA an SM, bound by the splitting: about 14
// instructions a pair of numbers, 2,900 clocks a stage of 128 + 112 rows where its MMAs run for 1,360.
// The groups of a tile may be dealt over the CTAs of a cluster, which add their sums through distributed shared memory.
// Measured on B200 (gemm_simple.cu before): 333 tokens by 4,096 rows of 1,024 30 us (81), 6,144 of 1,024 31 (107), 1,024 of 3,072 29 (108), 19,456 of
// 2,560 282 (790), 2,560 of 9,728 138 (615); 16 tokens by 6,144 of 1,024 15 (34), 2,560 of 9,728 53 (133).
#define MB_LIB "gemm_f32"
#define MB_LIB_ID 26
#include "tc_common.cuh"
#include "launch.cuh"

#define GF_BM 128
#define GF_BK 64
#define GF_THREADS 512

struct GfTrue { static constexpr bool value = true; };
struct GfFalse { static constexpr bool value = false; };

template <int BN, int STAGES>
struct GfTile {
    static constexpr int A_PLANE = GF_BM * GF_BK * 2, B_PLANE = BN * GF_BK * 2, STAGE = 3 * (A_PLANE + B_PLANE);
    static constexpr int SUMS = GF_BM * BN;                         // numbers of one group's tile on its way to the cluster
    static constexpr int SMEM = STAGES * STAGE + 1024;
    // Warps that fetch and split, two rows of 64 numbers a round (16 lanes of 16 bytes a row).  With two stages the last warp hands the MMAs over instead: it
    // stands where it does so while they run.  With one stage everyone waits for them.
    static constexpr int PUTTERS = STAGES > 1 ? 15 : 16;
    static constexpr int ROUNDS = (GF_BM / 2 + BN / 2 + PUTTERS - 1) / PUTTERS, CW = BN / 4;   // rounds of rows a warp; columns a warp adds up
    static constexpr bool PARK = CW > 16;                           // the finished groups' sums wait in tensor memory, not in registers
    static constexpr int USED = (STAGES + (PARK ? 1 : 0)) * BN;
    static constexpr uint32_t COLS = USED <= 32 ? 32 : USED <= 64 ? 64 : USED <= 128 ? 128 : USED <= 256 ? 256 : 512;
    static_assert(A_PLANE == B_PLANE || STAGES == 1, "round 4 is of both kinds");
    static_assert(2 * SUMS * 4 <= STAGES * STAGE, "two groups' sums fit where the stages were");
};

template <int N> __device__ __forceinline__ void gf_tmem_ld(uint32_t taddr, float* v);
template <> __device__ __forceinline__ void gf_tmem_ld<16>(uint32_t taddr, float* v) { tmem_ld16(taddr, v); }
template <> __device__ __forceinline__ void gf_tmem_ld<8>(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void gf_tmem_st16(uint32_t taddr, const float* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]),
          "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Two numbers as three pairs of bf16 numbers.  What the third pair cannot hold shows in the low halves of `left`.
__device__ __forceinline__ void gf_split(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo, uint32_t& left) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const float ra = a - __uint_as_float(hi << 16), rb = b - __uint_as_float(hi & 0xffff0000u);
    const __nv_bfloat162 m = __floats2bfloat162_rn(ra, rb);
    mid = *reinterpret_cast<const uint32_t*>(&m);
    const uint32_t la = __float_as_uint(ra - __uint_as_float(mid << 16)), lb = __float_as_uint(rb - __uint_as_float(mid & 0xffff0000u));
    lo = __byte_perm(la, lb, 0x7632);
    left |= la | lb;
}

__device__ __forceinline__ void gf_st(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
// Four numbers of a row into its three planes.
template <int PLANE> __device__ __forceinline__ void gf_put(uint32_t at, const float4& v, uint32_t& left) {
    uint32_t h0, h1, m0, m1, l0, l1;
    gf_split(v.x, v.y, h0, m0, l0, left);
    gf_split(v.z, v.w, h1, m1, l1, left);
    gf_st(at, h0, h1);
    gf_st(at + PLANE, m0, m1);
    gf_st(at + 2 * PLANE, l0, l1);
}

// A row of x times a row of w by float32 multiply-adds, by a warp: a lane four k of every 128, the lanes' sums in a tree.  (One output at a
// time: what a call may touch is taken from the kernel around it.  4 x 4 of them a call made the kernel 2 to 10% slower, for 340 us of the 697 above.)
__device__ __noinline__ float gf_dot(const float* x, const float* w, int K) {
    float sum = 0.0f;
#pragma unroll 4
    for (int k = 4 * (threadIdx.x & 31); k < K; k += 128) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        sum = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// Whether all numbers of a row split: asked by a warp.
__device__ __noinline__ bool gf_splits(const float* row, int K) {
    uint32_t left = 0;
    for (int k = 4 * (threadIdx.x & 31); k < K; k += 128) {
        const float4 v = *reinterpret_cast<const float4*>(row + k);
        uint32_t hi, mid, lo;
        gf_split(v.x, v.y, hi, mid, lo, left);
        gf_split(v.z, v.w, hi, mid, lo, left);
    }
    return __all_sync(0xffffffffu, (left & 0xffffu) == 0);
}

__device__ __forceinline__ bool gf_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// The thread's number, asked for once more: what is worked out from it behind the loop then takes no registers in the loop, which has none to spare (with the flags'
// places from the first one 333 tokens by 4,096 rows of 1,024 took 30.6 us for 29.3).
__device__ __forceinline__ int gf_thread() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

__device__ __forceinline__ uint32_t gf_peer(const void* p, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}

// groups: parts of K whose sums are chains of their own, group_chunks stages each (the last may have fewer or none); splits CTAs of a cluster (along z)
// take groups / splits each: one or two, or all with one CTA.
template <int BN, int STAGES, bool ACC>
__global__ void __launch_bounds__(GF_THREADS, STAGES == 1 ? 2 : 1) gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                                                                                   int T, int N, int K, int width, int groups, int group_chunks,
                                                                                   int* __restrict__ error_flag) {
    typedef GfTile<BN, STAGES> S;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[STAGES], done[STAGES];               // a stage is filled (and its accumulator read); its MMAs are done
    __shared__ uint32_t tmem_slot;
    __shared__ int bad_any;                                       // something is flagged, or a sum is not finite
    __shared__ uint8_t bad_x[BN], bad_w[GF_BM];                   // tokens and weight rows with a number that does not split, in this CTA's k
    __shared__ uint8_t all_x[BN], all_w[GF_BM];                   // in all of it: 1; 2: a token of this CTA's with a sum that is not finite
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * GF_BM, t0 = blockIdx.y * width, splits = gridDim.z, rank = blockIdx.z;
    const int mine = groups / splits, chunks_all = (K + GF_BK - 1) / GF_BK;
    const int first = rank * mine * group_chunks, count = max(0, min(chunks_all, first + mine * group_chunks) - first);
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], S::PUTTERS); mbar_init(&done[s], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bad_any = 0;
    }
    if (tid < BN) bad_x[tid] = all_x[tid] = 0;
    if (tid < GF_BM) bad_w[tid] = all_w[tid] = 0;
    if (warp == 0) tmem_alloc<false>(&tmem_slot, S::COLS);
    // A warp's rounds: two rows each, of the weights (pairs of rows 0 to 63: rounds 0 to 3 and some of 4) or of x.  No round but the last few is behind a
    // branch, so that several are worked on side by side: a pair past the last one is the last one once more (the same numbers to the same place), and a row that is
    // not there repeats the last that is (nobody stores what comes of it).
    const int j = lane & 15, last_pair = GF_BM / 2 + width / 2 - 1;
    float4 p[S::ROUNDS];
    uint32_t left_w = 0, left[S::ROUNDS - 4];
    int at[S::ROUNDS], put[STAGES > 1 ? S::ROUNDS : 1];           // the row's number in its matrix; where its numbers go in a stage
    int k = first * GF_BK + 4 * j;                                // of the numbers on their way
    auto pair_of = [&](int i) { return STAGES > 1 ? min(warp + S::PUTTERS * i, last_pair) : warp + S::PUTTERS * i; };
    auto of_w = [&](int i) { return i < 4 || (STAGES > 1 && i == 4 && pair_of(4) < GF_BM / 2); };
#pragma unroll
    for (int i = 0; i < S::ROUNDS; ++i) {
        const int r = (pair_of(i) & (GF_BM / 2 - 1)) * 2 + (lane >> 4);
        at[i] = of_w(i) ? min(n0 + r, N - 1) : min(t0 + r, T - 1);
        if (STAGES > 1 || i == 0) put[i] = (of_w(i) ? 0 : 3 * S::A_PLANE) + r * 128 + ((((j >> 1) ^ r) & 7) << 4) + ((j & 1) << 3);
        if (i >= 4) left[i - 4] = 0;
    }
    static_assert(4 * S::PUTTERS <= GF_BM / 2 && 5 * S::PUTTERS >= GF_BM / 2 && (STAGES > 1 || (4 * S::PUTTERS == GF_BM / 2 && S::ROUNDS == 5)), "round 4 is where the weights' rows end");
    auto put_at = [&](int i) { return STAGES > 1 ? put[STAGES > 1 ? i : 0] : put[0] + (i < 4 ? i * 2 * S::PUTTERS * 128 : 3 * S::A_PLANE); };
    auto load = [&](int i, bool there) {
        p[i] = there ? *reinterpret_cast<const float4*>((of_w(i) ? w : x) + (size_t)at[i] * K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    // the weights of stages ahead on their way from HBM to L2: a row's 256 bytes of a stage are two lines
    constexpr int AHEAD = 3;
    const float* next = w + (size_t)min(n0 + (tid >> 1), N - 1) * K + (tid & 1) * (GF_BK / 2);
    auto ahead = [&](int c) {
        const int k2 = (first + c) * GF_BK;
        if (tid < 2 * GF_BM && c < count && k2 + (tid & 1) * (GF_BK / 2) < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(next + k2));
    };
    for (int c = 1; c < AHEAD; ++c) ahead(c);
    if (count > 0) {                                              // (weights are written by no kernel)
#pragma unroll
        for (int i = 0; i < S::ROUNDS; ++i)
            if (of_w(i)) load(i, k < K);
    }
    PDL_ENTER();
    x = pdl_fresh(x);
    if (count > 0) {
#pragma unroll
        for (int i = 0; i < S::ROUNDS; ++i)
            if (!of_w(i)) load(i, k < K);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(width >> 3) << 17) | ((uint32_t)(GF_BM >> 4) << 24);
    const int quarter = warp & 3, c0 = (warp >> 2) * S::CW;       // this warp's lanes and columns of an accumulator
    constexpr int STEP = S::CW < 16 ? S::CW : 16;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, parked = lanes + STAGES * BN;
    float cur[S::CW], held[S::PARK ? 1 : S::CW];                  // the group's chain so far; the groups before it
#pragma unroll
    for (int i = 0; i < S::CW; ++i) cur[i] = 0.0f;
    bool folded = false;
    auto before = [&](int i, float* v) {                          // the groups before, columns i .. i + STEP - 1
        if (S::PARK) {
            if (folded) gf_tmem_ld<STEP>(parked + i, v);
            else {
#pragma unroll
                for (int e = 0; e < STEP; ++e) v[e] = 0.0f;
            }
        } else {
#pragma unroll
            for (int e = 0; e < STEP; ++e) v[e] = folded ? held[S::PARK ? 0 : i + e] : 0.0f;
        }
    };
    const int in = quarter * 32 + lane;
    float* sums = reinterpret_cast<float*>(smem);                 // on the way to the cluster: [group][token][weight row], where the stages were
    int until = group_chunks;                                     // stages to add until the group ends
    bool ok = true;
    auto add = [&](int c) {                                       // the accumulator of stage c, once its MMAs are done
        if (ok && !mbar_wait(&done[c % STAGES], (c / STAGES) & 1)) { atomicExch(error_flag, 31); ok = false; }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int i = 0; i < S::CW; i += STEP) {
            if (c0 + i >= width) continue;
            float v[STEP];
            gf_tmem_ld<STEP>(lanes + (c % STAGES) * BN + i, v);
#pragma unroll
            for (int e = 0; e < STEP; ++e) cur[i + e] += v[e];
        }
        if (--until == 0 && c + 1 < count) {
#pragma unroll
            for (int i = 0; i < S::CW; i += STEP) {
                if (c0 + i >= width) continue;
                float v[STEP];
                before(i, v);
#pragma unroll
                for (int e = 0; e < STEP; ++e) { v[e] += cur[i + e]; cur[i + e] = 0.0f; }
                if (S::PARK) gf_tmem_st16(parked + i, v);
                else {
#pragma unroll
                    for (int e = 0; e < STEP; ++e) held[S::PARK ? 0 : i + e] = v[e];
                }
            }
            folded = true;
            until = group_chunks;
        }
    };
    // whole: the next stage lies within K.  (A row's next numbers are asked for as soon as its present ones are put away.)
    auto stage = [&](int c, auto whole) {
        const uint32_t to = smem_u32(smem) + (c % STAGES) * S::STAGE;
        k += GF_BK;
        const bool more = decltype(whole)::value || (c + 1 < count && k < K);
#pragma unroll
        for (int i = 0; i < S::ROUNDS; ++i) {
            if (STAGES > 1 && i >= 6 && S::PUTTERS * i > last_pair) continue;   // (the same for every warp)
            uint32_t& l = i < 4 ? left_w : left[i < 4 ? 0 : i - 4];
            if (S::A_PLANE == S::B_PLANE || i < 4) gf_put<S::A_PLANE>(to + put_at(i), p[i], l);
            else gf_put<S::B_PLANE>(to + put_at(i), p[i], l);
            load(i, more);
        }
    };
    const uint32_t elected = elect_one();
    auto issue = [&](int c) {                                     // a whole warp: a stage's MMAs
        const int st = c % STAGES;
        if (ok && !mbar_wait(&full[st], (c / STAGES) & 1)) { atomicExch(error_flag, 32); ok = false; }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = smem_u32(smem) + st * S::STAGE, d = tmem + (uint32_t)(st * BN);
        const uint64_t da = umma_desc(a), db = umma_desc(a + 3 * S::A_PLANE);
        constexpr uint64_t AP = S::A_PLANE >> 4, BP = S::B_PLANE >> 4;
        // the smallest products first: each addition drops what lies below the accumulator's last bit
#pragma unroll
        for (int kk = 0; kk < GF_BK / 16; ++kk) {
            umma_bf16(d, da + 2 * AP + 2 * kk, db + 2 * kk, idesc, kk > 0 ? 1u : 0u, elected);
            umma_bf16(d, da + 2 * kk, db + 2 * BP + 2 * kk, idesc, 1u, elected);
            umma_bf16(d, da + AP + 2 * kk, db + BP + 2 * kk, idesc, 1u, elected);
        }
#pragma unroll
        for (int kk = 0; kk < GF_BK / 16; ++kk) {
            umma_bf16(d, da + AP + 2 * kk, db + 2 * kk, idesc, 1u, elected);
            umma_bf16(d, da + 2 * kk, db + BP + 2 * kk, idesc, 1u, elected);
        }
#pragma unroll
        for (int kk = 0; kk < GF_BK / 16; ++kk) umma_bf16(d, da + 2 * kk, db + 2 * kk, idesc, 1u, elected);
        umma_commit(&done[st], elected);
        __syncwarp();
    };
    const int role = __shfl_sync(0xffffffffu, warp, 0);           // (known to be the same in a whole warp)
    if (role == S::PUTTERS) {
        for (int c = 0; c < count; ++c) {
            issue(c);
            if (c > 0) add(c - 1);                                // (before its accumulator is written again)
        }
        if (count > 0) add(count - 1);
    } else {
        for (int c = 0; c < count; ++c) {
            ahead(c + AHEAD);
            if (c >= STAGES) add(c - STAGES);
            if (STAGES > 1 && c + 1 < count && (first + c + 2) * GF_BK <= K) stage(c, GfTrue());
            else stage(c, GfFalse());
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[c % STAGES])) : "memory");
            if (STAGES == 1 && role == 0) issue(c);
        }
        for (int c = max(0, count - STAGES); c < count; ++c) add(c);
    }
    const int tid2 = gf_thread(), warp2 = tid2 >> 5, lane2 = tid2 & 31, in2 = (warp2 & 3) * 32 + lane2;
    auto pair2 = [&](int i) { return STAGES > 1 ? min(warp2 + S::PUTTERS * i, last_pair) : warp2 + S::PUTTERS * i; };
    auto of_w2 = [&](int i) { return i < 4 || (STAGES > 1 && i == 4 && pair2(4) < GF_BM / 2); };
#pragma unroll
    for (int i = 0; i < S::ROUNDS; ++i) {
        if (((i < 4 ? left_w : left[i < 4 ? 0 : i - 4]) & 0xffffu) == 0) continue;
        (of_w2(i) ? bad_w : bad_x)[(pair2(i) & (GF_BM / 2 - 1)) * 2 + (lane2 >> 4)] = 1;      // (of the weights: one of four rows)
        bad_any = 1;
    }
    bool finite = true;
#pragma unroll
    for (int i = 0; i < S::CW; i += STEP) {
        if (c0 + i >= width) continue;
        float v[STEP];
        before(i, v);
        if (splits == 1) {
#pragma unroll
            for (int e = 0; e < STEP; ++e) {
                cur[i + e] = v[e] + cur[i + e];
                finite &= gf_finite(cur[i + e]);
            }
        } else {
#pragma unroll
            for (int e = 0; e < STEP; ++e) {
                float* to = sums + (c0 + i + e) * GF_BM + in2;
                if (mine > 1) { to[0] = folded ? v[e] : cur[i + e]; to[S::SUMS] = folded ? cur[i + e] : 0.0f; }
                else to[0] = cur[i + e];
            }
        }
    }
    if (!finite) bad_any = 1;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                                              // tensor memory has been read, and everyone has said what was bad
    if (warp2 == 0) tmem_free<false>(tmem, S::COLS);
            auto store = [&](auto flagged) {
                float* to = out + (size_t)(t0 + c0) * N + n0 + in2;
                const int rows = min(width, T - t0) - c0;
    #pragma unroll
                for (int i = 0; i < S::CW; i += 8) {
                    float old[8];
    #pragma unroll
                    for (int e = 0; e < 8; ++e) old[e] = ACC && i + e < rows ? to[(size_t)(i + e) * N] : 0.0f;
    #pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        if (i + e >= rows || (decltype(flagged)::value && (all_w[in2] | all_x[c0 + i + e]))) continue;
                        to[(size_t)(i + e) * N] = ACC ? old[e] + cur[i + e] : cur[i + e];
                    }
                }
            };
    bool any = bad_any != 0;
    if (splits == 1 && !any) {
        if (n0 + in2 < N) store(GfFalse());
        return;
    }
    if (any) {
        for (int r = warp2; r < GF_BM; r += GF_THREADS / 32)
            if (bad_w[r] != 0 && gf_splits(w + (size_t)min(n0 + r, N - 1) * K, K)) bad_w[r] = 0;
        __syncthreads();
    }
    if (splits > 1) {
        cluster_sync();
        for (int z = 0; z < splits; ++z) {
            int v;
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(gf_peer(&bad_any, z)) : "memory");
            any |= v != 0;
        }
    }
    if (any) {
        if (tid2 < BN + GF_BM) {
            const uint8_t* own = tid2 < BN ? bad_x + tid2 : bad_w + (tid2 - BN);
            uint32_t all = splits == 1 ? *own : 0;
            for (int z = 0; splits > 1 && z < splits; ++z) {
                uint32_t u;
                asm volatile("ld.shared::cluster.u8 %0, [%1];" : "=r"(u) : "r"(gf_peer(own, z)) : "memory");
                all |= u;
            }
            (tid2 < BN ? all_x + tid2 : all_w + (tid2 - BN))[0] = (uint8_t)all;
        }
        __syncthreads();
        if (!finite && all_w[in2] == 0) {                         // (with one CTA a tile; several see the whole sum only below)
#pragma unroll
            for (int i = 0; i < S::CW; ++i)
                if (c0 + i < width && !gf_finite(cur[i]) && all_x[c0 + i] == 0) all_x[c0 + i] = 2;
        }
        __syncthreads();
    }
    if (splits == 1) {
        if (n0 + in2 < N) {
            store(GfTrue());
        }
    } else {
        bool odd = false;
        for (int idx = rank * GF_THREADS + tid2; idx < width * (GF_BM / 4); idx += splits * GF_THREADS) {
            const int t = idx / (GF_BM / 4), n = idx % (GF_BM / 4) * 4;      // (a warp a token)
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int z = 0; z < splits; ++z) {
                const uint32_t peer = gf_peer(sums + t * GF_BM + n, z);
                for (int g = 0; g < mine; ++g) {
                    float4 p;
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w) : "r"(peer + (uint32_t)(g * S::SUMS * 4)) : "memory");
                    v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
                }
            }
            if (__any_sync(0xffffffffu, !(gf_finite(v[0]) && gf_finite(v[1]) && gf_finite(v[2]) && gf_finite(v[3])))) {
                bool mine_is = false;
#pragma unroll
                for (int e = 0; e < 4; ++e) mine_is |= !gf_finite(v[e]) && all_w[n + e] == 0;
                if (__any_sync(0xffffffffu, mine_is)) {
                    odd = true;
                    if (all_x[t] == 0) all_x[t] = 2;
                }
            }
            if (t0 + t >= T || n0 + n >= N) continue;
            float* to = out + (size_t)(t0 + t) * N + n0 + n;
            if (!any && !odd && n0 + n + 4 <= N && (N & 3) == 0 && ((uintptr_t)out & 15) == 0) {
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (ACC) {
                    const float4 old = *reinterpret_cast<const float4*>(to);
                    r = make_float4(old.x + v[0], old.y + v[1], old.z + v[2], old.w + v[3]);
                }
                *reinterpret_cast<float4*>(to) = r;
            } else {
                for (int e = 0; e < 4 && n0 + n + e < N; ++e)
                    if ((all_x[t] | all_w[n + e]) == 0) to[e] = ACC ? to[e] + v[e] : v[e];
            }
        }
        cluster_sync();                                           // nobody leaves while its sums are read
        any = __syncthreads_or(any || odd) != 0;
    }
    if (!any) return;
    // The flagged ones, an output a warp of all the tile's CTAs: tokens with all weight rows, then weight rows with the other tokens.  (Tokens that this CTA alone
    // knows of: its warps, and the flagged weight rows are among the others'.)
    const int tokens = min(width, T - t0), weights = min(GF_BM, N - n0), me = rank * (GF_THREADS / 32) + warp2, warps = splits * (GF_THREADS / 32);
    for (int a = 0; a < tokens + weights; ++a) {
        const bool token = a < tokens;
        const int flag = token ? all_x[a] : all_w[a - tokens];
        if (flag == 0) continue;
        for (int b = flag == 2 ? warp2 : me; b < (token ? weights : tokens); b += flag == 2 ? GF_THREADS / 32 : warps) {
            const int t = token ? a : b, n = token ? b : a - tokens;
            if (token ? flag == 2 && all_w[n] != 0 : all_x[t] == 1) continue;
            const float v = gf_dot(x + (size_t)(t0 + t) * K, w + (size_t)(n0 + n) * K, K);
            float* to = out + (size_t)(t0 + t) * N + n0 + n;
            if (lane2 == 0) *to = ACC ? *to + v : v;
        }
    }
}

// Parts of K whose sums are chains of their own, by N alone (a row's result must not follow the batch): with few weight rows more CTAs share a tile.
#define GF_FEW_ROWS 3072
static int gf_groups(int N) { return N <= GF_FEW_ROWS ? 8 : 4; }

template <int BN, int STAGES, bool ACC>
static int gf_launch(const float* x, const float* w, float* out, int T, int N, int K, int width, int splits, int* error_flag, cudaStream_t s) {
    typedef GfTile<BN, STAGES> S;
    auto kernel = gemm_f32_kernel<BN, STAGES, ACC>;
    static LaunchSmem smem;
    const int rc = smem.allow(kernel, S::SMEM);
    if (rc) return rc;
    const int groups = gf_groups(N), chunks = (K + GF_BK - 1) / GF_BK;
    const dim3 grid((N + GF_BM - 1) / GF_BM, (T + width - 1) / width, splits);
    if (grid.y > 65535) return MB_ERR_BAD_SIZE;
    return launch_kernel(kernel, grid, GF_THREADS, S::SMEM, s, splits, x, w, out, T, N, K, width, groups, (chunks + groups - 1) / groups, error_flag);
}

// x float32 [T, K], w float32 [N, K], out float32 [T, N]; accumulate: out +=.  K a multiple of 4, x and w 16-byte aligned.  width: tokens a tile (a multiple
// of 16 up to 128; up to 32 by the kernel for few tokens); splits: CTAs a tile, 1, or such that each takes one or two of the 4 (more than 3,072 weight rows)
// or 8 parts of K.  Neither changes a bit of the result.
MB_API int mb_gemm_f32(const float* x, const float* w, float* out, int T, int N, int K, int accumulate, int width, int splits, int* error_flag, cudaStream_t s) {
    if (T <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 != 0 || (((uintptr_t)x | (uintptr_t)w) & 15) != 0 || width < 16 || width > 128 || width % 16 != 0) return MB_ERR_BAD_SIZE;
    const int groups = gf_groups(N);
    if (splits != 1 && splits != groups && splits * 2 != groups) return MB_ERR_BAD_SIZE;
    if (width <= 32) return accumulate ? gf_launch<32, 1, true>(x, w, out, T, N, K, width, splits, error_flag, s) : gf_launch<32, 1, false>(x, w, out, T, N, K, width, splits, error_flag, s);
    return accumulate ? gf_launch<128, 2, true>(x, w, out, T, N, K, width, splits, error_flag, s) : gf_launch<128, 2, false>(x, w, out, T, N, K, width, splits, error_flag, s);
}
