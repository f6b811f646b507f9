// Matrix product on the CUDA cores: out[t, n] = sum_k x[t, k] * w[n, k], float32 accumulate.  Every output is one fixed chain (or,
// for few weight rows, a fixed number of chains added in order) of fused multiply-adds over increasing k that depends on N and K
// alone, so a row's result does not depend on how many other rows the batch holds.  This is the 32-bit path's product where rows of K
// numbers are not whole 16-byte units (gemm_f32.cu has the others) and the plain twin the tensor-core kernels are tested against.  The reference's
// counterpart is its warp-per-row kernel (crates/cuda/src/kernels.cu:73-116).
//
// Bound by the multiply-adds (128 a clock and SM: 72 TFLOP/s at 1.9 GHz) and by shared memory: a 16-byte load of a warp takes four of its
// cycles, so a step over k with an 8 x 8 tile a thread takes 16 of them for 16 cycles of multiply-adds (with 4 x 8: 12 for 8).  The 64 sums
// lie in registers as pairs along n, so that one instruction does two multiply-adds (fma.rn.f32x2, each rounded as fmaf rounds); tiles
// arrive by 16-byte loads a k-step ahead, in registers, and lie in shared memory by k, in two buffers: one barrier a k-step.
#define MB_LIB "gemm_simple"
#define MB_LIB_ID 6
#include "common.cuh"
#include "launch.cuh"

#define GS_BK 16

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 both(float a) { f32x2 r; asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a)); return r; }
__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ float2 halves(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }

// Four numbers of a row from k on, zeros behind the row's end (and for a row that is not there).
__device__ __forceinline__ float4 load4(const float* p, bool there, int k, int K, bool vec) {
    if (!there || k >= K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (vec) return *reinterpret_cast<const float4*>(p + k);
    return make_float4(p[k], k + 1 < K ? p[k + 1] : 0.0f, k + 2 < K ? p[k + 2] : 0.0f, k + 3 < K ? p[k + 3] : 0.0f);
}
__device__ __forceinline__ float4 load4(const bf16* p, bool there, int k, int K, bool vec) {
    if (!there || k >= K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (vec) {
        const uint2 u = *reinterpret_cast<const uint2*>(p + k);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
        return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
    }
    return make_float4(to_f32(p[k]), k + 1 < K ? to_f32(p[k + 1]) : 0.0f, k + 2 < K ? to_f32(p[k + 2]) : 0.0f, k + 3 < K ? to_f32(p[k + 3]) : 0.0f);
}

// BT tokens x BN weight rows a block, TT x 8 a thread, KG groups of threads that each take one part of k.
template <int BT, int BN, int TT, int KG>
struct Tile {
    static constexpr int GROUP = (BT / TT) * (BN / 8), THREADS = GROUP * KG;
    static constexpr int LX = BT + 4, LW = BN + 4;              // padded rows: 16-byte aligned, neighbours in other banks
    static constexpr int STAGE = GS_BK * (LX + LW);             // floats of one buffer of one group
    static constexpr int FLOATS = 2 * KG * STAGE > KG * BT * BN ? 2 * KG * STAGE : KG * BT * BN;
    static_assert((BT * 4) % GROUP == 0 && (BN * 4) % GROUP == 0, "whole rounds of 16-byte loads");
};

template <typename TX, typename TW, typename TO, bool ACC, int BT, int BN, int TT, int KG>
__global__ void __launch_bounds__(Tile<BT, BN, TT, KG>::THREADS) gemm_simple_kernel(const TX* __restrict__ x, const TW* __restrict__ w,
                                                                                    TO* __restrict__ out, int T, int N, int K, int vec) {
    typedef Tile<BT, BN, TT, KG> S;
    constexpr int XL = BT * 4 / S::GROUP, WL = BN * 4 / S::GROUP;
    PDL_ENTER();
    x = pdl_fresh(x);
    extern __shared__ __align__(16) float smem[];
    const int group = KG > 1 ? threadIdx.x / S::GROUP : 0, id = threadIdx.x - group * S::GROUP;
    float* mine = smem + group * 2 * S::STAGE;
    const int t0 = blockIdx.y * BT, n0 = blockIdx.x * BN;
    const int tx = id % (BN / 8), ty = id / (BN / 8);           // tx: n direction (columns 4 tx.. and BN/2 + 4 tx..), ty: t direction (likewise, in runs of four)
    // k in whole steps over the groups: which part a group takes depends on K alone
    const int steps_all = (K + GS_BK - 1) / GS_BK, steps = (steps_all + KG - 1) / KG;
    const int k_first = group * steps * GS_BK;
    f32x2 acc[TT][4];
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    float4 px[XL], pw[WL];
    auto fetch = [&](int step) {
        const int k = k_first + step * GS_BK + (id & 3) * 4;
#pragma unroll
        for (int r = 0; r < XL; ++r) {
            const int t = t0 + ((id + r * S::GROUP) >> 2);
            px[r] = load4(x + (size_t)t * K, t < T, k, K, vec);
        }
#pragma unroll
        for (int r = 0; r < WL; ++r) {
            const int n = n0 + ((id + r * S::GROUP) >> 2);
            pw[r] = load4(w + (size_t)n * K, n < N, k, K, vec);
        }
    };
    auto put = [&](int step) {
        float* sx = mine + (step & 1) * S::STAGE + (id & 3) * 4 * S::LX;
        float* sw = mine + (step & 1) * S::STAGE + GS_BK * S::LX + (id & 3) * 4 * S::LW;
#pragma unroll
        for (int r = 0; r < XL; ++r) {
            float* d = sx + ((id + r * S::GROUP) >> 2);
            d[0] = px[r].x; d[S::LX] = px[r].y; d[2 * S::LX] = px[r].z; d[3 * S::LX] = px[r].w;
        }
#pragma unroll
        for (int r = 0; r < WL; ++r) {
            float* d = sw + ((id + r * S::GROUP) >> 2);
            d[0] = pw[r].x; d[S::LW] = pw[r].y; d[2 * S::LW] = pw[r].z; d[3 * S::LW] = pw[r].w;
        }
    };
    fetch(0);
    put(0);
    __syncthreads();
    for (int step = 0; step < steps; ++step) {
        if (step + 1 < steps) fetch(step + 1);
        const float* sx = mine + (step & 1) * S::STAGE + ty * 4;
        const float* sw = mine + (step & 1) * S::STAGE + GS_BK * S::LX + tx * 4;
#pragma unroll
        for (int kk = 0; kk < GS_BK; ++kk) {
            float a[TT];
#pragma unroll
            for (int i = 0; i < TT; i += 4) *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(sx + kk * S::LX + i / 4 * (BT * 4 / TT));
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(sw + kk * S::LW), b1 = *reinterpret_cast<const ulonglong2*>(sw + kk * S::LW + BN / 2);
#pragma unroll
            for (int i = 0; i < TT; ++i) {
                const f32x2 aa = both(a[i]);
                fma2(acc[i][0], aa, b0.x); fma2(acc[i][1], aa, b0.y); fma2(acc[i][2], aa, b1.x); fma2(acc[i][3], aa, b1.y);
            }
        }
        if (step + 1 < steps) put(step + 1);
        __syncthreads();
    }
    float sum[TT][8];
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 v = halves(acc[i][j]); sum[i][2 * j] = v.x; sum[i][2 * j + 1] = v.y; }
    if (KG > 1) {
        // the groups' sums meet in shared memory; group 0 adds them in the groups' order
        if (group > 0) {
#pragma unroll
            for (int i = 0; i < TT; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) smem[(group * TT * 8 + i * 8 + j) * S::GROUP + id] = sum[i][j];
        }
        __syncthreads();
        if (group > 0) return;
        for (int g = 1; g < KG; ++g)
#pragma unroll
            for (int i = 0; i < TT; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) sum[i][j] += smem[(g * TT * 8 + i * 8 + j) * S::GROUP + id];
    }
#pragma unroll
    for (int i = 0; i < TT; ++i) {
        const int t = t0 + i / 4 * (BT * 4 / TT) + ty * 4 + (i & 3);
        if (t >= T) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + (j >> 2) * (BN / 2) + tx * 4 + (j & 3);
            if (n >= N) continue;
            const size_t at = (size_t)t * N + n;
            if (ACC) out[at] = from_f32<TO>(to_f32(out[at]) + sum[i][j]);
            else out[at] = from_f32<TO>(sum[i][j]);
        }
    }
}

template <typename TX, typename TW, typename TO, bool ACC, int BT, int BN, int TT, int KG>
static int launch_tile(const void* x, const void* w, void* out, int T, int N, int K, int vec, cudaStream_t s) {
    typedef Tile<BT, BN, TT, KG> S;
    const size_t smem = S::FLOATS * sizeof(float);
    auto kernel = gemm_simple_kernel<TX, TW, TO, ACC, BT, BN, TT, KG>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    dim3 grid((N + BN - 1) / BN, (T + BT - 1) / BT);
    return launch_kernel(kernel, grid, S::THREADS, smem, s, 0, (const TX*)x, (const TW*)w, (TO*)out, T, N, K, vec);
}

// A block's tile is worked on by groups that cut k, so that a few hundred tokens put enough warps on every SM: two groups of two warps on 64 x 64, and
// with few weight rows eight half warps on 32 x 32 (333 tokens by 4,096 + 6,144 weight rows of 1,024: 190 us with two groups, 346 us with one; by 1,024
// rows of 2,048 and 3,072: 206 us).  The border lies in N alone (the order of a row's sums must not follow the batch).
#define GS_FEW_ROWS 3072

template <typename TX, typename TW, typename TO, bool ACC>
static int launch(const void* x, const void* w, void* out, int T, int N, int K, int vec, cudaStream_t s) {
    if (N <= GS_FEW_ROWS) return launch_tile<TX, TW, TO, ACC, 32, 32, 8, 8>(x, w, out, T, N, K, vec, s);
    return launch_tile<TX, TW, TO, ACC, 64, 64, 8, 2>(x, w, out, T, N, K, vec, s);
}

template <typename TX, typename TW, typename TO>
static int launch(const void* x, const void* w, void* out, int T, int N, int K, int accumulate, cudaStream_t s) {
    const int vec = K % 4 == 0 && ((uintptr_t)x) % (4 * sizeof(TX)) == 0 && ((uintptr_t)w) % (4 * sizeof(TW)) == 0;
    if (accumulate) return launch<TX, TW, TO, true>(x, w, out, T, N, K, vec, s);
    return launch<TX, TW, TO, false>(x, w, out, T, N, K, vec, s);
}

// x [T, K] (x_dtype), w [N, K] (w_dtype), out [T, N] (out_dtype); accumulate: out += (float32 out only).
MB_API int mb_gemm_simple(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                          int T, int N, int K, int accumulate, cudaStream_t s) {
    if (T <= 0 || N <= 0) return 0;
    if (K <= 0) return MB_ERR_BAD_SIZE;
    if (accumulate && out_dtype != MB_F32) return MB_ERR_BAD_DTYPE;
    if (x_dtype == MB_F32 && w_dtype == MB_F32 && out_dtype == MB_F32) return launch<float, float, float>(x, w, out, T, N, K, accumulate, s);
    if (x_dtype == MB_BF16 && w_dtype == MB_BF16 && out_dtype == MB_BF16) return launch<bf16, bf16, bf16>(x, w, out, T, N, K, accumulate, s);
    if (x_dtype == MB_BF16 && w_dtype == MB_BF16 && out_dtype == MB_F32) return launch<bf16, bf16, float>(x, w, out, T, N, K, accumulate, s);
    return MB_ERR_BAD_DTYPE;
}
