// The gated delta rule over prompt portions, 64 tokens at a time on the tensor cores (mma.sync), compiled for one head layout:
// -DQK_DIM (key channels, a multiple of 16 up to 128), -DV_SLICE (value channels a CTA of the walk takes: 16, 32 or 64).
//
// The recurrence (delta_rule.cu) per head:  S <- g S,  u = beta (v - S^T k),  S <- S + k u^T,  o = S^T q.  With S0 the state before
// a chunk of 64 tokens, G_i the sum of the log-decays of its tokens 0 .. i (per key channel), and the weighted products
//     A_ij = sum_c k_i[c] k_j[c] exp(G_i[c] - G_j[c])  (j < i),      P_ij = sum_c q_i[c] k_j[c] exp(G_i[c] - G_j[c])  (j <= i),
// unrolling it gives (Yang, Wang, Zhang, Shen, Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence Length")
//     (I + diag(beta) A) U = diag(beta) (V - K+ S0),   K+_i = exp(G_i) k_i,
//     O = Q+ S0 + P U,   Q+_i = exp(G_i) q_i,          S = exp(G_63) S0 + sum_j (exp(G_63 - G_j) k_j) u_j^T.
// prepare_kernel (a CTA per chunk and head, all of them side by side) makes what does not need the state: P, W = (I + diag(beta) A)^-1
// diag(beta) K+ and U0 = (I + diag(beta) A)^-1 diag(beta) V, by forward substitution over blocks of 16 tokens.  walk_kernel (a CTA per request,
// head and slice of value channels) walks the chunks in order and does only what the next chunk waits for: U = U0 - W S0 and S; it leaves U and
// each chunk's S0.  read_kernel (a CTA per chunk and head, side by side again) makes O and, where it has a whole head, its norm, weight and gate.
//
// Exactness.  Every exponent that is taken is of a non-positive number: with one decay per channel a block of 16 rows is worked out
// against a reference between it and the earlier rows (exp(G_i - R) exp(R - G_j), both at most 1), the lower half of a block's diagonal
// square against one in its middle, and the 8 x 8 squares left on the diagonal pair by pair.  Decays, sums, unit vectors, A, the inverses of the diagonal blocks, what
// the substitution adds up and the state are float32; where a float32 number has to be an operand of a product it is split into two bf16
// numbers (value = hi + lo) and the three larger products are taken, so that about 16 bits of it enter (of a block's inverse only what lies
// below its unit diagonal).
// Measured on B200, two prompts of 712 and 1,188 tokens, 20 heads of 128 x 128, a decay per channel: prepare 91 us (141 with a column of the substitution a
// thread), walk 65 (124 with the outputs made in it, 32 value channels a CTA and operands from shared memory on both sides), read 39 (with the norm, 12 us as a
// kernel of its own).
#define MB_LIB "delta_rule_chunked"
#define MB_LIB_ID 21
#include "common.cuh"
#include "launch.cuh"
#include "mma_helpers.cuh"
#include "tc_common.cuh"

#ifndef QK_DIM
#define QK_DIM 128
#endif
#ifndef V_SLICE
#define V_SLICE 64
#endif
static_assert(QK_DIM % 16 == 0 && QK_DIM >= 16 && QK_DIM <= 128, "key channels: a multiple of 16 up to 128");
static_assert(V_SLICE == 16 || V_SLICE == 32 || V_SLICE == 64, "a CTA takes 16, 32 or 64 value channels");

#define DQ QK_DIM
#define VS V_SLICE
#define CH 64
#define LOG2E 1.4426950408889634f
#define UNIT_EPS 1e-6f

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float softplus_f(float v) { return fmaxf(v, 0.0f) + log1pf(expf(-fabsf(v))); }
__device__ __forceinline__ float2 bf2(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }

__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 back = __bfloat1622float2(h);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = pack_bf16(x - back.x, y - back.y);
}
__device__ __forceinline__ void mma3(float* c, const uint32_t* ah, const uint32_t* al, uint32_t bh0, uint32_t bh1, uint32_t bl0, uint32_t bl1) {
    mma_bf16_16816(c, ah, bh0, bh1);
    mma_bf16_16816(c, al, bh0, bh1);
    mma_bf16_16816(c, ah, bl0, bl1);
}

// The same into three sums (added up at the end): three chains of products instead of one three times as long.
struct Sums3 {
    float hh[2][4], lh[2][4], hl[2][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) hh[n][e] = lh[n][e] = hl[n][e] = 0.0f;
    }
    __device__ __forceinline__ void add(const uint32_t* ah, const uint32_t* al, const uint32_t* bh, const uint32_t* bl) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            mma_bf16_16816(hh[n], ah, bh[2 * n], bh[2 * n + 1]);
            mma_bf16_16816(lh[n], al, bh[2 * n], bh[2 * n + 1]);
            mma_bf16_16816(hl[n], ah, bl[2 * n], bl[2 * n + 1]);
        }
    }
    __device__ __forceinline__ float at(int n, int e) const { return hh[n][e] + (lh[n][e] + hl[n][e]); }
};

// What a chunk and head hands over, every piece laid out as its reader holds it, so that one bulk copy (or a warp's 16-byte loads) brings it.  bf16
// planes, hi then lo: W transposed [DQ][LDW], K exp(G_63 - G) and Q+ [64][LDQ], P [64][LDW], rows padded against bank conflicts; S0 as row operands of
// (value channels x key channels): [dv / 16][DQ / 16][hi, lo][lane][8].  float32: U0 transposed [dv][64], its runs of eight tokens swapped by TURN0, 16 columns
// of it replaced by the walk with U as row operands (value channels x tokens): [dv / 16][4][hi, lo][lane][8] bf16; exp(G_63) [DQ].
#define LDQ (DQ + 8)
#define LDW (CH + 8)
#define WPLANE (DQ * LDW)
#define KPLANE (CH * LDQ)
#define PPLANE (CH * LDW)
#define AT_K (2 * WPLANE)
#define AT_Q (AT_K + 2 * KPLANE)
#define AT_P (AT_Q + 2 * KPLANE)
#define AT_S (AT_P + 2 * PPLANE)
#define CHUNK_BF16(dv) (AT_S + 2 * DQ * (dv))
#define CHUNK_F32(dv) (CH * (dv) + DQ)
#define TURN0(column) (8 * ((column) & 3))
#define KT (DQ / 16)                  // blocks of 16 key channels

// Where request r's chunks start among all chunks of the step (room is left for a partial chunk per request).
__device__ __forceinline__ int first_chunk(const int* cu_tokens, int first_req, int r) { return (cu_tokens[r] - cu_tokens[first_req]) / CH + (r - first_req); }

#define LDR (DQ + 8)                  // raw q and k rows in shared memory (bf16) and sums (float32): eight rows of four lanes meet all banks
#define LDG (DQ + 8)
#define LDL (CH + 8)                  // the matrix of the substitution, bf16 planes
#define LDD 20                        // its diagonal blocks, float32
#define PREP_SMEM(CHANNEL, dv) (2 * CH * LDR * 2 + ((CHANNEL) ? CH * LDG : CH) * 4 + 2 * CH * LDL * 2 + 4 * 16 * LDD * 4 + 4 * CH * 4 + CH * ((dv) + 8) * 2 + 16)
#define PREP_THREADS 256

template <bool CHANNEL>
__global__ void __launch_bounds__(PREP_THREADS, 2) prepare_kernel(
    const bf16* __restrict__ qkv, const bf16* __restrict__ b_rows, int b_stride, const bf16* __restrict__ a_rows, int a_stride,
    const float* __restrict__ rate_log, const float* __restrict__ dt_bias, const int* __restrict__ cu_tokens, int first_req,
    bf16* __restrict__ planes, float* __restrict__ floats, int H, int G, int dv, int a_vec) {
    PDL_ENTER();
    qkv = pdl_fresh(qkv); b_rows = pdl_fresh(b_rows); a_rows = pdl_fresh(a_rows);
    extern __shared__ __align__(128) uint8_t smem_raw[];
    bf16* sq = reinterpret_cast<bf16*>(smem_raw);              // [CH][LDR]
    bf16* sk = sq + CH * LDR;
    bf16* sL = sk + CH * LDR;                                  // [2][CH][LDL] hi, lo: -beta_i A_ij of earlier blocks; in a diagonal block its inverse less 1
    float* sD = reinterpret_cast<float*>(sL + 2 * CH * LDL);   // [4][16][LDD] beta_i A_ij of the diagonal blocks
    float* sG = sD + 4 * 16 * LDD;                             // [CH][LDG], or [CH] with one decay per head (log2 units)
    float* s_beta = sG + (CHANNEL ? CH * LDG : CH);
    float* s_fq = s_beta + CH;
    float* s_fk = s_fq + CH;
    float* s_qk = s_fk + CH;                                   // q_i . k_i as they are
    const int req = first_req + blockIdx.z, head = blockIdx.y;
    const int tok0 = cu_tokens[req] + blockIdx.x * CH;
    const int rows = min(CH, cu_tokens[req + 1] - tok0);
    if (rows <= 0) return;
    const int kh = head / (H / G), channels = 2 * G * DQ + H * dv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t2 = 2 * (lane & 3);
    const size_t slot = (size_t)(first_chunk(cu_tokens, first_req, req) + blockIdx.x) * H + head;
    bf16* out = planes + slot * CHUNK_BF16(dv);
    float* fout = floats + slot * CHUNK_F32(dv);
    // ---- q, k and v as the convolution left them; rows past the request's tokens are zero
    bf16* sv = reinterpret_cast<bf16*>(s_qk + CH);             // [CH][dv + 8]
    {
        const bf16* base = qkv + (size_t)tok0 * channels;
        for (int idx = tid; idx < 2 * CH * (DQ / 8); idx += PREP_THREADS) {
            const int which = idx / (CH * (DQ / 8)), rest = idx % (CH * (DQ / 8));
            const int row = rest / (DQ / 8), c = rest % (DQ / 8);
            bf16* dst = (which ? sk : sq) + row * LDR + c * 8;
            if (row < rows) cp_async16(dst, base + (size_t)row * channels + (size_t)which * G * DQ + (size_t)kh * DQ + c * 8);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
        }
        const int per = dv / 8;
        for (int idx = tid; idx < CH * per; idx += PREP_THREADS) {
            const int row = idx / per, c = idx - row * per;
            bf16* dst = sv + row * (dv + 8) + c * 8;
            if (row < rows) cp_async16(dst, base + (size_t)row * channels + (size_t)2 * G * DQ + (size_t)head * dv + c * 8);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
        }
        cp_async_commit();
    }
    const float rate = expf(rate_log[head]) * LOG2E;
    if (CHANNEL && a_vec) {
        constexpr int ITERS = (CH * (DQ / 8) + PREP_THREADS - 1) / PREP_THREADS;
        uint4 raw[ITERS];
#pragma unroll
        for (int u = 0; u < ITERS; ++u) {
            const int idx = tid + u * PREP_THREADS, row = idx / (DQ / 8), c = idx % (DQ / 8) * 8;
            raw[u] = make_uint4(0, 0, 0, 0);
            if (row < rows) raw[u] = *reinterpret_cast<const uint4*>(a_rows + (size_t)(tok0 + row) * a_stride + (size_t)head * DQ + c);
        }
#pragma unroll
        for (int u = 0; u < ITERS; ++u) {
            const int idx = tid + u * PREP_THREADS, row = idx / (DQ / 8), c = idx % (DQ / 8) * 8;
            if (row >= CH) continue;
            const float4 d0 = *reinterpret_cast<const float4*>(dt_bias + head * DQ + c), d1 = *reinterpret_cast<const float4*>(dt_bias + head * DQ + c + 4);
            const float bias[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
            const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
            float* dst = sG + row * LDG + c;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 a2 = bf2(w[e]);
                dst[2 * e] = row < rows ? -rate * softplus_f(a2.x + bias[2 * e]) : 0.0f;
                dst[2 * e + 1] = row < rows ? -rate * softplus_f(a2.y + bias[2 * e + 1]) : 0.0f;
            }
        }
    } else if (CHANNEL) {
        for (int idx = tid; idx < CH * DQ; idx += PREP_THREADS) {
            const int row = idx / DQ, c = idx % DQ;
            float lg = 0.0f;
            if (row < rows) lg = -rate * softplus_f(__bfloat162float(a_rows[(size_t)(tok0 + row) * a_stride + (size_t)head * DQ + c]) + dt_bias[head * DQ + c]);
            sG[row * LDG + c] = lg;
        }
    } else if (tid < CH) {
        sG[tid] = tid < rows ? -rate * softplus_f(__bfloat162float(a_rows[(size_t)(tok0 + tid) * a_stride + head]) + dt_bias[head]) : 0.0f;
    }
    if (tid < CH) s_beta[tid] = tid < rows ? 1.0f / (1.0f + expf(-__bfloat162float(b_rows[(size_t)(tok0 + tid) * b_stride + head]))) : 0.0f;
    cp_async_wait<0>();
    __syncthreads();
    // ---- running sums of the log-decays; unit lengths
    if (CHANNEL) {
        for (int c = tid; c < DQ; c += PREP_THREADS) {
            float run = 0.0f;
            for (int i = 0; i < CH; ++i) { run += sG[i * LDG + c]; sG[i * LDG + c] = run; }
        }
    } else if (tid == 0) {
        float run = 0.0f;
        for (int i = 0; i < CH; ++i) { run += sG[i]; sG[i] = run; }
    }
    {                                                          // eight rows a warp side by side, four lanes a row
        const int row = warp * 8 + g;
        float qq = 0.0f, kk = 0.0f, qk = 0.0f;
        for (int c = lane & 3; c < DQ / 8; c += 4) {
            const uint4 q8 = *reinterpret_cast<const uint4*>(sq + row * LDR + c * 8), k8 = *reinterpret_cast<const uint4*>(sk + row * LDR + c * 8);
            const uint32_t qw[4] = {q8.x, q8.y, q8.z, q8.w}, kw[4] = {k8.x, k8.y, k8.z, k8.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float2 x = bf2(qw[u]), y = bf2(kw[u]);
                qq = fmaf(x.x, x.x, qq); qq = fmaf(x.y, x.y, qq);
                kk = fmaf(y.x, y.x, kk); kk = fmaf(y.y, y.y, kk);
                qk = fmaf(x.x, y.x, qk); qk = fmaf(x.y, y.y, qk);
            }
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            qq += __shfl_xor_sync(0xffffffffu, qq, o);
            kk += __shfl_xor_sync(0xffffffffu, kk, o);
            qk += __shfl_xor_sync(0xffffffffu, qk, o);
        }
        if ((lane & 3) == 0) {
            s_fq[row] = 1.0f / (sqrtf((float)DQ) * sqrtf(qq + UNIT_EPS));
            s_fk[row] = 1.0f / sqrtf(kk + UNIT_EPS);
            s_qk[row] = qk;
        }
    }
    // (the upper triangles stay zero; of P's only what lies in a diagonal block is ever read)
    for (int idx = tid; idx < 4 * 16 * LDD; idx += PREP_THREADS) sD[idx] = 0.0f;
    bf16* ph = out + AT_P;
    for (int idx = tid; idx < 4 * 16 * 2; idx += PREP_THREADS) {
        const int row = (idx >> 1), at = row * LDW + (row & ~15) + (idx & 1) * 8;
        *reinterpret_cast<uint4*>(ph + at) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(ph + PPLANE + at) = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    // ---- A and P: two warps make the rows 16 I .. 16 I + 15, with one decay per head each eight columns of every block of sixteen.  With one per channel each
    // half of the channels (so that no row's exponentials and splits are made twice), and they exchange the halves of the sums: with the
    // rows' lengths found four lanes a row, 102 -> 91 us for 620 chunks and heads (the rows of the last block had 2.6 times the first one's work).
    {
        const int I = warp >> 1, half = warp & 1;
        const int i0 = I * 16 + g, i1 = i0 + 8;
        constexpr int NH = CHANNEL ? 2 : 1;                    // runs of eight columns
        float accA[4][4], accP[4][4];                          // [block of columns]; the fourth: this block's own
        float farA[3][4], farP[3][4];                          // the run of eight columns that the other warp will finish
#pragma unroll
        for (int J = 0; J < 4; ++J)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                accA[J][e] = 0.0f; accP[J][e] = 0.0f;
                if (J < 3) { farA[J < 3 ? J : 0][e] = 0.0f; farP[J < 3 ? J : 0][e] = 0.0f; }
            }
        // a reference for the rows of this block against earlier ones: the sum at the last row before it; for its rows 8 .. 15 against
        // its rows 0 .. 7 (each warp its half of the channels, as of all else): the sum at its row 7
        const float* ref = sG + (I > 0 ? I * 16 - 1 : 0) * LDG;
        const float* mid = sG + (I * 16 + 7) * LDG;
#pragma unroll 1
        for (int kk = CHANNEL ? half * ((KT + 1) / 2) : 0; kk < (CHANNEL && half == 0 ? (KT + 1) / 2 : KT); ++kk) {
            uint32_t rk[4], rq[4];                             // raw bf16 pairs: rows i0, i1 at channels c, c + 8
            const int c = kk * 16 + t2;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int row = (u & 1) ? i1 : i0;
                rk[u] = *reinterpret_cast<const uint32_t*>(sk + row * LDR + c + (u >> 1) * 8);
                rq[u] = *reinterpret_cast<const uint32_t*>(sq + row * LDR + c + (u >> 1) * 8);
            }
            if (!CHANNEL) {
#pragma unroll
                for (int J = 0; J < 4; ++J) {
                    const int jb = J < 3 ? J : I;
                    if (J < 3 && J >= I) continue;
                    const bf16* row = sk + (jb * 16 + half * 8 + g) * LDR + c;
                    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(row), b1 = *reinterpret_cast<const uint32_t*>(row + 8);
                    mma_bf16_16816(accA[J], rk, b0, b1);
                    mma_bf16_16816(accP[J], rq, b0, b1);
                }
            } else {
                uint32_t kh_[4], kl_[4], qh_[4], ql_[4];
                if (I > 0) {
                    const float2 ra = *reinterpret_cast<const float2*>(ref + c), rb = *reinterpret_cast<const float2*>(ref + c + 8);
                    const float r[4] = {ra.x, ra.y, rb.x, rb.y};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float2 gi = *reinterpret_cast<const float2*>(sG + ((u & 1) ? i1 : i0) * LDG + c + (u >> 1) * 8);
                        const float e0 = ex2_approx(gi.x - r[(u >> 1) * 2]), e1 = ex2_approx(gi.y - r[(u >> 1) * 2 + 1]);
                        const float2 k2 = bf2(rk[u]), q2 = bf2(rq[u]);
                        split_bf16(k2.x * e0, k2.y * e1, kh_[u], kl_[u]);
                        split_bf16(q2.x * e0, q2.y * e1, qh_[u], ql_[u]);
                    }
#pragma unroll
                    for (int J = 0; J < 3; ++J) {
                        if (J >= I) continue;
#pragma unroll
                        for (int far = 0; far < NH; ++far) {
                            const int j = J * 16 + (half ^ far) * 8 + g;
                            const float2 ga = *reinterpret_cast<const float2*>(sG + j * LDG + c), gb = *reinterpret_cast<const float2*>(sG + j * LDG + c + 8);
                            const float2 x = bf2(*reinterpret_cast<const uint32_t*>(sk + j * LDR + c)), y = bf2(*reinterpret_cast<const uint32_t*>(sk + j * LDR + c + 8));
                            uint32_t bh0, bl0, bh1, bl1;
                            split_bf16(x.x * ex2_approx(r[0] - ga.x), x.y * ex2_approx(r[1] - ga.y), bh0, bl0);
                            split_bf16(y.x * ex2_approx(r[2] - gb.x), y.y * ex2_approx(r[3] - gb.y), bh1, bl1);
                            mma3(far ? farA[J] : accA[J], kh_, kl_, bh0, bh1, bl0, bl1);
                            mma3(far ? farP[J] : accP[J], qh_, ql_, bh0, bh1, bl0, bl1);
                        }
                    }
                }
                {                                              // rows 8 .. 15 of the block (the operands of rows 0 .. 7 are zero)
                    const float2 ra = *reinterpret_cast<const float2*>(mid + c), rb = *reinterpret_cast<const float2*>(mid + c + 8);
                    const float r[4] = {ra.x, ra.y, rb.x, rb.y};
                    kh_[0] = kh_[2] = kl_[0] = kl_[2] = qh_[0] = qh_[2] = ql_[0] = ql_[2] = 0u;
#pragma unroll
                    for (int u = 1; u < 4; u += 2) {
                        const float2 gi = *reinterpret_cast<const float2*>(sG + i1 * LDG + c + (u >> 1) * 8);
                        const float e0 = ex2_approx(gi.x - r[(u >> 1) * 2]), e1 = ex2_approx(gi.y - r[(u >> 1) * 2 + 1]);
                        const float2 k2 = bf2(rk[u]), q2 = bf2(rq[u]);
                        split_bf16(k2.x * e0, k2.y * e1, kh_[u], kl_[u]);
                        split_bf16(q2.x * e0, q2.y * e1, qh_[u], ql_[u]);
                    }
                    const float2 ga = *reinterpret_cast<const float2*>(sG + i0 * LDG + c), gb = *reinterpret_cast<const float2*>(sG + i0 * LDG + c + 8);   // token g of the block: the same index as row i0
                    const float2 x = bf2(rk[0]), y = bf2(rk[2]);
                    uint32_t bh0, bl0, bh1, bl1;
                    split_bf16(x.x * ex2_approx(r[0] - ga.x), x.y * ex2_approx(r[1] - ga.y), bh0, bl0);
                    split_bf16(y.x * ex2_approx(r[2] - gb.x), y.y * ex2_approx(r[3] - gb.y), bh1, bl1);
                    mma3(accA[3], kh_, kl_, bh0, bh1, bl0, bl1);
                    mma3(accP[3], qh_, ql_, bh0, bh1, bl0, bl1);
                }
            }
        }
        float* given = reinterpret_cast<float*>(sL) + (I * I * 8 + (half ? 8 * I + 4 : 0)) * 32 + lane;    // (nothing of L is there yet)
        if (CHANNEL) {
#pragma unroll
            for (int J = 0; J < 3; ++J) {
                if (J >= I) continue;
#pragma unroll
                for (int e = 0; e < 4; ++e) { given[(J * 8 + e) * 32] = farA[J][e]; given[(J * 8 + 4 + e) * 32] = farP[J][e]; }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) { given[(I * 8 + e) * 32] = accA[3][2 + e]; given[(I * 8 + 2 + e) * 32] = accP[3][2 + e]; }
        }
        if (CHANNEL && lane < 28) {                            // the 8 x 8 square on the diagonal that is this warp's, a pair of rows per lane
            int ii = 1;
            while ((ii + 1) * ii / 2 <= lane) ++ii;
            const int i = warp * 8 + ii, j = warp * 8 + lane - ii * (ii - 1) / 2;
            float a = 0.0f, b = 0.0f;
#pragma unroll 4
            for (int c = 0; c < DQ; c += 2) {
                const float2 ki = bf2(*reinterpret_cast<const uint32_t*>(sk + i * LDR + c)), kj = bf2(*reinterpret_cast<const uint32_t*>(sk + j * LDR + c));
                const float2 qi = bf2(*reinterpret_cast<const uint32_t*>(sq + i * LDR + c));
                const float2 gi = *reinterpret_cast<const float2*>(sG + i * LDG + c), gj = *reinterpret_cast<const float2*>(sG + j * LDG + c);
                const float x = kj.x * ex2_approx(gi.x - gj.x), y = kj.y * ex2_approx(gi.y - gj.y);
                a = fmaf(ki.x, x, a); a = fmaf(ki.y, y, a);
                b = fmaf(qi.x, x, b); b = fmaf(qi.y, y, b);
            }
            sD[i * LDD + (j & 15)] = s_beta[i] * s_fk[i] * s_fk[j] * a;
            b *= s_fq[i] * s_fk[j];
            const bf16 hi = __float2bfloat16_rn(b);
            const int at = i * LDW + j;
            ph[at] = hi;
            ph[PPLANE + at] = __float2bfloat16_rn(b - __bfloat162float(hi));
        }
        if (CHANNEL) {
            __syncthreads();
            const float* got = reinterpret_cast<float*>(sL) + (I * I * 8 + (half ? 0 : 8 * I + 4)) * 32 + lane;
#pragma unroll
            for (int J = 0; J < 3; ++J) {
                if (J >= I) continue;
#pragma unroll
                for (int e = 0; e < 4; ++e) { accA[J][e] += got[(J * 8 + e) * 32]; accP[J][e] += got[(J * 8 + 4 + e) * 32]; }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) { accA[3][2 + e] += got[(I * 8 + e) * 32]; accP[3][2 + e] += got[(I * 8 + 2 + e) * 32]; }
            __syncthreads();
        }
#pragma unroll
        for (int J = 0; J < 4; ++J) {
            const int jb = J < 3 ? J : I;
            if ((J < 3 && J >= I) || (CHANNEL && J == 3 && half == 1)) continue;
            const int j = jb * 16 + half * 8 + t2;
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                if (CHANNEL && J == 3 && rr == 0) continue;    // rows 0 .. 7 of the block's own square: pair by pair above
                const int i = rr ? i1 : i0;
                float a[2], b[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float w = CHANNEL ? 1.0f : j + e <= i ? ex2_approx(sG[i] - sG[j + e]) : 0.0f;
                    a[e] = s_beta[i] * s_fk[i] * s_fk[j + e] * accA[J][rr * 2 + e] * w;
                    b[e] = s_fq[i] * s_fk[j + e] * accP[J][rr * 2 + e] * w;
                    if (J == 3 && j + e < i) sD[i * LDD + ((j + e) & 15)] = a[e];
                }
                uint32_t hi, lo;                               // (a weight of zero where j > i)
                if (J < 3) {
                    split_bf16(-a[0], -a[1], hi, lo);
                    *reinterpret_cast<uint32_t*>(sL + i * LDL + j) = hi;
                    *reinterpret_cast<uint32_t*>(sL + CH * LDL + i * LDL + j) = lo;
                }
                split_bf16(b[0], b[1], hi, lo);
                const int at = i * LDW + j;
                *reinterpret_cast<uint32_t*>(ph + at) = hi;
                *reinterpret_cast<uint32_t*>(ph + PPLANE + at) = lo;
            }
        }
        if (CHANNEL && tid < CH) {                             // P_ii = q_i . k_i
            const float b = s_qk[tid] * s_fq[tid] * s_fk[tid];
            const bf16 hi = __float2bfloat16_rn(b);
            const int at = tid * LDW + tid;
            ph[at] = hi;
            ph[PPLANE + at] = __float2bfloat16_rn(b - __bfloat162float(hi));
        }
    }
    __syncthreads();
    // ---- two warps: the inverse of each diagonal block, a column a thread (x_i = [i = j] - sum_(k < i) L_ik x_k), less its unit diagonal
    if (warp < 2) {
        const int b = tid >> 4, j = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = i == j ? 1.0f : 0.0f;
#pragma unroll
        for (int i = 1; i < 16; ++i) {
            float acc0 = x[i], acc1 = 0.0f;
#pragma unroll
            for (int k = 0; k < i; k += 4) {
                const float4 l = *reinterpret_cast<const float4*>(sD + (b * 16 + i) * LDD + k);       // (zero from the diagonal on)
                acc0 = fmaf(-l.x, x[k], acc0);
                if (k + 1 < i) acc1 = fmaf(-l.y, x[k + 1], acc1);
                if (k + 2 < i) acc0 = fmaf(-l.z, x[k + 2], acc0);
                if (k + 3 < i) acc1 = fmaf(-l.w, x[k + 3], acc1);
            }
            x[i] = acc0 + acc1;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float v = i > j ? x[i] : 0.0f;
            const bf16 hi = __float2bfloat16_rn(v);
            sL[(b * 16 + i) * LDL + b * 16 + j] = hi;
            sL[CH * LDL + (b * 16 + i) * LDL + b * 16 + j] = __float2bfloat16_rn(v - __bfloat162float(hi));
        }
    } else {
        // ---- the others: Q+, K exp(G_63 - G), exp(G_63)
        for (int idx = tid - 64; idx < CH * DQ / 8; idx += PREP_THREADS - 64) {
            const int i = idx / (DQ / 8), c = idx % (DQ / 8) * 8;
            const uint4 kraw = *reinterpret_cast<const uint4*>(sk + i * LDR + c), qraw = *reinterpret_cast<const uint4*>(sq + i * LDR + c);
            const uint32_t kw[4] = {kraw.x, kraw.y, kraw.z, kraw.w}, qw[4] = {qraw.x, qraw.y, qraw.z, qraw.w};
            uint32_t kh_[4], kl_[4], qh_[4], ql_[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float2 k2 = bf2(kw[u]), q2 = bf2(qw[u]);
                const float2 g2 = CHANNEL ? *reinterpret_cast<const float2*>(sG + i * LDG + c + 2 * u) : make_float2(sG[i], sG[i]);
                const float2 e2 = CHANNEL ? *reinterpret_cast<const float2*>(sG + (CH - 1) * LDG + c + 2 * u) : make_float2(sG[CH - 1], sG[CH - 1]);
                split_bf16(k2.x * s_fk[i] * ex2_approx(e2.x - g2.x), k2.y * s_fk[i] * ex2_approx(e2.y - g2.y), kh_[u], kl_[u]);
                split_bf16(q2.x * s_fq[i] * ex2_approx(g2.x), q2.y * s_fq[i] * ex2_approx(g2.y), qh_[u], ql_[u]);
            }
            bf16* at = out + AT_K + i * LDQ + c;
            *reinterpret_cast<uint4*>(at) = make_uint4(kh_[0], kh_[1], kh_[2], kh_[3]);
            *reinterpret_cast<uint4*>(at + KPLANE) = make_uint4(kl_[0], kl_[1], kl_[2], kl_[3]);
            *reinterpret_cast<uint4*>(at + 2 * KPLANE) = make_uint4(qh_[0], qh_[1], qh_[2], qh_[3]);
            *reinterpret_cast<uint4*>(at + 3 * KPLANE) = make_uint4(ql_[0], ql_[1], ql_[2], ql_[3]);
        }
        for (int c = tid - 64; c < DQ; c += PREP_THREADS - 64) fout[CH * dv + c] = ex2_approx(CHANNEL ? sG[(CH - 1) * LDG + c] : sG[CH - 1]);
    }
    __syncthreads();
    // ---- forward substitution by blocks of 16 tokens, transposed (the rows of a product are 16 columns of W or U0, its columns tokens):
    //     Z_I = rhs_I - sum_(J < I) L_IJ X_J,   X_I = Z_I + (L_II^-1 - 1) Z_I.
    // A lane holds tokens 4 q .. 4 q + 3 of a block (columns t2, t2 + 1 of both products of eight), so that sums become row operands as they lie, an
    // operand is one 8-byte load and a result 8 or 16 bytes of a column.  (A thread a column with all its 64 numbers in registers is bound
    // by the loads of L, the same numbers for all threads: 16,000 of the SM's cycles a chunk.)
    const int q4 = 4 * (lane & 3), brow = 4 * (g >> 1) + (g & 1);
    for (int tile = warp; tile < (DQ + dv) / 16; tile += PREP_THREADS / 32) {
        const bool is_w = tile * 16 < DQ;
        const int col = is_w ? tile * 16 + g : tile * 16 - DQ + g;
        uint32_t xh[3][4], xl[3][4];
#pragma unroll
        for (int I = 0; I < 4; ++I) {
            float z[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = I * 16 + q4 + 2 * nt + (e & 1), c = col + (e >> 1) * 8;
                    if (is_w) z[nt][e] = s_beta[i] * s_fk[i] * __bfloat162float(sk[i * LDR + c]) * ex2_approx(CHANNEL ? sG[i * LDG + c] : sG[i]);
                    else z[nt][e] = s_beta[i] * __bfloat162float(sv[i * (dv + 8) + c]);
                }
#pragma unroll
            for (int J = 0; J < 4; ++J) {
                if (J >= I) continue;
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const bf16* row = sL + (I * 16 + brow + 2 * nt) * LDL + J * 16 + q4;
                    const uint2 bh = *reinterpret_cast<const uint2*>(row), bl = *reinterpret_cast<const uint2*>(row + CH * LDL);
                    mma3(z[nt], xh[J], xl[J], bh.x, bh.y, bl.x, bl.y);
                }
            }
            uint32_t zh[4], zl[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) split_bf16(z[u >> 1][(u & 1) * 2], z[u >> 1][(u & 1) * 2 + 1], zh[u], zl[u]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const bf16* row = sL + (I * 16 + brow + 2 * nt) * LDL + I * 16 + q4;
                const uint2 bh = *reinterpret_cast<const uint2*>(row), bl = *reinterpret_cast<const uint2*>(row + CH * LDL);
                mma3(z[nt], zh, zl, bh.x, bh.y, bl.x, bl.y);
            }
            if (is_w || I < 3)
#pragma unroll
                for (int u = 0; u < 4; ++u) split_bf16(z[u >> 1][(u & 1) * 2], z[u >> 1][(u & 1) * 2 + 1], zh[u], zl[u]);
            if (I < 3)
#pragma unroll
                for (int u = 0; u < 4; ++u) { xh[I < 3 ? I : 0][u] = zh[u]; xl[I < 3 ? I : 0][u] = zl[u]; }
#pragma unroll
            for (int h = 0; h < 2; ++h) {                      // column col + 8 h
                const int c = col + 8 * h, i = I * 16 + q4;
                if (is_w) {
                    *reinterpret_cast<uint2*>(out + c * LDW + i) = make_uint2(zh[h], zh[2 + h]);
                    *reinterpret_cast<uint2*>(out + WPLANE + c * LDW + i) = make_uint2(zl[h], zl[2 + h]);
                } else {
                    *reinterpret_cast<float4*>(fout + c * CH + (i ^ TURN0(c))) = make_float4(z[0][2 * h], z[0][2 * h + 1], z[1][2 * h], z[1][2 * h + 1]);
                }
            }
        }
    }
}

// ---- the walk -------------------------------------------------------------------------------------------------------------------------
#define VG (VS / 16)                  // groups of 16 value channels: a pair of warps each
#define WALK_THREADS (64 * VG)
#define HT ((KT + 1) / 2)             // blocks of key channels a warp of a pair has
#define STAGE_BYTES (2 * WPLANE * 2 + 2 * KPLANE * 2 + VS * CH * 4)
#define WALK_SMEM (2 * STAGE_BYTES + VG * 2 * 16 * CH * 4)

__device__ __forceinline__ void bulk_in(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Transposed: a pair of warps has 16 value channels, a warp of it half of the key channels of their state in registers, as the sums of
// S^T += U^T (K exp(G_63 - G)) leave them, which is how the row operand of U^T = U0^T - S^T W^T wants them; U^T goes on to the next product likewise.  Only
// the two halves of S^T W^T meet in shared memory.  Bound by mma.sync (8 cycles of a scheduler each: 1.6 us a chunk for 64 value and 128 key channels) and the
// operands' way from shared memory, which two chunks' worth of bulk copies fill.  64 value channels a CTA: fewer fetch W and K through L2 too often.
__global__ void __launch_bounds__(WALK_THREADS, 1) walk_kernel(bf16* planes, float* floats, float* __restrict__ state, const int* __restrict__ cu_tokens,
                                                               const int* __restrict__ slots, int first_req, int H, int dv, int* error_flag) {
    PDL_ENTER_WALK();
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ uint64_t w_there[2], k_there[2];
    const int req = first_req + blockIdx.x, head = blockIdx.y, vs0 = blockIdx.z * VS;
    const int first = cu_tokens[req], count = cu_tokens[req + 1] - first;
    if (count <= 0) return;
    const int chunks = (count + CH - 1) / CH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t2 = 2 * (lane & 3);
    const int vg = warp >> 1, half = warp & 1;
    const size_t slot0 = (size_t)first_chunk(cu_tokens, first_req, req) * H + head;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) { mbar_init(&w_there[i], 1); mbar_init(&k_there[i], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto load = [&](int c) {                           // (one thread) W, U0 and K of a chunk
        if (c >= chunks) return;
        uint8_t* stage = smem_raw + (c & 1) * STAGE_BYTES;
        const bf16* p = planes + (slot0 + (size_t)c * H) * CHUNK_BF16(dv);
        const float* f = floats + (slot0 + (size_t)c * H) * CHUNK_F32(dv);
        mbar_expect_tx(&w_there[c & 1], 2 * WPLANE * 2 + VS * CH * 4);
        bulk_in(stage, p, 2 * WPLANE * 2, &w_there[c & 1]);
        bulk_in(stage + 2 * WPLANE * 2 + 2 * KPLANE * 2, f + (size_t)vs0 * CH, VS * CH * 4, &w_there[c & 1]);
        mbar_expect_tx(&k_there[c & 1], 2 * KPLANE * 2);
        bulk_in(stage + 2 * WPLANE * 2, p + AT_K, 2 * KPLANE * 2, &k_there[c & 1]);
    };
    if (threadIdx.x == 0) { load(0); load(1); }
    // S^T: value channels g and g + 8 of the group x key channels t2, t2 + 1 of every run of eight
    float* st = state + (((size_t)slots[req] * H + head) * DQ) * dv + vs0 + vg * 16 + g;
    float S[HT][2][4];
#pragma unroll
    for (int i = 0; i < HT; ++i)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tile = half * HT + i;
                S[i][n][e] = tile < KT ? st[(size_t)(tile * 16 + n * 8 + t2 + (e & 1)) * dv + (e >> 1) * 8] : 0.0f;
            }
    const int b_row = (lane & 7) + ((lane >> 3) & 1) * 8, b_col = (lane >> 4) * 8;           // column operands that lie by their k, read transposed
    const uint32_t w_addr = smem_u32(smem_raw) + (b_row * LDW + b_col) * 2, k_addr = smem_u32(smem_raw) + 2 * WPLANE * 2 + (b_row * LDQ + b_col) * 2;
    float4* mine = reinterpret_cast<float4*>(smem_raw + 2 * STAGE_BYTES) + warp * (16 * CH / 4) + lane;       // [8][32 lanes]
    const float4* other = reinterpret_cast<const float4*>(smem_raw + 2 * STAGE_BYTES) + (warp ^ 1) * (16 * CH / 4) + lane;
    bool ok = true;
    for (int c = 0; c < chunks; ++c) {
        bf16* p = planes + (slot0 + (size_t)c * H) * CHUNK_BF16(dv);
        float* f = floats + (slot0 + (size_t)c * H) * CHUNK_F32(dv);
        const uint32_t at = (c & 1) * STAGE_BYTES, parity = (c >> 1) & 1;
        float2 last[HT][2];
#pragma unroll
        for (int i = 0; i < HT; ++i)
#pragma unroll
            for (int n = 0; n < 2; ++n)
                last[i][n] = half * HT + i < KT ? *reinterpret_cast<const float2*>(f + CH * dv + (half * HT + i) * 16 + n * 8 + t2) : make_float2(0.0f, 0.0f);
        ok = ok && mbar_wait(&w_there[c & 1], parity);
        // U^T = U0^T - S^T W^T (the pair's first warp begins with U0, the second with zeros)
        float u[8][4];
        {
            const float* u0 = reinterpret_cast<const float*>(smem_raw + at + 2 * WPLANE * 2 + 2 * KPLANE * 2) + (vg * 16 + g) * CH;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                u[n][0] = u[n][1] = u[n][2] = u[n][3] = 0.0f;
                if (half == 0) {
                    const float2 a = *reinterpret_cast<const float2*>(u0 + ((n * 8 + t2) ^ TURN0(g))), b = *reinterpret_cast<const float2*>(u0 + 8 * CH + ((n * 8 + t2) ^ TURN0(g)));
                    u[n][0] = a.x; u[n][1] = a.y; u[n][2] = b.x; u[n][3] = b.y;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < HT; ++i) {
            const int tile = half * HT + i;
            if (tile >= KT) continue;
            uint32_t sh[4], sl[4], mh[4], ml[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                split_bf16(S[i][r >> 1][(r & 1) * 2], S[i][r >> 1][(r & 1) * 2 + 1], sh[r], sl[r]);
                mh[r] = sh[r] ^ 0x80008000u; ml[r] = sl[r] ^ 0x80008000u;          // -S
            }
            bf16* s0 = p + AT_S + (size_t)((((vs0 >> 4) + vg) * KT + tile) * 2) * 256 + lane * 8;
            *reinterpret_cast<uint4*>(s0) = make_uint4(sh[0], sh[1], sh[2], sh[3]);
            *reinterpret_cast<uint4*>(s0 + 256) = make_uint4(sl[0], sl[1], sl[2], sl[3]);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                uint32_t bh[4], bl[4];
                ldsm_x4_trans(w_addr + at + (tile * 16 * LDW + n * 16) * 2, bh[0], bh[1], bh[2], bh[3]);
                ldsm_x4_trans(w_addr + at + WPLANE * 2 + (tile * 16 * LDW + n * 16) * 2, bl[0], bl[1], bl[2], bl[3]);
                mma3(u[2 * n], mh, ml, bh[0], bh[1], bl[0], bl[1]);
                mma3(u[2 * n + 1], mh, ml, bh[2], bh[3], bl[2], bl[3]);
            }
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) mine[n * 32] = make_float4(u[n][0], u[n][1], u[n][2], u[n][3]);
        asm volatile("bar.sync %0, 64;" ::"r"(1 + vg) : "memory");
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const float4 v = other[n * 32];
            u[n][0] += v.x; u[n][1] += v.y; u[n][2] += v.z; u[n][3] += v.w;
        }
#pragma unroll
        for (int i = 0; i < HT; ++i)
#pragma unroll
            for (int n = 0; n < 2; ++n) { S[i][n][0] *= last[i][n].x; S[i][n][1] *= last[i][n].y; S[i][n][2] *= last[i][n].x; S[i][n][3] *= last[i][n].y; }
        ok = ok && mbar_wait(&k_there[c & 1], parity);
        // S^T = S^T exp(G_63) + U^T (K exp(G_63 - G))
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk) {
            uint32_t uh[4], ul[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) split_bf16(u[2 * kk + (r >> 1)][(r & 1) * 2], u[2 * kk + (r >> 1)][(r & 1) * 2 + 1], uh[r], ul[r]);
            if ((kk >> 1) == half) {                   // in U0's place, whose copy has arrived; either warp half of it
                bf16* u0 = reinterpret_cast<bf16*>(f) + (size_t)((((vs0 >> 4) + vg) * 4 + kk) * 2) * 256 + lane * 8;
                *reinterpret_cast<uint4*>(u0) = make_uint4(uh[0], uh[1], uh[2], uh[3]);
                *reinterpret_cast<uint4*>(u0 + 256) = make_uint4(ul[0], ul[1], ul[2], ul[3]);
            }
#pragma unroll
            for (int i = 0; i < HT; ++i) {
                const int tile = half * HT + i;
                if (tile >= KT) continue;
                uint32_t bh[4], bl[4];
                ldsm_x4_trans(k_addr + at + (kk * 16 * LDQ + tile * 16) * 2, bh[0], bh[1], bh[2], bh[3]);
                ldsm_x4_trans(k_addr + at + KPLANE * 2 + (kk * 16 * LDQ + tile * 16) * 2, bl[0], bl[1], bl[2], bl[3]);
                mma3(S[i][0], uh, ul, bh[0], bh[1], bl[0], bl[1]);
                mma3(S[i][1], uh, ul, bh[2], bh[3], bl[2], bl[3]);
            }
        }
        __syncthreads();                               // everyone is done with this chunk's operands (and a pair with each other's halves)
        if (threadIdx.x == 0) load(c + 2);
    }
    if (!ok && lane == 0) atomicExch(error_flag, 41);
#pragma unroll
    for (int i = 0; i < HT; ++i)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tile = half * HT + i;
                if (tile < KT) st[(size_t)(tile * 16 + n * 8 + t2 + (e & 1)) * dv + (e >> 1) * 8] = S[i][n][e];
            }
}

// ---- the outputs ----------------------------------------------------------------------------------------------------------------------
// O^T = S0^T Q+^T + U^T P^T: a CTA per chunk, head and up to 128 value channels, a warp per 16 of them, whose operands it loads as the walk left them; Q+ and
// P come to shared memory by bulk copies, which then holds the sums by token.  Bound by what the kernels before left (230 KB a chunk and head of 128 x 128, 150
// of them read here).  NORM: out = O / rms(O) * weight * gate * factor (a whole head a CTA), else the sums to o.
#define READ_THREADS 256
#define READ_COLS 128
#define READ_OPERANDS (2 * KPLANE * 2 + 2 * PPLANE * 2)
#define READ_SUMS(cols) (CH * ((cols) + 4) * 4)

template <bool NORM>
__global__ void __launch_bounds__(READ_THREADS, 2) read_kernel(const bf16* __restrict__ planes, const float* __restrict__ floats, const int* __restrict__ cu_tokens,
                                                               float* __restrict__ o, int first_req, int H, int dv, int parts, const bf16* __restrict__ gate_rows,
                                                               int gate_stride, int gate, const float* __restrict__ norm_w, float eps, float factor,
                                                               bf16* __restrict__ out, int out_stride, int* error_flag) {
    PDL_ENTER();
    planes = pdl_fresh(planes); floats = pdl_fresh(floats); gate_rows = pdl_fresh(gate_rows);
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ uint64_t there;
    const int req = first_req + blockIdx.z / parts, head = blockIdx.y, c0 = blockIdx.z % parts * READ_COLS, cols = min(READ_COLS, dv - c0);
    const int tok0 = cu_tokens[req] + blockIdx.x * CH;
    const int rows = min(CH, cu_tokens[req + 1] - tok0);
    if (rows <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t2 = 2 * (lane & 3);
    const size_t slot = (size_t)(first_chunk(cu_tokens, first_req, req) + blockIdx.x) * H + head;
    const bf16* p = planes + slot * CHUNK_BF16(dv);
    const bf16* f = reinterpret_cast<const bf16*>(floats + slot * CHUNK_F32(dv));
    if (threadIdx.x == 0) {
        mbar_init(&there, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(&there, READ_OPERANDS);
        bulk_in(smem_raw, p + AT_Q, READ_OPERANDS, &there);           // Q+ and, behind it, P
    }
    const bool some = warp * 16 < cols;                // (all lanes of a warp)
    const int vg = (c0 >> 4) + (some ? warp : 0);
    uint4 ah[KT], al[KT];
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
        const bf16* at = p + AT_S + (size_t)((vg * KT + kk) * 2) * 256 + lane * 8;
        ah[kk] = *reinterpret_cast<const uint4*>(at);
        al[kk] = *reinterpret_cast<const uint4*>(at + 256);
    }
    float acc[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    const int b_row = (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 8;             // column operands that lie by their columns
    const uint32_t q_addr = smem_u32(smem_raw) + (b_row * LDQ + b_col) * 2, p_addr = smem_u32(smem_raw) + 2 * KPLANE * 2 + (b_row * LDW + b_col) * 2;
    auto add = [&](const uint4& h4, const uint4& l4, uint32_t addr, int ld, int plane, int from) {
        const uint32_t xh[4] = {h4.x, h4.y, h4.z, h4.w}, xl[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            if (n < from) continue;
            uint32_t bh[4], bl[4];
            ldsm_x4(addr + n * 16 * ld * 2, bh[0], bh[1], bh[2], bh[3]);
            ldsm_x4(addr + plane * 2 + n * 16 * ld * 2, bl[0], bl[1], bl[2], bl[3]);
            mma3(acc[2 * n], xh, xl, bh[0], bh[1], bl[0], bl[1]);
            mma3(acc[2 * n + 1], xh, xl, bh[2], bh[3], bl[2], bl[3]);
        }
    };
    __syncthreads();                                   // the barrier is set up
    const bool ok = mbar_wait(&there, 0);
    if (some) {
        uint4 uh[4], ul[4];
#pragma unroll
        for (int kk = 0; kk < KT; ++kk) {
            if (kk == KT / 2) {                        // (asked for where half of S's registers are free again)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bf16* at = f + (size_t)((vg * 4 + j) * 2) * 256 + lane * 8;
                    uh[j] = *reinterpret_cast<const uint4*>(at);
                    ul[j] = *reinterpret_cast<const uint4*>(at + 256);
                }
            }
            add(ah[kk], al[kk], q_addr + kk * 32, LDQ, KPLANE, 0);
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) add(uh[kk], ul[kk], p_addr + kk * 32, LDW, PPLANE, kk);       // (no earlier token has a weight)
    }
    __syncthreads();                                   // everyone has left Q+ and P
    float* sums = reinterpret_cast<float*>(smem_raw);  // [CH][cols + 4]
    const int ld = cols + 4;
    if (some) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) sums[(n * 8 + t2 + (e & 1)) * ld + warp * 16 + g + (e >> 1) * 8] = acc[n][e];
    }
    if (!ok && lane == 0) atomicExch(error_flag, 42);
    __syncthreads();
    const bool here = lane * 4 < cols;                 // four columns of a token a lane
    for (int i = warp; i < rows; i += READ_THREADS / 32) {
        const float4 v = here ? *reinterpret_cast<const float4*>(sums + i * ld + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (!NORM) {
            float* to = o + (size_t)(tok0 + i) * H * dv + (size_t)head * dv + c0 + lane * 4;
            if (here && (((uintptr_t)to) & 15) == 0) *reinterpret_cast<float4*>(to) = v;
            else if (here) { to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w; }
            continue;
        }
        uint2 raw = make_uint2(0u, 0u);
        if (here) raw = *reinterpret_cast<const uint2*>(gate_rows + (size_t)(tok0 + i) * gate_stride + (size_t)head * dv + lane * 4);
        const float scale = factor / sqrtf(warp_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w)) / (float)dv + eps);
        if (!here) continue;
        const float4 w = *reinterpret_cast<const float4*>(norm_w + lane * 4);
        const float2 a = bf2(raw.x), b = bf2(raw.y);
        float4 s4 = make_float4(__fdividef(1.0f, 1.0f + __expf(-a.x)), __fdividef(1.0f, 1.0f + __expf(-a.y)), __fdividef(1.0f, 1.0f + __expf(-b.x)),
                                __fdividef(1.0f, 1.0f + __expf(-b.y)));
        if (gate == 1) { s4.x *= a.x; s4.y *= a.y; s4.z *= b.x; s4.w *= b.y; }
        *reinterpret_cast<uint2*>(out + (size_t)(tok0 + i) * out_stride + (size_t)head * dv + lane * 4) =
            make_uint2(pack_bf16(v.x * scale * w.x * s4.x, v.y * scale * w.y * s4.y), pack_bf16(v.z * scale * w.z * s4.z, v.w * scale * w.w * s4.w));
    }
}

// How many bf16 and float32 numbers a chunk and head needs between the kernels.
MB_API int mb_delta_chunked_scratch(int dv, int* bf16s, int* floats) { *bf16s = CHUNK_BF16(dv); *floats = CHUNK_F32(dv); return 0; }

// Requests first_req .. requests - 1; which: 0 prepares, 1 walks, 2 reads (in this order).  qkv: bf16 [tokens][2 G QK_DIM + H dv] after the convolution (rows
// 16-byte aligned); b, a, their strides, per_channel, rate_log, dt_bias and state as mb_delta_scan takes them; dv a multiple of V_SLICE.  planes and
// floats hold (tokens / 64 + requests) * H pieces of mb_delta_chunked_scratch each.  The sums go to o as mb_delta_scan leaves them or, where out is
// given (dv up to 128), through norm and gate to out: gate_rows, gate, norm_w, eps and factor as mb_delta_norm takes them, all three at 8-byte addresses
// (norm_w: 16).
MB_API int mb_delta_chunked(const void* qkv, const void* b_rows, int b_stride, const void* a_rows, int a_stride, int per_channel, const float* rate_log,
                            const float* dt_bias, float* state, const int* cu_tokens, const int* slots, float* o, void* planes, float* floats,
                            const void* gate_rows, int gate_stride, int gate, const float* norm_w, float eps, float factor, void* out, int out_stride,
                            int* error_flag, int first_req, int requests, int max_query_len, int H, int G, int dv, int which, cudaStream_t s) {
    if (requests <= first_req || max_query_len <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G != 0 || dv <= 0 || dv % VS != 0 || first_req < 0 || ((2 * G * DQ + H * dv) % 8) != 0) return MB_ERR_BAD_SIZE;
    if ((((uintptr_t)qkv | (uintptr_t)planes | (uintptr_t)floats) & 15) != 0) return MB_ERR_BAD_SIZE;
    if (out != nullptr && (dv > READ_COLS || gate_rows == nullptr || norm_w == nullptr || ((gate_stride | out_stride) & 3) != 0 ||
                           (((uintptr_t)gate_rows | (uintptr_t)out) & 7) != 0 || ((uintptr_t)norm_w & 15) != 0))
        return MB_ERR_BAD_SIZE;
    if (which == 0) {
        const int a_vec = a_stride % 8 == 0 && (((uintptr_t)a_rows | (uintptr_t)dt_bias) & 15) == 0;      // decays per channel by 16-byte loads
        dim3 grid((max_query_len + CH - 1) / CH, H, requests - first_req);
        if (per_channel) {
            cudaFuncSetAttribute(prepare_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_SMEM(1, dv));
            return launch_kernel(prepare_kernel<true>, grid, PREP_THREADS, PREP_SMEM(1, dv), s, 0, (const bf16*)qkv, (const bf16*)b_rows, b_stride,
                                 (const bf16*)a_rows, a_stride, rate_log, dt_bias, cu_tokens, first_req, (bf16*)planes, floats, H, G, dv, a_vec);
        }
        cudaFuncSetAttribute(prepare_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_SMEM(0, dv));
        return launch_kernel(prepare_kernel<false>, grid, PREP_THREADS, PREP_SMEM(0, dv), s, 0, (const bf16*)qkv, (const bf16*)b_rows, b_stride,
                             (const bf16*)a_rows, a_stride, rate_log, dt_bias, cu_tokens, first_req, (bf16*)planes, floats, H, G, dv, a_vec);
    }
    if (which == 1) {
        cudaFuncSetAttribute(walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WALK_SMEM);
        return launch_kernel(walk_kernel, dim3(requests - first_req, H, dv / VS), WALK_THREADS, WALK_SMEM, s, 0, (bf16*)planes, floats, state, cu_tokens, slots,
                             first_req, H, dv, error_flag);
    }
    const int parts = (dv + READ_COLS - 1) / READ_COLS, sums = READ_SUMS(dv < READ_COLS ? dv : READ_COLS);
    const int smem = sums > READ_OPERANDS ? sums : READ_OPERANDS;
    const dim3 grid((max_query_len + CH - 1) / CH, H, (requests - first_req) * parts);
    if (out != nullptr) {
        cudaFuncSetAttribute(read_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        return launch_kernel(read_kernel<true>, grid, READ_THREADS, smem, s, 0, (const bf16*)planes, (const float*)floats, cu_tokens, o, first_req, H, dv, parts,
                             (const bf16*)gate_rows, gate_stride, gate, norm_w, eps, factor, (bf16*)out, out_stride, error_flag);
    }
    cudaFuncSetAttribute(read_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return launch_kernel(read_kernel<false>, grid, READ_THREADS, smem, s, 0, (const bf16*)planes, (const float*)floats, cu_tokens, o, first_req, H, dv, parts,
                         (const bf16*)gate_rows, gate_stride, gate, norm_w, eps, factor, (bf16*)out, out_stride, error_flag);
}
