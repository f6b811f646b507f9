// Attention over a latent that keys and values share (one row of `r` numbers per position, plus `dr` rotated numbers that
// serve as a key part for every head).  Per head a the key is [W_uk_a c | k_rot] and the value W_uv_a c, so with
//     q'_a = [W_uk_a^T q_a(unrotated) | q_a(rotated)],   score = q'_a . [c | k_rot],   out_a = W_uv_a (sum_j p_j c_j)
// every head reads the same cached row: grouped-query attention with one kv head whose key is the cached row and whose
// value is the row's first r elements.  This file holds what surrounds that attention:
//   * the head preparation: rotation of the queries' rotated part into q', and (for a layer that owns its cache) the RMS
//     norm of the latent and the rotation of the shared key part, written into the page;
//   * a product per head over strided rows, out[t][a][:] = W_a x[t][a][:], used for q' (W_a = W_uk_a^T) and for the value
//     expansion (W_a = W_uv_a): the plain kernel for any size and float32, and for bf16 a tensor-core kernel (mma.sync) over
//     tiles of 64 tokens x 64 columns.
// Rotation: of the rotated part's first `rot_dims` elements, (2i, 2i + 1) or (i, i + rot_dims/2) turn by pos * inv_freq[i].
// Norms, angles and sums are float32.
#define MB_LIB "attention_latent"
#define MB_LIB_ID 16
#include "common.cuh"
#include "launch.cuh"
#include "mma_helpers.cuh"

#define LF_THREADS 128

// row: [tokens][row_stride]: H heads of (dn + dr) query numbers, then (if write_kv) r latent numbers and dr key numbers.
// q_out: [tokens][H][r + dr]; only [r, r + dr) of every head is written here.  Page rows: [r + dr] = normed latent | rotated key part.
template <typename T>
__global__ void __launch_bounds__(LF_THREADS) latent_finish_kernel(
    const T* __restrict__ row, int row_stride, T* __restrict__ q_out, const float* __restrict__ c_weight, float eps,
    const int* __restrict__ positions, const float* __restrict__ inv_freq, int rot_dims, int interleaved,
    const int* __restrict__ slot_mapping, T* __restrict__ k_cache, int H, int dn, int dr, int r, int page_size, int write_kv,
    const T* __restrict__ kv_row, int kv_stride) {
    PDL_ENTER();
    row = pdl_fresh(row); kv_row = pdl_fresh(kv_row);
    extern __shared__ float smem[];
    float* cs_tab = smem;                      // [half] cosines, [half] sines
    const int half = rot_dims >> 1;
    float* lat = smem + 2 * half;              // [r + dr]
    __shared__ float scratch[32];
    const int t = blockIdx.x;
    const T* src = row + (size_t)t * row_stride;
    if (half > 0) {
        const float pos = (float)positions[t];
        for (int i = threadIdx.x; i < half; i += LF_THREADS) {
            float sn, cs;
            sincosf(pos * inv_freq[i], &sn, &cs);
            cs_tab[i] = cs;
            cs_tab[half + i] = sn;
        }
    }
    __syncthreads();
    const int D = r + dr;
    // the queries' rotated part
    for (int idx = threadIdx.x; idx < H * dr; idx += LF_THREADS) {
        const int a = idx / dr, i = idx - a * dr;
        const T* part = src + (size_t)a * (dn + dr) + dn;
        float v = to_f32(part[i]);
        if (i < rot_dims) {
            const bool low = interleaved ? (i & 1) == 0 : i < half;
            const int j = interleaved ? i >> 1 : low ? i : i - half;
            const int other = interleaved ? i ^ 1 : low ? i + half : i - half;
            const float b = to_f32(part[other]);
            v = low ? v * cs_tab[j] - b * cs_tab[half + j] : v * cs_tab[j] + b * cs_tab[half + j];
        }
        q_out[((size_t)t * H + a) * D + r + i] = from_f32<T>(v);
    }
    if (!write_kv) return;
    const int slot = slot_mapping[t];
    // the latent and the key part: behind the queries in the same row, or (queries that went through a latent of their own
    // come from a second product) in rows of their own
    const T* kv = kv_row != nullptr ? kv_row + (size_t)t * kv_stride : src + (size_t)H * (dn + dr);
    float ss = 0.0f;
    for (int i = threadIdx.x; i < D; i += LF_THREADS) {
        const float v = to_f32(kv[i]);
        lat[i] = v;
        if (i < r) ss += v * v;
    }
    ss = block_sum(ss, scratch);               // (its barriers publish lat)
    if (slot < 0) return;
    const float factor = 1.0f / sqrtf(ss / (float)r + eps);
    T* dst = k_cache + (size_t)slot * D;       // one kv head: page * page_size + offset is the row
    for (int i = threadIdx.x; i < D; i += LF_THREADS) {
        float v;
        if (i < r) {
            v = lat[i] * factor * c_weight[i];
        } else {
            const int e = i - r;
            v = lat[i];
            if (e < rot_dims) {
                const bool low = interleaved ? (e & 1) == 0 : e < half;
                const int j = interleaved ? e >> 1 : low ? e : e - half;
                const int other = interleaved ? e ^ 1 : low ? e + half : e - half;
                const float b = lat[r + other];
                v = low ? v * cs_tab[j] - b * cs_tab[half + j] : v * cs_tab[j] + b * cs_tab[half + j];
            }
        }
        dst[i] = from_f32<T>(v);
    }
}

// The same for bf16 rows in runs of 8 numbers (16 bytes): a thread a run of a head's rotated part, and one more warp the latent, whose sum of squares goes
// by shuffles.  Bound by latency: what a token needs is asked for before the angles are worked out.  2,000 tokens of 32 heads of 64 + 32 over a latent of 128:
// 6.1 us (number by number 17.6).
#define LV_THREADS 160
__device__ __forceinline__ void lv_rotate(float* x, const float* other, int i0, int rot_dims, int interleaved, const float* cs_tab) {
    const int half = rot_dims >> 1;
    if (interleaved) {
        const int j0 = i0 >> 1;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float a = x[2 * e], b = x[2 * e + 1], cs = cs_tab[j0 + e], sn = cs_tab[half + j0 + e];
            x[2 * e] = a * cs - b * sn;
            x[2 * e + 1] = b * cs + a * sn;
        }
    } else {
        const bool low = i0 < half;
        const int j0 = low ? i0 : i0 - half;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float cs = cs_tab[j0 + e], sn = cs_tab[half + j0 + e];
            x[e] = low ? x[e] * cs - other[e] * sn : x[e] * cs + other[e] * sn;
        }
    }
}
__device__ __forceinline__ void lv_unpack(const uint4& raw, float* x) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { x[2 * e] = __uint_as_float(w[e] << 16); x[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u); }
}
__device__ __forceinline__ uint4 lv_pack(const float* x) { return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7])); }

__global__ void __launch_bounds__(LV_THREADS) latent_finish_vec_kernel(
    const bf16* __restrict__ row, int row_stride, bf16* __restrict__ q_out, const float* __restrict__ c_weight, float eps, const int* __restrict__ positions,
    const float* __restrict__ inv_freq, int rot_dims, int interleaved, const int* __restrict__ slot_mapping, bf16* __restrict__ k_cache, int H, int dn, int dr,
    int r, int write_kv, const bf16* __restrict__ kv_row, int kv_stride) {
    PDL_ENTER();
    row = pdl_fresh(row); kv_row = pdl_fresh(kv_row);
    extern __shared__ float cs_tab[];          // [half] cosines, [half] sines
    const int half = rot_dims >> 1, t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, D = r + dr;
    const bf16* src = row + (size_t)t * row_stride;
    const bool latent = warp == LV_THREADS / 32 - 1;
    const int runs = H * dr / 8, per_head = dr / 8;
    // the first run of this thread (and its partner) on its way before the angles are there
    auto take = [&](int run, uint4& mine, uint4& other) {
        const int a = run / per_head, i0 = (run - a * per_head) * 8;
        const bf16* part = src + (size_t)a * (dn + dr) + dn;
        mine = *reinterpret_cast<const uint4*>(part + i0);
        if (!interleaved && i0 < rot_dims) other = *reinterpret_cast<const uint4*>(part + (i0 < half ? i0 + half : i0 - half));
    };
    uint4 mine = make_uint4(0, 0, 0, 0), other = mine;
    const bf16* kv = kv_row != nullptr ? kv_row + (size_t)t * kv_stride : src + (size_t)H * (dn + dr);
    const int slot = write_kv ? slot_mapping[t] : -1;
    if (latent) {
        if (write_kv && lane * 8 < D) mine = *reinterpret_cast<const uint4*>(kv + lane * 8);
    } else if ((int)threadIdx.x < runs) {
        take(threadIdx.x, mine, other);
    }
    if (half > 0) {
        const float pos = (float)positions[t];
        for (int i = threadIdx.x; i < half; i += LV_THREADS) {
            float sn, cs;
            sincosf(pos * inv_freq[i], &sn, &cs);
            cs_tab[i] = cs;
            cs_tab[half + i] = sn;
        }
    }
    __syncthreads();
    if (!latent) {
        for (int run = threadIdx.x; run < runs; run += LV_THREADS - 32) {
            if (run != (int)threadIdx.x) take(run, mine, other);
            const int a = run / per_head, i0 = (run - a * per_head) * 8;
            float x[8], y[8];
            lv_unpack(mine, x);
            lv_unpack(other, y);
            if (i0 < rot_dims) lv_rotate(x, y, i0, rot_dims, interleaved, cs_tab);
            *reinterpret_cast<uint4*>(q_out + ((size_t)t * H + a) * D + r + i0) = lv_pack(x);
        }
        return;
    }
    if (!write_kv) return;
    // a lane a run of 8: the latent's, then the key part's
    float x[8], ss = 0.0f;
    lv_unpack(mine, x);
    if (lane * 8 < r)
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += x[e] * x[e];
    ss = warp_sum(ss);
    if (slot < 0 || lane * 8 >= D) return;
    bf16* dst = k_cache + (size_t)slot * D + lane * 8;
    if (lane * 8 < r) {
        const float factor = 1.0f / sqrtf(ss / (float)r + eps);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = x[e] * factor * c_weight[lane * 8 + e];
    } else {
        const int i0 = lane * 8 - r;
        if (i0 < rot_dims) {
            float y[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            if (!interleaved) lv_unpack(*reinterpret_cast<const uint4*>(kv + r + (i0 < half ? i0 + half : i0 - half)), y);
            lv_rotate(x, y, i0, rot_dims, interleaved, cs_tab);
        }
    }
    *reinterpret_cast<uint4*>(dst) = lv_pack(x);
}

MB_API int mb_latent_finish(const void* row, int row_stride, int dtype, void* q_out, const float* c_weight, float eps, const int* positions,
                            const float* inv_freq, int rot_dims, int interleaved, const int* slot_mapping, void* k_cache, int tokens, int H,
                            int dn, int dr, int r, int page_size, int write_kv, const void* kv_row, int kv_stride, cudaStream_t s) {
    if (tokens <= 0) return 0;
    if (H <= 0 || dn < 0 || dr < 0 || r <= 0 || rot_dims < 0 || rot_dims > dr || (rot_dims & 1)) return MB_ERR_BAD_SIZE;
    if (inv_freq == nullptr) rot_dims = 0;
    const size_t smem = (size_t)(rot_dims + r + dr) * sizeof(float);
    if (smem > 48 * 1024) return MB_ERR_BAD_SIZE;
    if (dtype == MB_F32)
        return launch_kernel(latent_finish_kernel<float>, tokens, LF_THREADS, smem, s, 0, (const float*)row, row_stride, (float*)q_out, c_weight,
                             eps, positions, inv_freq, rot_dims, interleaved, slot_mapping, (float*)k_cache, H, dn, dr, r, page_size, write_kv,
                             (const float*)kv_row, kv_stride);
    // rows in whole runs of 8 numbers on 16-byte boundaries, a latent and key part of a warp at most, rotated parts in whole runs (half-split: both halves)
    if (dtype == MB_BF16 && dn % 8 == 0 && dr % 8 == 0 && r % 8 == 0 && (interleaved ? rot_dims % 8 == 0 : rot_dims % 16 == 0) && row_stride % 8 == 0 &&
        kv_stride % 8 == 0 && r + dr <= 256 && ((((uintptr_t)row | (uintptr_t)q_out | (uintptr_t)k_cache | (uintptr_t)kv_row) & 15) == 0))
        return launch_kernel(latent_finish_vec_kernel, tokens, LV_THREADS, (size_t)rot_dims * sizeof(float), s, 0, (const bf16*)row, row_stride, (bf16*)q_out,
                             c_weight, eps, positions, inv_freq, rot_dims, interleaved, slot_mapping, (bf16*)k_cache, H, dn, dr, r, write_kv,
                             (const bf16*)kv_row, kv_stride);
    if (dtype == MB_BF16)
        return launch_kernel(latent_finish_kernel<bf16>, tokens, LF_THREADS, smem, s, 0, (const bf16*)row, row_stride, (bf16*)q_out, c_weight,
                             eps, positions, inv_freq, rot_dims, interleaved, slot_mapping, (bf16*)k_cache, H, dn, dr, r, page_size, write_kv,
                             (const bf16*)kv_row, kv_stride);
    return MB_ERR_BAD_DTYPE;
}

// ---- a product per head: out[t][a][n] = sum_k w[a][n][k] x[t][a][k] -------------------------------------------------------
// x: element (t, a, k) at x + t x_ld + a x_head + k;  w: [H][N][K];  out: element (t, a, n) at out + t o_ld + a o_head + n.
// Plain kernel: a block per (token, head, run of HP_COLS output columns); a warp per column, lanes along k in a fixed order,
// so a token's result does not depend on the batch.  (Few tokens bring few blocks otherwise: a single-token step of eight
// requests took 28 us for a product of half a megabyte of weights with one block per token and head.)
#define HP_THREADS 128
#define HP_COLS 16
template <typename T>
__global__ void __launch_bounds__(HP_THREADS) heads_product_kernel(const T* __restrict__ x, int x_ld, int x_head, const T* __restrict__ w,
                                                                   T* __restrict__ out, int o_ld, int o_head, int N, int K) {
    PDL_ENTER();
    x = pdl_fresh(x);
    extern __shared__ float xs[];              // [K]
    const int t = blockIdx.x, a = blockIdx.y;
    const T* xr = x + (size_t)t * x_ld + (size_t)a * x_head;
    for (int k = threadIdx.x; k < K; k += HP_THREADS) xs[k] = to_f32(xr[k]);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* wa = w + (size_t)a * N * K;
    T* dst = out + (size_t)t * o_ld + (size_t)a * o_head;
    const int n_end = min(N, (int)(blockIdx.z + 1) * HP_COLS);
    for (int n = blockIdx.z * HP_COLS + warp; n < n_end; n += HP_THREADS / 32) {
        const T* wr = wa + (size_t)n * K;
        float dot = 0.0f;
        for (int k = lane; k < K; k += 32) dot = fmaf(xs[k], to_f32(wr[k]), dot);
        dot = warp_sum(dot);
        if (lane == 0) dst[n] = from_f32<T>(dot);
    }
}

// bf16 on the tensor cores: a CTA takes 64 tokens x COLS columns of one head (all 128 of a latent at once, so that x is read once); K in steps of 64
// (zero-filled past K) through two buffers; rows of x and w must start on 16-byte boundaries (K, x_ld, x_head multiples of 8).  Bound by the bytes of x and the
// results, which leave through shared memory in 16-byte stores where rows allow.  2,000 tokens of 32 heads, 64 numbers to 128 and 128 to 64: 9.0 and 9.3 us (by 64 x 64 with 4-byte
// stores 11.5 each).
#define HT_M 64
#define HT_K 64
#define HT_LD (HT_K + 8)
template <int COLS> struct HtTile {
    static constexpr int STAGE = (HT_M + COLS) * HT_LD, OUT_LD = COLS + 8;
    static constexpr int SMEM = 2 * STAGE * 2;
    static_assert(HT_M * OUT_LD <= 2 * STAGE, "the results fit where the operands were");
};
template <int COLS>
__global__ void __launch_bounds__(256) heads_product_tc_kernel(const bf16* __restrict__ x, int x_ld, int x_head, const bf16* __restrict__ w,
                                                               bf16* __restrict__ out, int o_ld, int o_head, int T, int N, int K, int wide) {
    typedef HtTile<COLS> S;
    PDL_ENTER();
    x = pdl_fresh(x);
    extern __shared__ __align__(16) uint8_t ht_smem[];
    bf16* smem = reinterpret_cast<bf16*>(ht_smem);
    const int a = blockIdx.x, n0 = blockIdx.y * COLS, t0 = blockIdx.z * HT_M;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = warp & 3, wn = warp >> 2;      // 16 tokens, half of the columns
    const bf16* xa = x + (size_t)a * x_head;
    const bf16* wa = w + (size_t)a * N * K;
    auto load = [&](int buf, int k0) {
#pragma unroll
        for (int i = 0; i < (HT_M + COLS) * (HT_K / 8); i += 256) {
            const int idx = i + threadIdx.x, rr = idx / (HT_K / 8), k = k0 + idx % (HT_K / 8) * 8;
            bf16* d = smem + buf * S::STAGE + rr * HT_LD + idx % (HT_K / 8) * 8;
            const bool of_x = rr < HT_M;
            const bool there = k < K && (of_x ? t0 + rr < T : n0 + rr - HT_M < N);
            if (there) cp_async16(d, of_x ? xa + (size_t)(t0 + rr) * x_ld + k : wa + (size_t)(n0 + rr - HT_M) * K + k);
            else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
        }
    };
    float acc[COLS / 16][4];
#pragma unroll
    for (int j = 0; j < COLS / 16; ++j) { acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f; }
    const int nk = (K + HT_K - 1) / HT_K;
    load(0, 0);
    cp_async_commit();
    for (int kt = 0; kt < nk; ++kt) {
        const int buf = kt & 1;
        if (kt + 1 < nk) load(buf ^ 1, (kt + 1) * HT_K);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const bf16* st = smem + buf * S::STAGE;
        const uint32_t a_addr = (uint32_t)__cvta_generic_to_shared(st + (wm * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * HT_LD + (lane >> 4) * 8);
        const uint32_t b_addr = (uint32_t)__cvta_generic_to_shared(st + (HT_M + wn * (COLS / 2) + (lane & 7) + (lane >> 4) * 8) * HT_LD + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int kk = 0; kk < HT_K / 16; ++kk) {
            uint32_t fa[4];
            ldsm_x4(a_addr + kk * 32, fa[0], fa[1], fa[2], fa[3]);
#pragma unroll
            for (int j = 0; j < COLS / 16; j += 2) {
                uint32_t b0, b1, b2, b3;
                ldsm_x4(b_addr + (uint32_t)(j * 8 * HT_LD * 2 + kk * 32), b0, b1, b2, b3);
                mma_bf16_16816(acc[j], fa, b0, b1);
                mma_bf16_16816(acc[j + 1], fa, b2, b3);
            }
        }
        __syncthreads();                       // everyone is done with this buffer before the load after next fills it
    }
    cp_async_wait<0>();
    if (wide) {
        // rows of whole 16-byte pieces: through shared memory
#pragma unroll
        for (int rr = 0; rr < 2; ++rr)
#pragma unroll
            for (int j = 0; j < COLS / 16; ++j)
                *reinterpret_cast<uint32_t*>(smem + (wm * 16 + (lane >> 2) + 8 * rr) * S::OUT_LD + wn * (COLS / 2) + j * 8 + 2 * (lane & 3)) = pack_bf16(acc[j][2 * rr], acc[j][2 * rr + 1]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < HT_M * (COLS / 8); i += 256) {
            const int idx = i + threadIdx.x, rr = idx / (COLS / 8), c = idx % (COLS / 8) * 8;
            if (t0 + rr < T && n0 + c < N) *reinterpret_cast<uint4*>(out + (size_t)(t0 + rr) * o_ld + (size_t)a * o_head + n0 + c) = *reinterpret_cast<const uint4*>(smem + rr * S::OUT_LD + c);
        }
        return;
    }
    const int col = n0 + wn * (COLS / 2) + 2 * (lane & 3);
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        const int t = t0 + wm * 16 + (lane >> 2) + 8 * rr;
        if (t >= T) continue;
        bf16* dst = out + (size_t)t * o_ld + (size_t)a * o_head;
#pragma unroll
        for (int j = 0; j < COLS / 16; ++j) {
            const int c = col + j * 8;
            if (c + 1 < N) *reinterpret_cast<uint32_t*>(dst + c) = pack_bf16(acc[j][2 * rr], acc[j][2 * rr + 1]);
            else if (c < N) dst[c] = __float2bfloat16_rn(acc[j][2 * rr]);
        }
    }
}

template <int COLS>
static int launch_heads_tc(const void* x, int x_ld, int x_head, const void* w, void* out, int o_ld, int o_head, int tokens, int H, int N, int K, cudaStream_t s) {
    auto kernel = heads_product_tc_kernel<COLS>;
    static LaunchSmem smem;
    const int rc = smem.allow(kernel, HtTile<COLS>::SMEM);
    if (rc) return rc;
    const int wide = N % 8 == 0 && o_ld % 8 == 0 && o_head % 8 == 0 && (((uintptr_t)out) & 15) == 0;
    return launch_kernel(kernel, dim3(H, (N + COLS - 1) / COLS, (tokens + HT_M - 1) / HT_M), 256, HtTile<COLS>::SMEM, s, 0, (const bf16*)x, x_ld, x_head,
                         (const bf16*)w, (bf16*)out, o_ld, o_head, tokens, N, K, wide);
}

static bool aligned16(const void* p) { return (((uintptr_t)p) & 15) == 0; }

// fast: 1 asks for the tensor-core kernel where the layout allows (bf16, rows on 16-byte boundaries, even output offsets).
MB_API int mb_heads_product(const void* x, int x_ld, int x_head, const void* w, void* out, int o_ld, int o_head, int dtype, int tokens, int H,
                            int N, int K, int fast, cudaStream_t s) {
    if (tokens <= 0) return 0;
    if (H <= 0 || N <= 0 || K <= 0 || (size_t)K * 4 > 48 * 1024) return MB_ERR_BAD_SIZE;
    if (dtype == MB_BF16 && fast && K % 8 == 0 && x_ld % 8 == 0 && x_head % 8 == 0 && o_ld % 2 == 0 && o_head % 2 == 0 && aligned16(x) &&
        aligned16(w) && (((uintptr_t)out) & 3) == 0 && tokens >= 16 && tokens <= 65535 * HT_M)
        return N > 64 ? launch_heads_tc<128>(x, x_ld, x_head, w, out, o_ld, o_head, tokens, H, N, K, s) : launch_heads_tc<64>(x, x_ld, x_head, w, out, o_ld, o_head, tokens, H, N, K, s);
    dim3 grid(tokens, H, (N + HP_COLS - 1) / HP_COLS);
    if (dtype == MB_F32)
        return launch_kernel(heads_product_kernel<float>, grid, HP_THREADS, (size_t)K * 4, s, 0, (const float*)x, x_ld, x_head, (const float*)w,
                             (float*)out, o_ld, o_head, N, K);
    if (dtype == MB_BF16)
        return launch_kernel(heads_product_kernel<bf16>, grid, HP_THREADS, (size_t)K * 4, s, 0, (const bf16*)x, x_ld, x_head, (const bf16*)w,
                             (bf16*)out, o_ld, o_head, N, K);
    return MB_ERR_BAD_DTYPE;
}
