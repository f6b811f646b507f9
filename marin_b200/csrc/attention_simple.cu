// Plain causal grouped-query attention over the paged cache: one block per (token, query head), keys
// in chunks of 128 with an online softmax in float32.  It serves prompt portions and decoded tokens
// alike, any head size, with or without a window.  It is the 32-bit path's attention and the plain twin
// of the fast kernels (the reference's generic kernel has the same shape, crates/cuda/src/attention.cu:6-96).
// Prompt portions of the 32-bit path run as tiles of 32 rows (attention_tile_kernel below) that do every row's arithmetic in the same
// order, bit for bit.
// Page layout: [page][kv_head][offset in page][d].
#define MB_LIB "attention_simple"
#define MB_LIB_ID 7
#include "common.cuh"
#include "launch.cuh"
#include "mma_helpers.cuh"

#define AS_THREADS 128
#define AS_MAX_D_PER_THREAD 4

template <typename T>
__global__ void __launch_bounds__(AS_THREADS) attention_simple_kernel(
    const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache, T* __restrict__ out,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ req_index,
    const int* __restrict__ positions, int H, int K, int d, int page_size, float scale, int window) {
    PDL_ENTER();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); v_cache = pdl_fresh(v_cache);
    extern __shared__ float smem[];
    float* qs = smem;                 // [d]
    float* ps = smem + d;             // [AS_THREADS]
    float* scratch = ps + AS_THREADS; // [32]
    const int t = blockIdx.x, head = blockIdx.y;
    const int kh = head / (H / K);
    const int req = req_index[t];
    const int pos = positions[t];
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int* table = block_table + (size_t)req * max_pages;
    const T* qrow = q + ((size_t)t * H + head) * d;
    for (int i = threadIdx.x; i < d; i += AS_THREADS) qs[i] = to_f32(qrow[i]);
    __syncthreads();

    float m = -INFINITY, l = 0.0f;
    float acc[AS_MAX_D_PER_THREAD];
#pragma unroll
    for (int r = 0; r < AS_MAX_D_PER_THREAD; ++r) acc[r] = 0.0f;

    for (int base = lo; base <= pos; base += AS_THREADS) {
        const int key = base + threadIdx.x;
        float s = -INFINITY;
        if (key <= pos) {
            const size_t page = (size_t)table[key / page_size];
            const T* krow = k_cache + ((page * K + kh) * page_size + (size_t)(key % page_size)) * d;
            float dot = 0.0f;
            for (int i = 0; i < d; ++i) dot = fmaf(qs[i], to_f32(krow[i]), dot);
            s = dot * scale;
        }
        const float chunk_max = block_max(s, scratch);
        const float m_new = fmaxf(m, chunk_max);
        const float corr = expf(m - m_new);   // exp(-inf) = 0 on the first chunk
        const float p = key <= pos ? expf(s - m_new) : 0.0f;
        __syncthreads();
        ps[threadIdx.x] = p;
        const float chunk_sum = block_sum(p, scratch);  // has the barriers that publish ps
        l = fmaf(l, corr, chunk_sum);
        m = m_new;
        const int count = min(AS_THREADS, pos - base + 1);
#pragma unroll
        for (int r = 0; r < AS_MAX_D_PER_THREAD; ++r) {
            const int dd = threadIdx.x + r * AS_THREADS;
            if (dd < d) {
                float a = acc[r] * corr;
                for (int j = 0; j < count; ++j) {
                    const int kj = base + j;
                    const size_t page = (size_t)table[kj / page_size];
                    const T* vrow = v_cache + ((page * K + kh) * page_size + (size_t)(kj % page_size)) * d;
                    a = fmaf(ps[j], to_f32(vrow[dd]), a);
                }
                acc[r] = a;
            }
        }
        __syncthreads();
    }
    T* orow = out + ((size_t)t * H + head) * d;
#pragma unroll
    for (int r = 0; r < AS_MAX_D_PER_THREAD; ++r) {
        const int dd = threadIdx.x + r * AS_THREADS;
        if (dd < d) orow[dd] = from_f32<T>(acc[r] / l);
    }
}

// Prompt portions in float32, every key visible up to a query's own position: a block takes up to 32 rows (consecutive queries of one
// request x the query heads of one kv head) over the keys in the same chunks of 128, so that a key and a value are fetched once for
// 32 rows instead of once for each.  A row's numbers are made in attention_simple_kernel's order (a score summed over d from 0 up, a chunk's
// sum as its warps' butterflies, values added key by key, chunks from position 0 on; a chunk behind a row's position changes nothing),
// so a token's result is the same bits whichever kernel it went through and however the prompt was cut.
// Bound by shared memory and the multiply-adds: a 16-byte load takes four cycles of a warp whatever it reads, so scores are made 4 rows x 4 keys a thread
// and values added 4 rows x 8 columns (1.5 to 2 cycles of loads for one of multiply-adds).  The keys' and values' half chunks arrive by cp.async one
// ahead of the arithmetic.  Measured on B200 (333 tokens, 16 heads of 128 over 8 kv heads): attention_simple_kernel 605 us, this
// one 88 us; with 2 x 4 and 2 x 8 a thread, or a lane a row with its query in registers and every key read by the whole warp, 115 us.
#define AT_ROWS 32
#define AT_THREADS 128
#define AT_WARPS (AT_THREADS / 32)
#define AT_CHUNK AS_THREADS
#define AT_HALF 64
#define AT_LD 132                     // floats a row of 128 takes in shared memory
#define AT_SMEM ((2 * AT_ROWS * AT_LD + 2 * AT_HALF * AT_LD + AT_ROWS) * 4)

__global__ void __launch_bounds__(AT_THREADS, 2) attention_tile_kernel(
    const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache, float* __restrict__ out,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens,
    int first_req, int H, int K, int d, int page_size, float scale) {
    PDL_ENTER();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); v_cache = pdl_fresh(v_cache);
    extern __shared__ __align__(16) float at_smem[];
    float* sQ = at_smem;                                   // [rows][d]
    float* sP = sQ + AT_ROWS * AT_LD;                      // [rows][128]: scores, then weights
    float* sKV = sP + AT_ROWS * AT_LD;                     // two half chunks of keys or values in turn
    float* sCorr = sKV + 2 * AT_HALF * AT_LD;              // [rows]
    const int G = H / K, per_tile = AT_ROWS / G;
    const int r = first_req + blockIdx.z, kh = blockIdx.y;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    const int q0 = (gridDim.x - 1 - blockIdx.x) * per_tile;                   // (the longest walks first)
    if (q0 >= n) return;
    const int queries = min(per_tile, n - q0), rows = queries * G;
    const int pos0 = seq_lens[r] - n + q0, last = pos0 + queries - 1;         // positions of the tile's first and last query
    const int* table = block_table + (size_t)r * max_pages;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d4 = d >> 2;

    // stage: chunk * 4 + {0, 1: its keys' halves; 2, 3: its values' halves}
    auto fetch = [&](int stage) {
        const float* src = (stage & 2) ? v_cache : k_cache;
        float* dst = sKV + (stage & 1) * AT_HALF * AT_LD;
        const int key0 = (stage >> 2) * AT_CHUNK + (stage & 1) * AT_HALF;
        for (int row = warp; row < AT_HALF; row += AT_WARPS) {               // a warp a row
            const int key = key0 + row;
            float* to = dst + row * AT_LD + 4 * lane;
            if (lane >= d4) continue;
            if (key <= last) cp_async16(to, src + (((size_t)table[key / page_size] * K + kh) * page_size + (size_t)(key % page_size)) * d + 4 * lane);
            else *reinterpret_cast<float4*>(to) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        cp_async_commit();
    };
    const int chunks = last / AT_CHUNK + 1, stages = chunks * 4;
    fetch(0);
    for (int row = warp; row < AT_ROWS; row += AT_WARPS) {
        if (lane >= d4) continue;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row < rows) v = *reinterpret_cast<const float4*>(q + ((size_t)(tok0 + q0 + row / G) * H + kh * G + row % G) * d + 4 * lane);
        *reinterpret_cast<float4*>(sQ + row * AT_LD + 4 * lane) = v;
    }
    // scores: rows ty + 8 i x keys tx + 16 j; values: rows 4 ty + i x columns 4 tx.. and 64 + 4 tx..; softmax: rows 8 warp ..
    const int tx = tid & 15, ty = tid >> 4;
    constexpr int OWN = AT_ROWS / AT_WARPS;
    float m[OWN], l[OWN], acc[4][8];
    int row_pos[4];                                        // (of rows that are not there: nobody reads their results)
#pragma unroll
    for (int i = 0; i < OWN; ++i) { m[i] = -INFINITY; l[i] = 0.0f; }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        row_pos[i] = pos0 + (4 * ty + i) / G;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    }
    for (int stage = 0; stage < stages; ++stage) {
        const int base = (stage >> 2) * AT_CHUNK, off = (stage & 1) * AT_HALF;
        cp_async_wait<0>();
        __syncthreads();                                   // this half is there, and nobody works on the other buffer any more
        if (stage + 1 < stages) fetch(stage + 1);
        const float* kv = sKV + (stage & 1) * AT_HALF * AT_LD;
        if (!(stage & 2)) {
            float s[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 2
            for (int c = 0; c < d4; ++c) {
                float4 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(sQ + (ty + 8 * i) * AT_LD + 4 * c);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 k = *reinterpret_cast<const float4*>(kv + (tx + 16 * j) * AT_LD + 4 * c);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        s[i][j] = fmaf(a[i].w, k.w, fmaf(a[i].z, k.z, fmaf(a[i].y, k.y, fmaf(a[i].x, k.x, s[i][j]))));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = ty + 8 * i, pos = pos0 + row / G;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = off + tx + 16 * j;
                    sP[row * AT_LD + key] = base + key <= pos ? s[i][j] * scale : -INFINITY;
                }
            }
            if (!(stage & 1)) continue;
            __syncthreads();                               // the chunk's scores are all there
#pragma unroll
            for (int i = 0; i < OWN; ++i) {
                const int row = OWN * warp + i, pos = pos0 + row / G;
                if (row >= rows) continue;
                float* p = sP + row * AT_LD + lane;        // a lane a key
                const float s0 = p[0], s1 = p[32], s2 = p[64], s3 = p[96];
                const float m_new = fmaxf(m[i], warp_max(fmaxf(fmaxf(s0, s1), fmaxf(s2, s3))));
                const float corr = expf(m[i] - m_new);
                const int key = base + lane;
                const float p0 = key <= pos ? expf(s0 - m_new) : 0.0f, p1 = key + 32 <= pos ? expf(s1 - m_new) : 0.0f;
                const float p2 = key + 64 <= pos ? expf(s2 - m_new) : 0.0f, p3 = key + 96 <= pos ? expf(s3 - m_new) : 0.0f;
                p[0] = p0; p[32] = p1; p[64] = p2; p[96] = p3;
                const float sum = (warp_sum(p0) + warp_sum(p2)) + (warp_sum(p1) + warp_sum(p3));      // block_sum's order
                l[i] = fmaf(l[i], corr, sum);
                m[i] = m_new;
                if (lane == 0) sCorr[row] = corr;
            }
            continue;                                      // (the barrier at the top of the next stage publishes the weights)
        }
        if (!(stage & 1)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float corr = 4 * ty + i < rows ? sCorr[4 * ty + i] : 1.0f;
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] *= corr;
            }
        }
        const float* p = sP + 4 * ty * AT_LD + off;
        const int first = base + off;
        // four keys at a time; `all`: every row of the tile sees them
        auto add = [&](int j, bool all) {
            float w[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(w[i]) = *reinterpret_cast<const float4*>(p + i * AT_LD + j);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* row = kv + (j + e) * AT_LD + 4 * tx;
                const float4 lo = *reinterpret_cast<const float4*>(row), hi = *reinterpret_cast<const float4*>(row + 64);
                const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!all && first + j + e > row_pos[i]) continue;
#pragma unroll
                    for (int c = 0; c < 8; ++c) acc[i][c] = fmaf(w[i][e], v[c], acc[i][c]);
                }
            }
        };
        const int whole = min(AT_HALF, max(0, pos0 - first + 1)) & ~3, most = min(AT_HALF, last - first + 1);
        int j = 0;
#pragma unroll 1
        for (; j < whole; j += 4) add(j, true);
#pragma unroll 1
        for (; j < most; j += 4) add(j, false);
    }
    __syncthreads();                                       // (sCorr takes the sums now)
#pragma unroll
    for (int i = 0; i < OWN; ++i)
        if (lane == 0) sCorr[OWN * warp + i] = l[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = 4 * ty + i;
        if (row >= rows) continue;
        float* o = out + ((size_t)(tok0 + q0 + row / G) * H + kh * G + row % G) * d;
        const float sum = sCorr[row];
#pragma unroll
        for (int c = 0; c < 8; c += 4) {
            const int col = c * 16 + 4 * tx;
            if (col < d) *reinterpret_cast<float4*>(o + col) = make_float4(acc[i][c] / sum, acc[i][c + 1] / sum, acc[i][c + 2] / sum, acc[i][c + 3] / sum);
        }
    }
}

// Float32 prompt portions: requests first_req .. first_req + count - 1, every earlier key visible; heads of up to 128 in whole 16-byte
// steps, up to 32 query heads a kv head.
MB_API int mb_attention_tile(const void* q, const void* k_cache, const void* v_cache, void* out, const int* block_table, int max_pages,
                             const int* cu_tokens, const int* seq_lens, int first_req, int count, int max_query_len, int H, int K, int d,
                             int page_size, float scale, cudaStream_t s) {
    if (count <= 0 || max_query_len <= 0) return 0;
    if (d <= 0 || d > 128 || d % 4 != 0 || K <= 0 || H % K != 0 || H / K > AT_ROWS || page_size <= 0) return MB_ERR_BAD_SIZE;
    const int per_tile = AT_ROWS / (H / K);
    if ((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) != 0) return MB_ERR_BAD_SIZE;
    cudaFuncSetAttribute(attention_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM);
    dim3 grid((max_query_len + per_tile - 1) / per_tile, K, count);
    return launch_kernel(attention_tile_kernel, grid, AT_THREADS, AT_SMEM, s, 0, (const float*)q, (const float*)k_cache, (const float*)v_cache,
                         (float*)out, block_table, max_pages, cu_tokens, seq_lens, first_req, H, K, d, page_size, scale);
}

MB_API int mb_attention_simple(const void* q, const void* k_cache, const void* v_cache, void* out, int dtype,
                               const int* block_table, int max_pages, const int* req_index, const int* positions,
                               int tokens, int H, int K, int d, int page_size, float scale, int window,
                               cudaStream_t s) {
    if (tokens <= 0) return 0;
    if (d <= 0 || d > AS_THREADS * AS_MAX_D_PER_THREAD || K <= 0 || H % K != 0) return MB_ERR_BAD_SIZE;
    dim3 grid(tokens, H);
    const size_t smem = (size_t)(d + AS_THREADS + 32) * sizeof(float);
    if (dtype == MB_F32)
        return launch_kernel(attention_simple_kernel<float>, grid, AS_THREADS, smem, s, 0,
            (const float*)q, (const float*)k_cache, (const float*)v_cache, (float*)out, block_table, max_pages,
            req_index, positions, H, K, d, page_size, scale, window);
    else if (dtype == MB_BF16)
        return launch_kernel(attention_simple_kernel<bf16>, grid, AS_THREADS, smem, s, 0,
            (const bf16*)q, (const bf16*)k_cache, (const bf16*)v_cache, (bf16*)out, block_table, max_pages,
            req_index, positions, H, K, d, page_size, scale, window);
    else return MB_ERR_BAD_DTYPE;
    return mb_last_error();
}
