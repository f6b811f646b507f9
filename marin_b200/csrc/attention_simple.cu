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
// Bound by the multiply-adds: a lane is a row, its query lies in registers, and a warp's lanes read the same key or value, which is
// one cycle of shared memory for 16 bytes (two rows x four keys a thread took three times the multiply-adds' cycles).  The keys' and values' half
// chunks arrive by cp.async one ahead of the arithmetic.  Measured on B200 (333 tokens, 16 heads of 128 over 8 kv heads):
// attention_simple_kernel 605 us.
#define AT_ROWS 32
#define AT_THREADS 128
#define AT_WARPS (AT_THREADS / 32)
#define AT_CHUNK AS_THREADS
#define AT_HALF 64
#define AT_LD 132                     // floats a row of 128 takes in shared memory
#define AT_PLD 33                     // floats a key's 32 scores take
#define AT_SMEM ((2 * AT_HALF * AT_LD + AT_CHUNK * AT_PLD + AT_ROWS) * 4)

template <int DM>                     // the most numbers of a head: 64 or 128
__global__ void __launch_bounds__(AT_THREADS) attention_tile_kernel(
    const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache, float* __restrict__ out,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens,
    int first_req, int H, int K, int d, int page_size, float scale) {
    PDL_ENTER();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); v_cache = pdl_fresh(v_cache);
    extern __shared__ __align__(16) float at_smem[];
    float* sKV = at_smem;                                  // two half chunks of keys or values in turn, rows of AT_LD
    float* sP = sKV + 2 * AT_HALF * AT_LD;                 // [128 keys][33]: scores of the 32 rows, then weights
    float* sCorr = sP + AT_CHUNK * AT_PLD;                 // [rows]
    const int G = H / K, per_tile = AT_ROWS / G;
    const int r = first_req + blockIdx.z, kh = blockIdx.y;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    const int q0 = (gridDim.x - 1 - blockIdx.x) * per_tile;                   // (the longest walks first)
    if (q0 >= n) return;
    const int queries = min(per_tile, n - q0), rows = queries * G;
    const int pos0 = seq_lens[r] - n + q0, last = pos0 + queries - 1;         // positions of the tile's first and last query
    const int* table = block_table + (size_t)r * max_pages;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d4 = d >> 2;
    const bool mine = lane < rows;                         // this lane's row: query lane / G, head lane % G of the group
    const int my_pos = pos0 + lane / G;
    const size_t my_row = ((size_t)(tok0 + q0 + lane / G) * H + kh * G + lane % G) * d;

    float4 qr[DM / 4];
#pragma unroll
    for (int c = 0; c < DM / 4; ++c) qr[c] = mine && c < d4 ? *reinterpret_cast<const float4*>(q + my_row + 4 * c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
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
    constexpr int KEYS = 8, COLS = DM / AT_WARPS;          // keys whose sums run side by side; columns of the values a warp has
    constexpr int OWN = AT_ROWS / AT_WARPS;                // rows whose softmax a warp does
    float m[OWN], l[OWN], acc[COLS];
#pragma unroll
    for (int i = 0; i < OWN; ++i) { m[i] = -INFINITY; l[i] = 0.0f; }
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
    for (int stage = 0; stage < stages; ++stage) {
        const int base = (stage >> 2) * AT_CHUNK, off = (stage & 1) * AT_HALF;
        cp_async_wait<0>();
        __syncthreads();                                   // this half is there, and nobody works on the other buffer any more
        if (stage + 1 < stages) fetch(stage + 1);
        const float* kv = sKV + (stage & 1) * AT_HALF * AT_LD;
        if (!(stage & 2)) {
#pragma unroll 1
            for (int k0 = warp * KEYS; k0 < AT_HALF; k0 += AT_WARPS * KEYS) {
                float s[KEYS];
#pragma unroll
                for (int j = 0; j < KEYS; ++j) s[j] = 0.0f;
#pragma unroll
                for (int c = 0; c < DM / 4; ++c) {
                    if (c >= d4) break;
#pragma unroll
                    for (int j = 0; j < KEYS; ++j) {
                        const float4 k = *reinterpret_cast<const float4*>(kv + (k0 + j) * AT_LD + 4 * c);
                        s[j] = fmaf(qr[c].w, k.w, fmaf(qr[c].z, k.z, fmaf(qr[c].y, k.y, fmaf(qr[c].x, k.x, s[j]))));
                    }
                }
#pragma unroll
                for (int j = 0; j < KEYS; ++j) sP[(off + k0 + j) * AT_PLD + lane] = base + off + k0 + j <= my_pos ? s[j] * scale : -INFINITY;
            }
            if (!(stage & 1)) continue;
            __syncthreads();                               // the chunk's scores are all there
#pragma unroll
            for (int i = 0; i < OWN; ++i) {
                const int row = OWN * warp + i, pos = pos0 + row / G;
                if (row >= rows) continue;
                float* p = sP + lane * AT_PLD + row;       // a lane a key
                const float s0 = p[0], s1 = p[32 * AT_PLD], s2 = p[64 * AT_PLD], s3 = p[96 * AT_PLD];
                const float m_new = fmaxf(m[i], warp_max(fmaxf(fmaxf(s0, s1), fmaxf(s2, s3))));
                const float corr = expf(m[i] - m_new);
                const int key = base + lane;
                const float p0 = key <= pos ? expf(s0 - m_new) : 0.0f, p1 = key + 32 <= pos ? expf(s1 - m_new) : 0.0f;
                const float p2 = key + 64 <= pos ? expf(s2 - m_new) : 0.0f, p3 = key + 96 <= pos ? expf(s3 - m_new) : 0.0f;
                p[0] = p0; p[32 * AT_PLD] = p1; p[64 * AT_PLD] = p2; p[96 * AT_PLD] = p3;
                const float sum = (warp_sum(p0) + warp_sum(p2)) + (warp_sum(p1) + warp_sum(p3));      // block_sum's order
                l[i] = fmaf(l[i], corr, sum);
                m[i] = m_new;
                if (lane == 0) sCorr[row] = corr;
            }
            continue;                                      // (the barrier at the top of the next stage publishes the weights)
        }
        if (!(stage & 1)) {
            const float corr = mine ? sCorr[lane] : 1.0f;
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] *= corr;
        }
        if (warp * COLS >= d) continue;
        const float* p = sP + off * AT_PLD + lane;
        const int seen = mine ? my_pos - base - off + 1 : 0;                 // keys of this half the row sees (may be beyond it)
        const int whole = min(AT_HALF, max(0, pos0 - base - off + 1));       // keys that every row of the tile sees
        auto add = [&](int j, bool all) {
            const float w = p[j * AT_PLD];
            if (!all && j >= seen) return;
#pragma unroll
            for (int c = 0; c < COLS; c += 4) {
                const float4 v = *reinterpret_cast<const float4*>(kv + j * AT_LD + warp * COLS + c);
                acc[c] = fmaf(w, v.x, acc[c]); acc[c + 1] = fmaf(w, v.y, acc[c + 1]); acc[c + 2] = fmaf(w, v.z, acc[c + 2]); acc[c + 3] = fmaf(w, v.w, acc[c + 3]);
            }
        };
        int j = 0;
#pragma unroll 4
        for (; j < whole; ++j) add(j, true);
        for (; j < min(AT_HALF, last - base - off + 1); ++j) add(j, false);
    }
    __syncthreads();                                       // (sCorr takes the sums now)
#pragma unroll
    for (int i = 0; i < OWN; ++i)
        if (lane == 0) sCorr[OWN * warp + i] = l[i];
    __syncthreads();
    if (!mine) return;
    const float sum = sCorr[lane];
#pragma unroll
    for (int c = 0; c < COLS; c += 4)
        if (warp * COLS + c < d)
            *reinterpret_cast<float4*>(out + my_row + warp * COLS + c) = make_float4(acc[c] / sum, acc[c + 1] / sum, acc[c + 2] / sum, acc[c + 3] / sum);
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
    auto kernel = d <= 64 ? attention_tile_kernel<64> : attention_tile_kernel<128>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM);
    dim3 grid((max_query_len + per_tile - 1) / per_tile, K, count);
    return launch_kernel(kernel, grid, AT_THREADS, AT_SMEM, s, 0, (const float*)q, (const float*)k_cache, (const float*)v_cache,
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
