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
// and values added 4 rows x 8 columns (half a cycle of loads for one of multiply-adds).  The keys' and values' half chunks arrive by cp.async one
// ahead of the arithmetic.  A few hundred tokens are few blocks, and the block with the last queries walks all keys while the first ones are long done: such a
// step goes by 16 rows and 64 threads a block, twice as many blocks of half the length.  Measured on B200 (333 tokens, 16 heads of 128 over 8 kv heads):
// attention_simple_kernel 605 us; by 32 rows, a half's rows looked up behind a division each (2,300 clocks a half) and the softmax row by row
// (6,000 a chunk) 88 us; rows looked up side by side 72; the softmax's rows interleaved and 16 rows a block 57 (400 tokens, 32 heads over 8, 32 rows
// a block: 109 and 91); all heads' last tiles first 45.  With 4 x 2 and 4 x 4 a thread and twice the threads 65.
#define AT_CHUNK AS_THREADS
#define AT_HALF 64
#define AT_LD 132                     // floats a row of 128 takes in shared memory
#define AT_SMEM(rows) ((2 * (rows) * AT_LD + 2 * AT_HALF * AT_LD + (rows)) * 4)

template <int AT_ROWS>
__global__ void __launch_bounds__(4 * AT_ROWS, 2) attention_tile_kernel(
    const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache, float* __restrict__ out,
    const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens, const int* __restrict__ seq_lens,
    int first_req, int H, int K, int d, int page_size, int page_shift, float scale) {
    constexpr int AT_WARPS = AT_ROWS / 8, OWN = AT_ROWS / AT_WARPS;
    PDL_ENTER();
    q = pdl_fresh(q); k_cache = pdl_fresh(k_cache); v_cache = pdl_fresh(v_cache);
    extern __shared__ __align__(16) float at_smem[];
    float* sQ = at_smem;                                   // [rows][d]
    float* sP = sQ + AT_ROWS * AT_LD;                      // [rows][128]: scores, then weights
    float* sKV = sP + AT_ROWS * AT_LD;                     // two half chunks of keys or values in turn
    float* sCorr = sKV + 2 * AT_HALF * AT_LD;              // [rows]
    const int G = H / K, per_tile = AT_ROWS / G;
    const int r = first_req + blockIdx.y, kh = blockIdx.x % K;
    const int tok0 = cu_tokens[r], n = cu_tokens[r + 1] - tok0;
    const int q0 = (gridDim.x - 1 - blockIdx.x) / K * per_tile;               // (the longest walks first, of all heads)
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
        // a warp a row; where its rows lie is looked up by as many lanes side by side (pages of a power of two: page_shift, else -1; a key behind the last one
        // repeats it: nobody adds what comes of it)
        constexpr int MINE = AT_HALF / AT_WARPS;
        const int key = min(key0 + warp + AT_WARPS * (lane % MINE), last), page = page_shift >= 0 ? key >> page_shift : key / page_size;
        const long long at = (((long long)table[page] * K + kh) * page_size + (key - page * page_size)) * d;
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const long long from = __shfl_sync(0xffffffffu, at, i);
            if (lane < d4) cp_async16(dst + (warp + AT_WARPS * i) * AT_LD + 4 * lane, src + from + 4 * lane);
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
    // scores: rows ty + AT_ROWS / 4 i x keys tx + 16 j; values: rows 4 ty + i x columns 4 tx.. and 64 + 4 tx..; softmax: rows 8 warp .., the warp's of the values
    const int tx = tid & 15, ty = tid >> 4;
    constexpr int RT = AT_ROWS / 4;
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
            // (the next four columns on their way while these are multiplied)
            float4 a[2][4], k[2][4];
            auto take = [&](int c, int to) {
#pragma unroll
                for (int i = 0; i < 4; ++i) a[to][i] = *reinterpret_cast<const float4*>(sQ + (ty + RT * i) * AT_LD + 4 * c);
#pragma unroll
                for (int j = 0; j < 4; ++j) k[to][j] = *reinterpret_cast<const float4*>(kv + (tx + 16 * j) * AT_LD + 4 * c);
            };
            auto add = [&](int of) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[of][i].x, k[of][j].x, s[i][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[of][i].y, k[of][j].y, s[i][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[of][i].z, k[of][j].z, s[i][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[of][i].w, k[of][j].w, s[i][j]);
            };
            take(0, 0);
            int c = 0;
#pragma unroll 1
            for (; c + 2 <= d4; c += 2) {
                take(c + 1, 1);
                add(0);
                take(c + 2 < d4 ? c + 2 : c, 0);
                add(1);
            }
            if (c < d4) add(0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = ty + RT * i, pos = pos0 + row / G;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = off + tx + 16 * j;
                    sP[row * AT_LD + key] = base + key <= pos ? s[i][j] * scale : -INFINITY;
                }
            }
            if (!(stage & 1)) continue;
            __syncthreads();                               // the chunk's scores are all there
#pragma unroll
            for (int half = 0; half < OWN; half += 4) {    // four rows side by side, a lane a key
                const int row0 = OWN * warp + half;
                float* p = sP + row0 * AT_LD + lane;
                float w[4][4], corr[4], top[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[i][e] = p[i * AT_LD + 32 * e];
                    top[i] = fmaxf(fmaxf(w[i][0], w[i][1]), fmaxf(w[i][2], w[i][3]));
                }
                {
                    // four rows' maxima at once: half of the lanes go on with half of the rows
                    const bool up = (lane & 16) != 0, on = (lane & 8) != 0;
                    const float u0 = fmaxf(up ? top[2] : top[0], __shfl_xor_sync(0xffffffffu, up ? top[0] : top[2], 16));
                    const float u1 = fmaxf(up ? top[3] : top[1], __shfl_xor_sync(0xffffffffu, up ? top[1] : top[3], 16));
                    float u = fmaxf(on ? u1 : u0, __shfl_xor_sync(0xffffffffu, on ? u0 : u1, 8));
                    u = fmaxf(u, __shfl_xor_sync(0xffffffffu, u, 4));
                    u = fmaxf(u, __shfl_xor_sync(0xffffffffu, u, 2));
                    u = fmaxf(u, __shfl_xor_sync(0xffffffffu, u, 1));
#pragma unroll
                    for (int i = 0; i < 4; ++i) top[i] = __shfl_sync(0xffffffffu, u, 8 * i);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float m_new = fmaxf(m[half + i], top[i]);
                    const int pos = pos0 + (row0 + i) / G;
                    corr[i] = expf(m[half + i] - m_new);
                    m[half + i] = m_new;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        w[i][e] = base + lane + 32 * e <= pos ? expf(w[i][e] - m_new) : 0.0f;
                        p[i * AT_LD + 32 * e] = w[i][e];
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    // the four warps' butterflies of block_sum at once (half of the lanes go on with half of them), then their sums in its order
                    const bool up = (lane & 16) != 0, on = (lane & 8) != 0;
                    const float u0 = (up ? w[i][2] : w[i][0]) + __shfl_xor_sync(0xffffffffu, up ? w[i][0] : w[i][2], 16);
                    const float u1 = (up ? w[i][3] : w[i][1]) + __shfl_xor_sync(0xffffffffu, up ? w[i][1] : w[i][3], 16);
                    float sum = (on ? u1 : u0) + __shfl_xor_sync(0xffffffffu, on ? u0 : u1, 8);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 16);              // 0 and 2; 1 and 3
                    sum += __shfl_xor_sync(0xffffffffu, sum, 8);
                    l[half + i] = fmaf(l[half + i], corr[i], sum);
                    if (lane == 0) sCorr[row0 + i] = corr[i];
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float corr = sCorr[4 * ty + i];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] *= corr;
            }
            continue;                                      // (the barrier at the top of the next stage publishes the weights)
        }
        const float* p = sP + 4 * ty * AT_LD + off;
        const int first = base + off;
        // four keys at a time; `all`: every row of the tile sees them
        auto add = [&](int j, bool all, const float4* v) {
            float w[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(w[i]) = *reinterpret_cast<const float4*>(p + i * AT_LD + j);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float x[8] = {v[2 * e].x, v[2 * e].y, v[2 * e].z, v[2 * e].w, v[2 * e + 1].x, v[2 * e + 1].y, v[2 * e + 1].z, v[2 * e + 1].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!all && first + j + e > row_pos[i]) continue;
#pragma unroll
                    for (int c = 0; c < 8; ++c) acc[i][c] = fmaf(w[i][e], x[c], acc[i][c]);
                }
            }
        };
        auto take = [&](int j, float4* v) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* row = kv + (j + e) * AT_LD + 4 * tx;
                v[2 * e] = *reinterpret_cast<const float4*>(row);
                v[2 * e + 1] = *reinterpret_cast<const float4*>(row + 64);
            }
        };
        const int whole = min(AT_HALF, max(0, pos0 - first + 1)) & ~3, most = min(AT_HALF, last - first + 1);
        int j = 0;
        float4 v0[8], v1[8];                               // (the next four keys' values on their way while these are added)
        take(0, v0);
#pragma unroll 1
        for (; j + 8 <= whole; j += 8) {
            take(j + 4, v1);
            add(j, true, v0);
            take(min(j + 8, AT_HALF - 4), v0);
            add(j + 4, true, v1);
        }
#pragma unroll 1
        for (; j < most; j += 4) {
            add(j, j < whole, v0);
            take(min(j + 4, AT_HALF - 4), v0);
        }
    }
    __syncwarp();                                          // (sCorr takes the sums now)
#pragma unroll
    for (int i = 0; i < OWN; ++i)
        if (lane == 0) sCorr[OWN * warp + i] = l[i];
    __syncwarp();
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
                             int page_size, float scale, int sms, cudaStream_t s) {
    if (count <= 0 || max_query_len <= 0) return 0;
    if (d <= 0 || d > 128 || d % 4 != 0 || K <= 0 || H % K != 0 || H / K > 32 || page_size <= 0) return MB_ERR_BAD_SIZE;
    if ((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) != 0) return MB_ERR_BAD_SIZE;
    int page_shift = -1;
    for (int i = 0; i < 31; ++i)
        if ((1 << i) == page_size) page_shift = i;
    // 32 rows a block where that makes two blocks an SM (what a block fetches is then shared by twice the rows); a row's bits do not depend on it
    const int G = H / K, tiles = (max_query_len + 32 / G - 1) / (32 / G);
    const bool wide = G > 16 || (long long)tiles * K * count >= 2 * sms;
    const int per_tile = (wide ? 32 : 16) / G;
    const dim3 grid((max_query_len + per_tile - 1) / per_tile * K, count);
    const auto kernel = wide ? attention_tile_kernel<32> : attention_tile_kernel<16>;
    const int rows = wide ? 32 : 16;
    static LaunchSmem smem[2];
    const int rc = smem[wide].allow(kernel, AT_SMEM(rows));
    if (rc) return rc;
    return launch_kernel(kernel, grid, 4 * rows, AT_SMEM(rows), s, 0, (const float*)q, (const float*)k_cache, (const float*)v_cache, (float*)out, block_table,
                         max_pages, cu_tokens, seq_lens, first_req, H, K, d, page_size, page_shift, scale);
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
