// Products of a routed feed-forward on the 5th-generation tensor cores: for every expert e, out[i, n] = sum_k x[i, k] w[e][n, k] over
// the rows i of that expert (rows sorted by expert, offsets[e] .. offsets[e + 1] - 1), all experts in one persistent launch that reads
// the experts' shares on the device.  A further group of rows with a matrix of its own (a shared expert: every token) may ride in the
// same launch.
//
// As in the dense product (gemm_tc.cu) 128 weight rows are the M operand and up to BNM rows of x the N operand of tcgen05.mma; TMA brings
// 64 k of both into a ring of STAGES buffers, one thread issues the MMAs into one of two accumulators in tensor memory, and eight warps
// empty the other one meanwhile.  What differs:
//   * tiles are found on the device: a warp lays the groups' tile counts end to end, every CTA takes every ctas-th tile, weight tiles of an
//     expert next to one another over its row tiles, so that a weight tile is fetched from HBM once;
//   * an expert's rows are cut into equal tiles of a width that is a multiple of 16 (540 rows: three tiles of 192, not two of 256 and
//     one of 28): the MMA's N is set per tile, and x arrives in boxes of BOX rows, as many as the width needs.
//   * PAIR (long products): two CTAs of a cluster on 256 weight rows, as gemm_tc.cu's pairs, widths then in steps of 32.
// Bound by the tensor pipe with hundreds of rows an expert, by the weights' bytes with few: BNM then is small and the ring deep (ten 20 KB
// stages a SM).
#define MB_LIB "moe_tc"
#define MB_LIB_ID 24
#include "tc_epilogue.cuh"
#include "launch.cuh"

#define MT_MAX_GROUPS 512

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One kind of rows: the experts' (with offsets) or the further group's.
struct MoeSide {
    void* out;           // [rows][N] (mode 0, 1, 4) or [rows][N / 2] (gated modes)
    int N, K;            // weight rows per expert, row length (a multiple of 64)
    long long part;      // numbers between the results of two parts of K (mode 1 with parts)
};

template <int BNM, int BOX, int STAGES, bool PAIR>
struct MoeRing {
    static constexpr int A_BYTES = TC_BM * TC_BK * 2, BOX_BYTES = BOX * TC_BK * 2, STAGE = A_BYTES + BNM / (PAIR ? 2 : 1) * TC_BK * 2;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
    static_assert(BOX % 8 == 0 && BNM / (PAIR ? 2 : 1) % BOX == 0, "boxes of whole swizzle groups");
};

// A walk over the tiles of one CTA (or pair), the same in every role.  ctas: CTAs a tile.  Group 0 is the further group, group e + 1 expert e.
struct MoeWalk {
    const int* first;    // [groups + 1]: tiles before each group
    const int* start;    // [groups + 1]: first row of each expert's group (entry 0 unused)
    int groups, at, step, extra_rows, widest, parts, ctas;
    int g;
    __device__ bool next(int& row0, int& rows_end, int& width, int& n0, int& part) {
        if (at >= first[groups]) return false;
        while (at >= first[g + 1]) ++g;
        const int count = g == 0 ? extra_rows : start[g + 1] - start[g];
        const int begin = g == 0 ? 0 : start[g];
        const int across = (count + widest - 1) / widest;
        width = ((count + across - 1) / across + 16 * ctas - 1) & ~(16 * ctas - 1);
        part = (at - first[g]) % parts;
        const int in = (at - first[g]) / parts;
        n0 = in / across * ctas * TC_BM;
        row0 = begin + in % across * width;
        rows_end = begin + count;
        at += step;
        return true;
    }
    // (across - 1 tiles of the widest kind are fewer rows than there are, so the last tile is never empty after rounding up)
};

template <int BNM, int BOX, int STAGES, bool PAIR>
__global__ void __launch_bounds__(320) moe_grouped_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                             const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x2,
                                                             const int* __restrict__ offsets, int E, const MoeSide ex, const MoeSide sh, int extra_rows,
                                                             int share, int widest, int parts, int mode, int* __restrict__ error_flag) {
    typedef MoeRing<BNM, BOX, STAGES, PAIR> R;
    constexpr int CTAS = PAIR ? 2 : 1;
    const int rank = PAIR ? (int)cluster_rank() : 0;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_first[MT_MAX_GROUPS + 2], s_start[MT_MAX_GROUPS + 2];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + STAGES * R::STAGE);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;       // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr uint32_t TMEM_COLS = 2 * BNM <= 32 ? 32 : 2 * BNM <= 64 ? 64 : 2 * BNM <= 128 ? 128 : 2 * BNM <= 256 ? 256 : 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8 * CTAS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        tmem_alloc<PAIR>(tmem_slot, TMEM_COLS);
    }
    PDL_ENTER_EARLY();
    offsets = pdl_fresh(offsets);
    if (warp == 1) {
        // the groups' tiles end to end
        const int tiles_n = parts * ((ex.N + CTAS * TC_BM - 1) / (CTAS * TC_BM));
        int run = extra_rows > 0 ? parts * ((sh.N + CTAS * TC_BM - 1) / (CTAS * TC_BM)) * ((extra_rows + widest - 1) / widest) : 0;
        if (lane == 0) { s_first[0] = 0; s_start[0] = 0; }
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            const int begin = e >= E ? 0 : offsets != nullptr ? offsets[e] : e * share, n = e >= E ? 0 : offsets != nullptr ? offsets[e + 1] - begin : share;
            const int tiles = tiles_n * ((n + widest - 1) / widest);
            int sum = tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += v;
            }
            if (e < E) {
                s_first[e + 1] = run + sum - tiles;
                s_start[e + 1] = begin;
                if (e == E - 1) { s_first[E + 1] = run + sum; s_start[E + 1] = begin + n; }
            }
            run += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();                  // (the other CTA's barriers are set up before anything is counted there)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    MoeWalk walk = {s_first, s_start, E + 1, (int)blockIdx.x / CTAS, (int)gridDim.x / CTAS, extra_rows, widest, parts, CTAS, 0};
    int row0, rows_end, width, n0, part;
    // the k-blocks of a part
    auto begin_of = [&](int nkb) { return part * ((nkb + parts - 1) / parts); };
    auto end_of = [&](int nkb) { return min(nkb, (part + 1) * ((nkb + parts - 1) / parts)); };

    const int role = warp_same(warp);
    if (warp == 0 && lane == 0) {
        int it = 0;                                                   // k-blocks issued so far, over all tiles
        bool ok = true;
        while (ok && walk.next(row0, rows_end, width, n0, part)) {
            const bool shared = walk.g == 0;
            const int nkb = (shared ? sh.K : ex.K) / TC_BK;
            const CUtensorMap* mw = shared ? &map_w2 : &map_w;
            const CUtensorMap* mx = shared ? &map_x2 : &map_x;
            const int wrow = (shared ? n0 : (walk.g - 1) * ex.N + n0) + rank * TC_BM;         // (a pair's second 128 rows may lie past the last: nobody stores what comes of them)
            const int boxes = (width / CTAS + BOX - 1) / BOX, xrow = row0 + rank * (width / CTAS);
            for (int kb = begin_of(nkb); kb < end_of(nkb); ++kb, ++it) {
                const int s = it % STAGES;
                if (!mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1)) { atomicExch(error_flag, 21); ok = false; break; }
                uint8_t* a = smem + s * R::STAGE;
                if (PAIR) {
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * (R::A_BYTES + boxes * R::BOX_BYTES));
                    const uint32_t bar = leader_addr(&full[s]);
                    tma_load_2d_pair(a, mw, kb * TC_BK, wrow, bar);
                    for (int b = 0; b < boxes; ++b) tma_load_2d_pair(a + R::A_BYTES + b * R::BOX_BYTES, mx, kb * TC_BK, xrow + b * BOX, bar);
                } else {
                    mbar_expect_tx(&full[s], R::A_BYTES + boxes * R::BOX_BYTES);
                    tma_load_2d(a, mw, kb * TC_BK, wrow, &full[s]);
                    for (int b = 0; b < boxes; ++b) tma_load_2d(a + R::A_BYTES + b * R::BOX_BYTES, mx, kb * TC_BK, xrow + b * BOX, &full[s]);
                }
            }
        }
    } else if (role == 1 && rank == 0) {
        const uint32_t elected = elect_one(), tmem_mma = warp_same(tmem_base);
        int it = 0, local = 0;
        bool ok = true;
        for (; ok && warp_same((int)walk.next(row0, rows_end, width, n0, part)); ++local) {
            const int buf = local & 1;
            part = warp_same(part);
            const int nkb = warp_same(walk.g == 0 ? sh.K : ex.K) / TC_BK;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(warp_same(width) >> 3) << 17) | ((uint32_t)(CTAS * TC_BM >> 4) << 24);
            if (!mbar_wait_warp(&acc_empty[buf], ((local >> 1) & 1) ^ 1)) { atomicExch(error_flag, 22); ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_mma + (uint32_t)(buf * BNM);
            const int kb0 = begin_of(nkb), kb1 = end_of(nkb);
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                const int s = it % STAGES;
                if (!mbar_wait_warp(&full[s], (it / STAGES) & 1)) { atomicExch(error_flag, 23); ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = smem_u32(smem + s * R::STAGE);
                const uint64_t adesc = umma_desc(a), bdesc = umma_desc(a + R::A_BYTES);
#pragma unroll
                for (int kk = 0; kk < TC_BK / 16; ++kk) {
                    if (PAIR) umma_bf16_pair(tmem_d, adesc + 2 * kk, bdesc + 2 * kk, idesc, (kb > kb0 || kk > 0) ? 1u : 0u, elected);
                    else umma_bf16(tmem_d, adesc + 2 * kk, bdesc + 2 * kk, idesc, (kb > kb0 || kk > 0) ? 1u : 0u, elected);
                }
                if (PAIR) umma_commit_pair(&empty[s], elected);
                else umma_commit(&empty[s], elected);
            }
            if (PAIR) umma_commit_pair(&acc_full[buf], elected);
            else umma_commit(&acc_full[buf], elected);
        }
    } else if (warp >= 2) {
        const int quarter = warp & 3;                                 // the 32 TMEM lanes this warp may read
        const int col_half = (warp - 2) >> 2;                         // two warps share a quarter: each takes half the columns
        int local = 0;
        bool ok = true;
        const TcGlu glu = {1.0f, 0, 0, nullptr};
        for (; walk.next(row0, rows_end, width, n0, part); ++local) {
            const MoeSide& side = walk.g == 0 ? sh : ex;
            n0 += rank * TC_BM;
            const int buf = local & 1;
            const int half = (width / 16 + 1) / 2 * 16;
            const int c_begin = col_half * half, c_end = col_half == 0 ? half : width;
            const int n = n0 + quarter * 32 + lane;
            // a warp whose wait gave up keeps walking the tiles but touches nothing
            if (ok && !mbar_wait(&acc_full[buf], (local >> 1) & 1)) { if (lane == 0) atomicExch(error_flag, 24); ok = false; }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) continue;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c0 = c_begin; c0 < c_end && row0 + c0 < rows_end; c0 += 16) {
                float v[16];
                tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BNM + c0), v);
                if (tc_gated(mode)) {
                    if (n0 + quarter * 32 < side.N) store_chunk_glu(side.out, mode, row0 + c0, n0 + quarter * 32, lane, rows_end, side.N, v, glu);
                } else if (n < side.N) {
                    store_chunk(parts > 1 ? (void*)((float*)side.out + part * side.part) : side.out, mode, row0 + c0, n, rows_end, side.N, v);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_leader(&acc_empty[buf]);
                else mbar_arrive(&acc_empty[buf]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();                  // nothing of the other CTA's is counted here any more, and its MMAs have left this one's memory
    if (warp == 0) {
        __syncwarp();
        tmem_free<PAIR>(tmem_base, TMEM_COLS);
    }
}

// ---- host side ----
template <int BNM, int BOX, int STAGES, bool PAIR = false>
static int launch_grouped(const void* x, const void* w, const int* offsets, int E, int pairs, const MoeSide& ex, const void* x2, const void* w2, int rows2,
                          const MoeSide& sh, int widest, int parts, int mode, int ctas, int* error_flag, cudaStream_t s) {
    typedef MoeRing<BNM, BOX, STAGES, PAIR> R;
    constexpr int CTAS = PAIR ? 2 : 1;
    static_assert(R::SMEM <= 220 * 1024, "the ring does not fit shared memory");
    CUtensorMap mw, mx, mw2, mx2;
    int rc = make_map(&mw, w, E * ex.N, ex.K, TC_BM);
    if (rc == 0) rc = make_map(&mx, x, pairs, ex.K, BOX);
    if (rc) return rc;
    mw2 = mw; mx2 = mx;
    if (rows2 > 0) {
        rc = make_map(&mw2, w2, sh.N, sh.K, TC_BM);
        if (rc == 0) rc = make_map(&mx2, x2, rows2, sh.K, BOX);
        if (rc) return rc;
    }
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(moe_grouped_tc_kernel<BNM, BOX, STAGES, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    // no more CTAs than there can be tiles (the shares are known on the device only)
    const long long across = (long long)(pairs / widest + (E < pairs ? E : pairs)), most = parts * (across * ((ex.N + TC_BM - 1) / TC_BM) +
        (rows2 > 0 ? (long long)((rows2 + widest - 1) / widest) * ((sh.N + TC_BM - 1) / TC_BM) : 0));
    return launch_kernel(moe_grouped_tc_kernel<BNM, BOX, STAGES, PAIR>, dim3((unsigned)(CTAS * (most < ctas / CTAS ? most : ctas / CTAS))), dim3(320), R::SMEM, s, PAIR ? -2 : 0, mw, mx, mw2, mx2,
                         offsets, E, ex, sh, rows2, pairs / E, widest, parts, mode, error_flag);
}

// x bf16 [pairs][K] (sorted by expert), w bf16 [E][N][K], offsets int32 [E + 1] on the device (null: every expert has pairs / E rows, E a divisor); out: mode 0
// bf16 [pairs][N], 1 float32 [pairs][N], 4 bf16 relu(.)^2 [pairs][N], gated modes bf16 [pairs][N / 2] (gate and up rows in alternating blocks of 16).  The
// further group: x2 bf16 [rows2][K2], w2 bf16 [N2][K2], out2 likewise (rows2 0: there is none).  K and K2 multiples of 64, pointers 16-byte aligned;
// widest: the widest tile, a multiple of 16 up to 256 rows (negative: -widest, a multiple of 32 above 128, by CTAs in pairs; one part).  parts: K in so many parts (mode 1 only), every part's sums in a result of its own, pairs * N (and rows2 *
// N2) numbers apart: with few rows there are few tiles, and whole tiles would leave SMs idle; whoever reads the results adds them.  No part may be empty.
MB_API int mb_moe_grouped_tc(const void* x, const void* w, const int* offsets, int E, int pairs, int N, int K, void* out, const void* x2, const void* w2,
                             int rows2, int N2, int K2, void* out2, int mode, int widest, int parts, int ctas, int* error_flag, cudaStream_t s) {
    if (pairs <= 0) return rows2 > 0 ? MB_ERR_BAD_SIZE : 0;
    if (E <= 0 || E > MT_MAX_GROUPS || N <= 0 || K <= 0 || K % TC_BK != 0 || ctas <= 0 || (long long)E * N > 0x7fffffffLL) return MB_ERR_BAD_SIZE;
    if (rows2 < 0 || (rows2 > 0 && (N2 <= 0 || K2 <= 0 || K2 % TC_BK != 0 || x2 == nullptr || w2 == nullptr || out2 == nullptr))) return MB_ERR_BAD_SIZE;
    if ((((uintptr_t)x | (uintptr_t)w | (uintptr_t)x2 | (uintptr_t)w2) & 15) != 0) return MB_ERR_BAD_SIZE;
    if (mode == TC_OUT_F32_ACC || mode < 0 || mode >= TC_OUT_MODES || (tc_gated(mode) && (N % 32 != 0 || (rows2 > 0 && N2 % 32 != 0)))) return MB_ERR_BAD_DTYPE;
    const bool pair = widest < 0;
    if (pair) widest = -widest;
    if (pair && (widest <= 128 || widest % 32 != 0 || parts != 1 || ctas < 2)) return MB_ERR_BAD_SIZE;
    if (widest < 16 || widest > 256 || widest % 16 != 0 || (offsets == nullptr && pairs % E != 0)) return MB_ERR_BAD_SIZE;
    const auto part_empty = [parts](int k) { const int nkb = k / TC_BK; return (parts - 1) * ((nkb + parts - 1) / parts) >= nkb; };
    if (parts < 1 || (parts > 1 && (mode != TC_OUT_F32 || part_empty(K) || (rows2 > 0 && part_empty(K2))))) return MB_ERR_BAD_SIZE;
    const MoeSide ex = {out, N, K, (long long)pairs * N}, sh = {out2, rows2 > 0 ? N2 : 0, rows2 > 0 ? K2 : 0, (long long)rows2 * N2};
    if (pair) return launch_grouped<256, 64, 6, true>(x, w, offsets, E, pairs, ex, x2, w2, rows2, sh, widest, parts, mode, ctas, error_flag, s);
    if (widest <= 32) return launch_grouped<32, 16, 10>(x, w, offsets, E, pairs, ex, x2, w2, rows2, sh, widest, parts, mode, ctas, error_flag, s);
    if (widest <= 64) return launch_grouped<64, 16, 8>(x, w, offsets, E, pairs, ex, x2, w2, rows2, sh, widest, parts, mode, ctas, error_flag, s);
    if (widest <= 128) return launch_grouped<128, 64, 6>(x, w, offsets, E, pairs, ex, x2, w2, rows2, sh, widest, parts, mode, ctas, error_flag, s);
    return launch_grouped<256, 64, 4>(x, w, offsets, E, pairs, ex, x2, w2, rows2, sh, widest, parts, mode, ctas, error_flag, s);
}
