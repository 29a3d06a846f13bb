// bf16 GEMM with fp32 accumulation and an optional bias epilogue for sm_100a: the projections either side of
// attention (qkv = x Wqkv + b before it, y W_out + b after it), forward and backward.
//
// Replaces, for those two layers, the reference's Linear::forward = matmul(x, W) + b
// (src/inferno/modules/linear.cpp:99-106 -> cublas_mm_row_major, src/inferno/cuda/cudamatmul.cu:1058-1112, plus the
// broadcast add kernel, src/inferno/cuda/cudaadd.cu:20-142) and the two GEMMs of its backward, MMBackward
// (src/inferno/gradfn/mmbackward.cpp:36-98): dX = dY W^T and dW = X^T dY.  The reference materialises every transpose with
// a copy kernel; here a transposed operand is only a different shared-memory descriptor (MN-major instead of K-major).
//
//   C[M, N] = A[M, K] * B[K, N] (+ bias[N])
//   a_mn = 0: A stored [M rows, K contiguous]        a_mn = 1: A stored [K rows, M contiguous]  (A = X^T)
//   b_mn = 1: B stored [K rows, N contiguous]        b_mn = 0: B stored [N rows, K contiguous] (B = W^T)
//
// A pair of CTAs (cta_group::2) owns a 256 x 256 output tile, each CTA 128 of its rows.  Per k-step of 16 a CTA then reads
// 4 KB of A and 4 KB of B (its half of B's rows) for 128 x 256 products: with the copies that fill the ring, 128 bytes per
// clock of shared memory, exactly what the SM can move while the tensor pipe needs 128 clocks.  The one-CTA form of the same
// tile (128 x 256) moves 192 bytes per clock and was bound by it: 16384 x 768 x 2304 in 46.5 us against 36 us at the rate of
// a library GEMM.
//
// One warp of each CTA streams A / B k-slices of 64 through a TMA ring, one lane of the even CTA's MMA warp issues 256x256x16
// MMAs into one of two 256-column TMEM accumulators, and eight warps drain the other accumulator (TMEM -> registers -> +bias ->
// TMA store), so the epilogue of a tile overlaps the main loop of the next.
//
// One launch runs up to two products ("tasks"), so that dX and dW of a projection share a grid:
//   task 0 is cut into whole tiles, dealt out round-robin;
//   task 1 is either cut the same way (its tiles follow task 0's), or, when it has too few tiles for the chip and a long K
//   (a weight gradient: K = tokens), into contiguous runs of k-slices, one per CTA pair, sized so that every pair ends up
//   with the same number of k-slices over both tasks.  The partial tiles meet by TMA reduction: in an fp32 workspace, zeroed
//   before and rounded once to bf16 afterwards by linear_finish_kernel, or, for callers without a workspace, in the zeroed
//   bf16 output itself (one rounding per partial, at most eight).
#pragma once

#include "sm100_ptx.cuh"

namespace ib200 {

struct GemmTraits {
    static constexpr int BM = 256, BN = 256, BK = 64;            // tile of a CTA pair
    static constexpr int CM = BM / 2, CN = BN / 2;               // rows of A and of B that one CTA loads
    static constexpr int STAGES = 6;
    static constexpr int A_BYTES = CM * BK * 2;                  // 16 KB
    static constexpr int B_BYTES = CN * BK * 2;                  // 16 KB
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int OFF_OUT = STAGES * STAGE_BYTES;
    static constexpr int STAGING_BYTES = 32 * 128;               // epilogue staging of one warp
    static constexpr int OFF_BAR = OFF_OUT + 8 * STAGING_BYTES;
    static constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
    static constexpr int EPI_WARPS = 8;                          // two per 32 rows of the tile, each with half of its columns
    static constexpr int THREADS = EPI_WARPS * 32 + 64;          // and the TMA warp and the MMA warp
    static constexpr uint32_t TM_COLS = 512;
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

struct GemmTask {
    int M, N;
    int tiles_m, tiles;    // tiles = 0: no such task
    int k_slices;          // of 64
    int a_mn, b_mn;
};

enum : int { kPartWhole = 0, kPartReduceBf16 = 1, kPartReduceF32 = 2 };

struct GemmParams {
    GemmTask t[2];
    int split;             // task 1: kPartWhole, or how partial tiles are added up
    // split runs: pair c starts at k-slice total1 * (min(c, heavy) * w_heavy + max(0, c - heavy) * w_light) / w_total of task 1
    int heavy;
    long long w_heavy, w_light, w_total;
    const void* bias;      // [N] of task 0 (task 1 when it is the only one), or null
    int bias_bf16;
    int* status;
};

__host__ __device__ __forceinline__ int gemm_split_start(const GemmParams& p, int pair) {
    const long long total = static_cast<long long>(p.t[1].tiles) * p.t[1].k_slices;
    const long long w = (pair < p.heavy ? pair : p.heavy) * p.w_heavy + (pair > p.heavy ? pair - p.heavy : 0) * p.w_light;
    return static_cast<int>(total * w / p.w_total);
}

// The parts of one CTA pair, in order: its run of split task-1 slices first, then its whole tiles.
struct GemmPart {
    int task, m0, n0, ks0, ks1;
    bool partial;          // added to other parts of its tile
};
constexpr int kBandRows = 8;
struct GemmWalk {
    const GemmParams& p;
    int pair, pairs;
    int f, hi;             // split run
    int tile;              // next whole tile
    __device__ __forceinline__ GemmWalk(const GemmParams& prm, int pair_, int pairs_) : p(prm), pair(pair_), pairs(pairs_), f(0), hi(0), tile(pair_) {
        if (p.split != kPartWhole) {
            f = gemm_split_start(p, pair);
            hi = gemm_split_start(p, pair + 1);
        }
    }
    __device__ __forceinline__ bool next(GemmPart& q) {
        int t;
        if (f < hi) {
            const GemmTask& k = p.t[1];
            t = f / k.k_slices;
            q.task = 1;
            q.ks0 = f - t * k.k_slices;
            q.ks1 = min(k.k_slices, q.ks0 + (hi - f));
            q.partial = true;
            f += q.ks1 - q.ks0;
        } else {
            const int whole = p.t[0].tiles + (p.split == kPartWhole ? p.t[1].tiles : 0);
            if (tile >= whole) return false;
            q.task = tile < p.t[0].tiles ? 0 : 1;
            t = q.task ? tile - p.t[0].tiles : tile;
            q.ks0 = 0;
            q.ks1 = p.t[q.task].k_slices;
            q.partial = false;
            tile += pairs;
        }
        // tiles are numbered in bands of eight tile rows, so that the pairs at work share few rows of A and few columns of B in L2
        // (16384 x 768 x 2304 and 8192^3: 3 % and 5 % over one column of tiles after the other)
        const int tm = p.t[q.task].tiles_m, tn = p.t[q.task].tiles / tm;
        const int band = t / (kBandRows * tn), r = t - band * (kBandRows * tn), rows = min(kBandRows, tm - band * kBandRows);
        q.m0 = (band * kBandRows + r % rows) * GemmTraits::BM;
        q.n0 = (r / rows) * GemmTraits::BN;
        return true;
    }
};

// The tensor maps of a launch: operands and outputs of the two tasks, and what a split task 1 is added into (its bf16 output,
// or the fp32 accumulation workspace).
struct GemmMaps {
    CUtensorMap a[2], b[2], c[2], sum;
};

__device__ __forceinline__ float2 load_bias2(const GemmParams& p, int col) {      // col is even
    if (!p.bias_bf16) return *reinterpret_cast<const float2*>(static_cast<const float*>(p.bias) + col);
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(static_cast<const __nv_bfloat16*>(p.bias) + col));
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GemmTraits::THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams prm) {
    using TR = GemmTraits;
    constexpr int BN = TR::BN, BK = TR::BK, NS = TR::STAGES, kTmaWarp = TR::EPI_WARPS, kMmaWarp = TR::EPI_WARPS + 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sOut = smem + TR::OFF_OUT;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TR::OFF_BAR);
    uint64_t* full = bars;                  // [NS]  TMA of both CTAs -> MMA (used in the even CTA)
    uint64_t* empty = full + NS;            // [NS]  MMA -> TMA (in both)
    uint64_t* acc_full = empty + NS;        // [2]   MMA -> epilogue (in both)
    uint64_t* acc_empty = acc_full + 2;     // [2]   the epilogues of both CTAs -> MMA (used in the even CTA)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    ResidentAbortCtx ab{abort_flag, prm.status};

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < NS; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * TR::EPI_WARPS); }
        fence_mbar_init();
    }
    if (warp == kMmaWarp) { tmem_alloc_pair(tmem_slot, TR::TM_COLS); tmem_relinquish_pair(); }
    if (warp == kTmaWarp && lane == 0) {
        for (int t = 0; t < 2; ++t)
            if (prm.t[t].tiles) { tma_prefetch_desc(&maps.a[t]); tma_prefetch_desc(&maps.b[t]); tma_prefetch_desc(&maps.c[t]); }
    }
    tc_fence_before_sync();
    cluster_sync_all();                     // the other CTA's barriers exist before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();

    GemmWalk walk(prm, pair, pairs);
    GemmPart q;
    if (warp == kTmaWarp) {
        // ------------------------------ TMA producer (each CTA loads its halves) ------------------------------
        // Like the MMA warp, this one stays converged and predicates the copies on an elected lane: a lone lane in a divergent
        // branch took 714 cycles to issue a k-slice, longer than the 512 the tensor pipe needs for it.
        const bool leader = elect_one_lane();
        uint32_t s = 0, phase = 0, used = 0;     // ring position
        const uint32_t full0 = mapa_u32(smem_u32(full), 0);
        while (walk.next(q)) {
            const GemmTask& k = prm.t[q.task];
            const CUtensorMap *ma = &maps.a[q.task], *mb = &maps.b[q.task];
            const int m0 = q.m0 + static_cast<int>(rank) * TR::CM, n0 = q.n0 + static_cast<int>(rank) * TR::CN;
            const bool a_mn = k.a_mn, b_mn = k.b_mn;
            for (int ks = q.ks0; ks < q.ks1; ++ks) {
                mbar_wait(&empty[s], phase ^ 1, ab, 10);
                const uint32_t bar = full0 + s * 8;
                uint8_t* sa = smem + s * TR::STAGE_BYTES;
                uint8_t* sb = sa + TR::A_BYTES;
                const int k0 = ks * BK;
                if (leader) {
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * TR::STAGE_BYTES);
                    if (!a_mn) {
                        tma_load_3d_pair(sa, ma, bar, k0, m0, 0);                          // [128 m-rows x 64 k]
                    } else {
                        tma_load_3d_pair(sa, ma, bar, m0, k0, 0);                          // two panels [64 k-rows x 64 m]
                        tma_load_3d_pair(sa + BK * 128, ma, bar, m0 + 64, k0, 0);
                    }
                    if (!b_mn) {
                        tma_load_3d_pair(sb, mb, bar, k0, n0, 0);                          // [128 n-rows x 64 k]
                    } else {
                        tma_load_3d_pair(sb, mb, bar, n0, k0, 0);                          // two panels [64 k-rows x 64 n]
                        tma_load_3d_pair(sb + BK * 128, mb, bar, n0 + 64, k0, 0);
                    }
                }
                if (++s == NS) { s = 0; phase ^= 1; }
                if (used < NS) ++used;
            }
        }
        if (leader) pdl_trigger();
        // the last MMAs' arrivals on this CTA's empty barriers must have landed before the CTA leaves
        for (; used > 0; --used) {
            mbar_wait(&empty[s], phase ^ 1, ab, 11);
            if (++s == NS) { s = 0; phase ^= 1; }
        }
    } else if (warp == kMmaWarp) {
        // ------------------------------ MMA issuer (even CTA) ------------------------------
        // The warp stays converged; only the MMA / commit instructions are predicated on one elected lane (commits are
        // then free, where a lone lane in a divergent branch pays ~44 cycles of tensor-pipe time for each).
        if (rank == 0) {
            const bool leader = elect_one_lane();
            uint32_t s = 0, phase = 0, n = 0;
            for (; walk.next(q); ++n) {
                const GemmTask& k = prm.t[q.task];
                const uint32_t idesc = make_idesc(kFmtBF16, TR::BM, TR::BN, k.a_mn ? kMajorMN : kMajorK, k.b_mn ? kMajorMN : kMajorK);
                const uint32_t a_step = k.a_mn ? 2048u >> 4 : 32u >> 4, b_step = k.b_mn ? 2048u >> 4 : 32u >> 4;
                const uint32_t a_lo0 = sdesc_lo(smem_u32(smem), k.a_mn ? BK * 128 : 16), b_lo0 = sdesc_lo(smem_u32(smem + TR::A_BYTES), k.b_mn ? BK * 128 : 16);
                const uint32_t buf = n & 1, acc = tmem + buf * BN;
                mbar_wait_cluster(&acc_empty[buf], ((n >> 1) & 1) ^ 1, ab, 20);            // both epilogues have drained this accumulator
                tc_fence_after_sync();
                for (int ks = q.ks0; ks < q.ks1; ++ks) {
                    mbar_wait(&full[s], phase, ab, 21);
                    tc_fence_after_sync();
                    const uint32_t a_lo = a_lo0 + s * (TR::STAGE_BYTES >> 4), b_lo = b_lo0 + s * (TR::STAGE_BYTES >> 4);
#pragma unroll
                    for (int j = 0; j < BK / 16; ++j)
                        if (leader) umma_ss_f16_pair(acc, sdesc_join(a_lo + j * a_step), sdesc_join(b_lo + j * b_step), idesc, (ks != q.ks0) || j != 0);
                    if (leader) umma_commit_pair(&empty[s]);
                    if (++s == NS) { s = 0; phase ^= 1; }
                }
                if (leader) umma_commit_pair(&acc_full[buf]);
            }
        }
    } else {
        // ------------------------------ epilogue (two threads per output row of this CTA, half of the columns each) ------------------------------
        // Every warp works for itself: it stages 32 rows x 128 bytes in its own 4 KB and has the TMA unit store them (or add them
        // to the other parts of the tile), so no barrier ties the warps together.  Registers straight to global memory (a 32-byte
        // sector per thread) took 6200 cycles a tile, at three cycles per sector, and 2800 more in the release of the accumulator, which
        // had to wait for the stores; four warps that shared staging panels under named barriers took 7300.
        const int h = warp >> 2, row0 = (warp & 3) * 32;
        const uint32_t lane_base = static_cast<uint32_t>(row0) << 16;
        uint8_t* stage = sOut + warp * TR::STAGING_BYTES;
        const uint32_t free_bar[2] = {mapa_u32(smem_u32(&acc_empty[0]), 0), mapa_u32(smem_u32(&acc_empty[1]), 0)};
        uint32_t n = 0;
        auto stage_out = [&](const CUtensorMap* m, bool add, int col, int row, const uint4 (&w)[8]) {
            if (lane == 0) tma_store_wait_read_all();            // the previous copy has read the staging rows
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 8; ++c) st_shared_sw128(stage, lane, c, w[c]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (add) tma_reduce_add_3d(m, stage, col, row, 0);       // rows / columns past M / N are clipped by the copy
                else tma_store_3d(m, stage, col, row, 0);
                tma_store_commit();
            }
        };
        for (; walk.next(q); ++n) {
            const GemmTask& k = prm.t[q.task];
            const uint32_t buf = n & 1;
            const int row = q.m0 + static_cast<int>(rank) * TR::CM + row0;
            const bool with_bias = prm.bias && q.ks0 == 0;       // the part that starts the tile's K range brings the bias in
            const bool f32_out = q.partial && prm.split == kPartReduceF32;
            const CUtensorMap* mc = q.partial ? &maps.sum : &maps.c[q.task];
            // two columns of bias per lane and 64-column step, fetched under the wait and handed round by shuffles (broadcast loads in
            // the element loop queued behind the MMAs' operand reads for 2000 cycles and more)
            float2 bias0 = make_float2(0.f, 0.f), bias1 = bias0;
            if (with_bias) {
                const int col = q.n0 + h * (BN / 2) + 2 * lane;
                if (col < k.N) bias0 = load_bias2(prm, col);
                if (col + 64 < k.N) bias1 = load_bias2(prm, col + 64);
            }
            mbar_wait(&acc_full[buf], (n >> 1) & 1, ab, 30);
            tc_fence_after_sync();
#pragma unroll 1
            for (int c0 = h * (BN / 2); c0 < (h + 1) * (BN / 2); c0 += 64) {
                const int col = q.n0 + c0;
                uint32_t v[2][32];
                tmem_ld_x32(tmem + buf * BN + c0 + lane_base, v[0]);
                tmem_ld_x32(tmem + buf * BN + c0 + 32 + lane_base, v[1]);
                tmem_wait_ld();
                if (c0 + 64 == (h + 1) * (BN / 2)) {
                    // every column of the accumulator is in registers: hand it back to the MMA warp
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster_relaxed(free_bar[buf]);
                }
                if (row >= k.M || col >= k.N) continue;
                if (with_bias) {
                    const float2 bc = c0 & 64 ? bias1 : bias0;
#pragma unroll
                    for (int e = 0; e < 64; ++e)
                        v[e >> 5][e & 31] = __float_as_uint(__uint_as_float(v[e >> 5][e & 31]) + __shfl_sync(0xffffffffu, e & 1 ? bc.y : bc.x, e >> 1));
                }
                uint4 w[8];
                if (!f32_out) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint32_t* x = &v[c >> 2][(c & 3) * 8];
                        w[c] = make_uint4(pack_bf16x2(__uint_as_float(x[0]), __uint_as_float(x[1])), pack_bf16x2(__uint_as_float(x[2]), __uint_as_float(x[3])),
                                          pack_bf16x2(__uint_as_float(x[4]), __uint_as_float(x[5])), pack_bf16x2(__uint_as_float(x[6]), __uint_as_float(x[7])));
                    }
                    stage_out(mc, q.partial, col, row, w);
                } else {
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
#pragma unroll
                        for (int c = 0; c < 8; ++c) w[c] = make_uint4(v[half][4 * c], v[half][4 * c + 1], v[half][4 * c + 2], v[half][4 * c + 3]);
                        if (col + 32 * half < k.N) stage_out(mc, true, col + 32 * half, row, w);
                    }
                }
            }
        }
        if (lane == 0) tma_store_wait_read_all();    // the CTA may leave once its shared memory has been read; the writes complete on their own
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag != 0) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    cluster_sync_all();                     // neither CTA leaves while the other may still signal it or use its half of an MMA
    if (warp == kMmaWarp) tmem_dealloc_pair(tmem, TR::TM_COLS);
}

// The backward's helper ahead of the GEMMs: column sums of dY [M, N] (the bias gradient: the reference's sum_to_shape after
// the broadcast add, src/inferno/core/broadcastops.cpp) as one row of partial sums per row slab, and the zeroing of the
// fp32 accumulation workspace.  Block (x, y): 256 columns, rows y * rows_per_block ...; a warp reads 512 contiguous bytes
// of a row (16 bytes a lane) and keeps four rows in flight.  HBM-bound: one read of dY.
constexpr int kColsumCols = 256, kMaxColsumSlabs = 128;
__global__ void __launch_bounds__(256) linear_prep_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ part, int M, int N, int rows_per_block,
                                                          int atomic, float4* __restrict__ zero, long zero4) {
    pdl_wait();
    pdl_trigger();
    const long zstep = static_cast<long>(gridDim.x) * gridDim.y * blockDim.x;
    for (long i = (static_cast<long>(blockIdx.y) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < zero4; i += zstep) zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!part) return;
    __shared__ float sums[8][kColsumCols + 4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = blockIdx.x * kColsumCols + lane * 8;
    const int row1 = min(M, static_cast<int>(blockIdx.y + 1) * rows_per_block);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add = [&](const uint4& v) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            acc[2 * e] += __uint_as_float(w[e] << 16);
            acc[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
        }
    };
    if (col < N) {
        const uint4* src = reinterpret_cast<const uint4*>(x + col);
        const long pitch = N / 8;
        int row = blockIdx.y * rows_per_block + warp;
        for (; row + 24 < row1; row += 32) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = src[(row + 8 * u) * pitch];
#pragma unroll
            for (int u = 0; u < 4; ++u) add(v[u]);
        }
        for (; row < row1; row += 8) add(src[row * pitch]);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) sums[warp][lane * 8 + e] = acc[e];
    __syncthreads();
    const int c = blockIdx.x * kColsumCols + threadIdx.x;
    if (c < N) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += sums[w][threadIdx.x];
        if (atomic) atomicAdd(part + c, s);                              // no workspace: the slabs meet in the zeroed output
        else part[static_cast<long>(blockIdx.y) * N + c] = s;
    }
}

// The backward's helper behind the GEMMs: dW = bf16(fp32 accumulator), 8 elements per thread, and db = the sum of the row
// slabs' partial sums, in a fixed order.  The first `db_blocks` blocks do db, 32 columns each (eight threads a column).
constexpr int kFinishCols = 32;
__global__ void __launch_bounds__(256) linear_finish_kernel(const float4* __restrict__ acc, uint4* __restrict__ out, long n8, const float* __restrict__ part,
                                                            int slabs, int N, void* __restrict__ db, int db_bf16, int db_blocks) {
    pdl_wait();
    pdl_trigger();
    if (static_cast<int>(blockIdx.x) < db_blocks) {
        __shared__ float sums[8][kFinishCols];
        const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, c = blockIdx.x * kFinishCols + lane;
        float s = 0.f;
        if (c < N)
            for (int j = grp; j < slabs; j += 8) s += part[static_cast<long>(j) * N + c];
        sums[grp][lane] = s;
        __syncthreads();
        if (grp == 0 && c < N) {
#pragma unroll
            for (int g = 1; g < 8; ++g) s += sums[g][lane];
            if (db_bf16) static_cast<__nv_bfloat16*>(db)[c] = __float2bfloat16(s);
            else static_cast<float*>(db)[c] = s;
        }
        return;
    }
    const long step = static_cast<long>(gridDim.x - db_blocks) * blockDim.x;
    for (long i = (static_cast<long>(blockIdx.x) - db_blocks) * blockDim.x + threadIdx.x; i < n8; i += step) {
        const float4 a = acc[2 * i], b = acc[2 * i + 1];
        out[i] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    }
}

}  // namespace ib200
