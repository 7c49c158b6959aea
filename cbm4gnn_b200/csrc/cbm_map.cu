// Dense maps of the GCN layers on the 5th-generation tensor cores (sm_100a): forward Y = X W^T and input
// gradient dX = dY W, fp32-accurate (see cbm_map.cuh).
//
// A GCN layer of the reference is `lin` followed by `propagate`
// (gnns/graph_convolutional_network/cbm_gcn.py:21-24): a bias-free [N,in] x [in,out] map in fp32.
// N is the number of nodes and the weights are small, so a map reads X once, writes Y once, and should be bound by
// HBM; what stood in the way was the split of both operands into bf16 terms, repeated for every tile.
//   * W is split once per block into shared memory (swizzled K-major rows, 3 terms, up to 192 KB) and stays
//     there: blocks are persistent and walk over row tiles of X.
//   * X goes from global memory to registers (16-byte loads, whole 32-byte sectors), is split there and stored
//     straight into tensor memory as the A operand: it never passes through shared memory, whose bandwidth
//     is left to the tensor cores for W.
//   * 8 warps load and split (two groups, alternate 32-deep chunks, the next chunk's loads in flight), one warp issues
//     the MMAs, 8 warps add up the accumulators and store Y with the ReLU or the mask applied (32 x 64 sums each).
//   * Y leaves (and the mask arrives) in whole 128-byte lines, 32 x 32 sums turned round through 4 KB of shared memory
//     per warp.
// Every 16-deep step has an accumulator of its own (see cbm_map.cuh), so the sums are added up every 16 columns; with
// accumulators of 64 columns 128 -> 256 took 96 us.  The warps that add up and store are what a map waits for: 52 % of their
// time went into adding, 34 - 49 % into storing.  So the next 8 columns leave tensor memory while 8 are added, and a
// block of 32 x 32 sums that is all there is stored without a question about single values.  235 868 rows: 128 -> 256 126
// -> 110 us, 256 -> 64 90 -> 85, 64 -> 256 masked 154 -> 137 (115 with the mask brought to L2 ahead); 400 000 rows 256 ->
// 256 342 -> 314, 100 -> 256 194 -> 176.  Where nothing masks the result, such a block leaves by one asynchronous copy of the
// TMA unit, and the warp goes on to the next: 110 -> 102, 85 -> 81; 314 -> 310, 176 -> 155, 256 -> 47 151 -> 129 (of which
// a step's MMAs issued as one 7).  Narrow tiles: see PAIR.
#include "cbm_launch.cuh"
#include "cbm_map.cuh"

#include <cuda.h>

#include <mutex>
#include <type_traits>

namespace cbm_map {

int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return n;
    n = cached[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 148;
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

int* timeout_word() {
    static std::mutex making;
    static std::atomic<int*> made{nullptr};
    if (int* word = made.load(std::memory_order_acquire)) return word;
    std::lock_guard<std::mutex> hold(making);
    if (int* word = made.load(std::memory_order_acquire)) return word;
    // The first map of a process may be one that is captured into a graph: the allocation is no part of it.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return nullptr;
    void* p = nullptr;
    const cudaError_t e = cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {  // the next call tries again
        cudaGetLastError();
        return nullptr;
    }
    *static_cast<int*>(p) = 0;
    made.store(static_cast<int*>(p), std::memory_order_release);
    return static_cast<int*>(p);
}

int check_timeout(const char* who) {
    int* w = timeout_word();
    if (!w) return cbm::fail(CBM_B200_ERR_CUDA, std::string(who) + ": no usable CUDA device on this thread");
    if (*(volatile int*)w) {
        *(volatile int*)w = 0;
        return cbm::fail(CBM_B200_ERR_TIMEOUT, std::string(who) + ": a bounded wait of an earlier dense map ran out; its result is invalid");
    }
    return CBM_B200_OK;
}

namespace {

// Two warps of each kind per scheduler: a warp alone on one issues an instruction every 4 - 5 cycles, and with 4
// epilogue warps (or 4 producers, also beside 16 epilogue warps) their work, not memory or the MMAs, was the bound.
constexpr int PRODUCER_WARPS = 8, EPILOGUE_WARPS = 8;
constexpr int MMA_WARP = PRODUCER_WARPS + EPILOGUE_WARPS;
constexpr int THREADS = 20 * 32;  // five warpgroups (of the last only one warp works), 96 registers a thread at launch ...
constexpr int LAUNCH_REGS = 96, PRODUCER_REGS = 104, EPILOGUE_REGS = 120, MMA_REGS = 24;  // ... and after the split
static_assert(PRODUCER_REGS > LAUNCH_REGS && EPILOGUE_REGS > LAUNCH_REGS && MMA_REGS < LAUNCH_REGS &&
                  256 * PRODUCER_REGS + 256 * EPILOGUE_REGS + 128 * MMA_REGS <= THREADS * LAUNCH_REGS,
              "setmaxnreg.inc and .dec only go up and down, within the registers of the launch");
constexpr int SMEM_MAX = 192 * 1024;     // for the split weights
constexpr int TURN_BYTES = 32 * 32 * 4;  // per epilogue warp
constexpr int SMEM_ALL = SMEM_MAX + EPILOGUE_WARPS * TURN_BYTES + 1024;
// An SM gives shared memory out in steps, and L1 the rest: 60 KB beside 196 KB (of which each block has 1 KB, and some bytes of
// its own), 28 KB beside more.  Rows that are no whole 128-byte lines need that room, as two chunks have a line
// in common.  A second place for results that takes it away costs more than it gives: 235 868 rows, 300 -> 80 156 us with it,
// 102 without; 300 -> 300 491 and 395; 180 000 rows, 200 -> 96 79 and 61.  Where it leaves it, it is worth having: 64 -> 128 29 us,
// 31 without.
constexpr int SMEM_BESIDE_L1 = 194 * 1024;

struct MapParams {
    CUtensorMap store;  // d, in boxes of 32 x 32, 128-byte swizzled; used where `boxes` is set
    const float* a;    // [m, k]
    const float* b;    // [n, k], or [k, n] when B_TRANS
    float* d;          // [m, n]
    const float* aux;  // [m, n]: the result is zeroed where aux <= 0
    int64_t lda, ldb, ldd, ldaux;
    int m, n, k;
    int bn;            // columns of a tile, a multiple of 16, at most 128
    int row_tiles;
    int steps;         // ceil(k / 16)
    int a_vec, d_vec, aux_vec;  // rows are 16-byte aligned
    int relu_in, relu_out, add; // max(a, 0) first; max(d, 0) last; d += instead of d =
    int boxes, places;  // 32 x 32 places of shared memory for each warp: 1 or 2
    int* timeout;
};

// One 16-deep step, issued as one: the five small products, smallest first, and the large one; then the arrival at `bar`
// once they are done.  `b_term`: distance of B's terms, as descriptors count it.
template <bool ARRIVE>
__device__ __forceinline__ void mma_step(u32 d, u32 a, u64 b, u64 b_term, u32 idesc, u32 bar) {
    asm volatile(
        "{\n\t.reg .pred e, no, yes;\n\t.reg .b64 b1, b2;\n\t.reg .b32 a1, a2;\n\t"
        "elect.sync _|e, 0xffffffff;\n\tsetp.ne.u32 no, 0, 0;\n\tsetp.eq.u32 yes, 0, 0;\n\t"
        "add.s64 b1, %2, %3;\n\tadd.s64 b2, b1, %3;\n\tadd.u32 a1, %1, 16;\n\tadd.u32 a2, %1, 32;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], %2, %4, no;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %4, yes;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b2, %4, yes;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], %2, %4, yes;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b1, %4, yes;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %4, yes;\n\t"
        "}" ::"r"(d),
        "r"(a), "l"(b), "l"(b_term), "r"(idesc)
        : "memory");
    if (ARRIVE) commit(bar);
}

__device__ __forceinline__ void ld8(float (&r)[8], u32 at) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(at));
}

// PAIR, for tiles of up to 64 columns: an accumulator's place holds two, those of a chunk's two steps, which go from the MMA
// warp to the sum warps and back together.  What bounds a narrow tile is that way, whatever is left out of the rest (256 ->
// 47: 130 us without the fetches, without the stores or with one product of six): 129 -> 115 us, 256 -> 64 82 -> 74.
// EXTRA: 0 plain, 1 with a mask, 2 with any of a mask and earlier passes' results to add to.
template <bool B_TRANS, int EXTRA, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1) map_kernel(const __grid_constant__ MapParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ u64 s_bar[2 * A_SLOTS + 5];  // A full x4, A empty x4, accumulator full x2, accumulator empty x2, drained
    __shared__ u32 s_tmem;
    __shared__ int s_gave_up;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const u32 bars = smem_u32(s_bar);
    const u32 a_full = bars, a_empty = bars + 8 * A_SLOTS, d_full = bars + 16 * A_SLOTS, d_empty = d_full + 16, drained = d_full + 32;
    const int n0 = blockIdx.x * p.bn;
    const int chunks = (p.steps + 1) / 2;                // 32-deep chunks of a row tile
    const int kblocks = (chunks + 1) / 2;                // 64-deep blocks
    const u32 block = (u32)p.bn * 128;                   // one 64-deep block of one term of W
    const u32 term = block * (u32)kblocks;
    unsigned char* turn = smem + 3 * term;

    if (warp == MMA_WARP) tmem_alloc(smem_u32(&s_tmem));
    if (threadIdx.x == 0) {
        for (int s = 0; s < A_SLOTS; ++s) {
            bar_init(a_full + 8 * s, 4);
            bar_init(a_empty + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            bar_init(d_full + 8 * s, 1);
            bar_init(d_empty + 8 * s, EPILOGUE_WARPS);
        }
        bar_init(drained, 1);
        s_gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cbm::wait_before();
    // The weights, split, into shared memory: two pieces of 8 values a thread at a time, so that their fetches overlap.
    const int k8s = 2 * p.steps, pieces = p.bn * k8s;
    const bool b_vec = !B_TRANS && p.ldb % 4 == 0 && (reinterpret_cast<u64>(p.b) & 15) == 0;
    for (int i0 = threadIdx.x; i0 < pieces; i0 += 2 * THREADS) {
        float x[2][8];
        int at_n[2], at_k[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + h * THREADS;
            const bool on = i < pieces;
            const int n = B_TRANS ? i % p.bn : i / k8s, k8 = B_TRANS ? i / p.bn : i % k8s;
            at_n[h] = n;
            at_k[h] = k8;
            const float* from = B_TRANS ? p.b + (int64_t)(k8 * 8) * p.ldb + n0 + n : p.b + (int64_t)(n0 + n) * p.ldb + k8 * 8;
            if (b_vec && k8 * 8 + 8 <= p.k) {
                const float4 lo = fetch4(from, on && n0 + n < p.n), hi = fetch4(from + 4, on && n0 + n < p.n);
                x[h][0] = lo.x, x[h][1] = lo.y, x[h][2] = lo.z, x[h][3] = lo.w;
                x[h][4] = hi.x, x[h][5] = hi.y, x[h][6] = hi.z, x[h][7] = hi.w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    x[h][j] = fetch1(from + (B_TRANS ? j * p.ldb : j), on && n0 + n < p.n && k8 * 8 + j < p.k);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (i0 + h * THREADS < pieces)
                store_split8(smem + (u32)(at_k[h] >> 3) * block + swizzled((u32)at_n[h], (u32)(at_k[h] & 7)), term, x[h]);
    }
    fence_async();
    fence_before();
    __syncthreads();
    fence_after();
    const u32 tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    volatile int* gave_up = &s_gave_up;

    if (warp < PRODUCER_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
        const int quarter = warp & 3, group = warp >> 2;
        const int row_in = quarter * 32 + (lane >> 2), k_in = 4 * (lane & 3);
        float4 v[2][4][2];  // [buffer][8-row group][16-deep step]
        // fetches only; what lies past column k is zeroed when the values are used
        auto load = [&](int buf, int tile, int c) {
            const float* s0 = p.a + (int64_t)(tile * 128 + row_in) * p.lda + c * CHUNK_K + k_in;
            const int left = p.m - (tile * 128 + row_in), k = c * CHUNK_K + k_in;
            if (p.a_vec) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int s = 0; s < 2; ++s) v[buf][i][s] = fetch4(s0 + 8 * i * p.lda + 16 * s, 8 * i < left && k + 16 * s < p.k);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const float* at = s0 + 8 * i * p.lda + 16 * s;
                        const bool row = 8 * i < left;
                        v[buf][i][s].x = fetch1(at, row && k + 16 * s < p.k);
                        v[buf][i][s].y = fetch1(at + 1, row && k + 16 * s + 1 < p.k);
                        v[buf][i][s].z = fetch1(at + 2, row && k + 16 * s + 2 < p.k);
                        v[buf][i][s].w = fetch1(at + 3, row && k + 16 * s + 3 < p.k);
                    }
            }
        };
        // this group's chunks: those whose running number has the group's parity
        int tile = blockIdx.y, c = group;
        while (c >= chunks) {
            c -= chunks;
            tile += gridDim.y;
        }
        if (tile < p.row_tiles) load(0, tile, c);
        for (u32 run = group; tile < p.row_tiles; run += 4) {
#pragma unroll
            for (int buf = 0; buf < 2; ++buf) {
                if (tile >= p.row_tiles) break;
                int next_tile = tile, next_c = c + 2;
                while (next_c >= chunks) {
                    next_c -= chunks;
                    next_tile += gridDim.y;
                }
                if (next_tile < p.row_tiles) load(buf ^ 1, next_tile, next_c);
                const u32 r = run + 2 * buf, slot = r % A_SLOTS;
                if (r >= A_SLOTS && !warp_wait(a_empty + 8 * slot, ((r / A_SLOTS) + 1) & 1, gave_up, p.timeout)) goto done;
                const u32 at = tmem + A_COL + slot * A_SLOT_COLS + ((u32)(quarter * 32) << 16);
                const bool ragged_k = p.a_vec && c * CHUNK_K + CHUNK_K > p.k;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    u32 t[3][8];
#pragma unroll
                    for (int i = 2 * h; i < 2 * h + 2; ++i)
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            float4 x = v[buf][i][s];
                            if (ragged_k) {  // an aligned row's last vector may reach past column k
                                const int k = c * CHUNK_K + 16 * s + k_in;
                                x.y = k + 1 < p.k ? x.y : 0.f;
                                x.z = k + 2 < p.k ? x.z : 0.f;
                                x.w = k + 3 < p.k ? x.w : 0.f;
                            }
                            if (p.relu_in) x = relu(x);
                            const int o = 4 * s + 2 * (i & 1);
                            split2(x.x, x.y, t[0][o], t[1][o], t[2][o]);
                            split2(x.z, x.w, t[0][o + 1], t[1][o + 1], t[2][o + 1]);
                        }
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        asm volatile(
                            "tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(
                                at + 16 * q + ((u32)(16 * h) << 16)),
                            "r"(t[q][0]), "r"(t[q][1]), "r"(t[q][2]), "r"(t[q][3]), "r"(t[q][4]), "r"(t[q][5]), "r"(t[q][6]),
                            "r"(t[q][7])
                            : "memory");
                }
                wait_st();
                fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(a_full + 8 * slot);
                tile = next_tile;
                c = next_c;
            }
        }
    } else if (warp >= MMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MMA_REGS));
        if (warp > MMA_WARP) goto done;
        const u32 idesc = idesc_of((u32)p.bn);
        const u32 b0 = smem_u32(smem);
        u32 run = 0, it = 0;
        bool ok = true;
        for (int tile = blockIdx.y; tile < p.row_tiles && ok; tile += gridDim.y)
            for (int c = 0; c < chunks && ok; ++c, ++run) {
                const u32 slot = run % A_SLOTS, a = tmem + A_COL + slot * A_SLOT_COLS;
                const u32 b = b0 + (u32)(c >> 1) * block + 64 * (c & 1);
                if (!(ok = warp_wait(a_full + 8 * slot, (run / A_SLOTS) & 1, gave_up, p.timeout))) break;
                if constexpr (PAIR) {
                    const u32 ds = it & 1, use = it >> 1, d = tmem + ds * D_COLS;
                    if (use > 0 && !(ok = warp_wait(d_empty + 8 * ds, (use + 1) & 1, gave_up, p.timeout))) break;
                    mma_step<false>(d, a, desc_of(b), (u64)(term >> 4), idesc, 0);
                    if (2 * c + 1 < p.steps) mma_step<false>(d + D_COLS / 2, a + 8, desc_of(b + 32), (u64)(term >> 4), idesc, 0);
                    commit(d_full + 8 * ds);
                    commit(a_empty + 8 * slot);
                    ++it;
                    continue;
                }
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    if (2 * c + s >= p.steps) break;
                    const u32 ds = it & 1, use = it >> 1, d = tmem + ds * D_COLS;
                    if (use > 0 && !(ok = warp_wait(d_empty + 8 * ds, (use + 1) & 1, gave_up, p.timeout))) break;
                    mma_step<true>(d, a + 8 * s, desc_of(b + 32 * s), (u64)(term >> 4), idesc, d_full + 8 * ds);
                    ++it;
                }
                if (ok) commit(a_empty + 8 * slot);
            }
        if (!ok) {  // the MMAs under way end before the block frees its tensor memory
            commit(drained);
            for (u32 spins = 0; spins < (1u << 20) && !bar_poll(drained, 0); ++spins) {
            }
            __syncwarp();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPILOGUE_REGS));
        // This warp: 32 rows by up to two blocks of 32 columns from column c_lo on; lane = row while the sums are
        // collected, then, block by block, lane = 4 columns from 4 * (lane % 8) on of the rows lane / 8 + 4 i.
        const int quarter = warp & 3, half = (warp - PRODUCER_WARPS) >> 2;
        const int first_width = min(p.bn, (p.bn + 63) / 64 * 32);
        const int c_lo = half * first_width, width = half ? p.bn - first_width : first_width;
        const int row_in = quarter * 32 + (lane >> 3), col_in = c_lo + 4 * (lane & 7);
        float4* const mine0 = reinterpret_cast<float4*>(turn + (warp - PRODUCER_WARPS) * p.places * TURN_BYTES);
        float4* mine = mine0;
        u32 it = 0, boxed = 0;
        for (int tile = blockIdx.y; tile < p.row_tiles; tile += gridDim.y) {
            const int row0 = tile * 128 + row_in;
            // Of the mask only one bit per value is kept, fetched while the products of this tile are under way.
            u32 keep[2] = {0xffffffffu, 0xffffffffu};
            if (EXTRA && p.aux) {
                float4 x[2][8];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int col = 32 * b + col_in, left = col < c_lo + width ? p.n - n0 - col : 0;
                    const float* s0 = p.aux + (int64_t)row0 * p.ldaux + n0 + col;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float* s = s0 + 4 * i * p.ldaux;
                        const bool in = row0 + 4 * i < p.m;
                        if (p.aux_vec) {
                            x[b][i] = fetch4(s, in && left > 0);  // what lies past column n is not stored
                        } else {
                            x[b][i].x = fetch1(s, in && left > 0);
                            x[b][i].y = fetch1(s + 1, in && left > 1);
                            x[b][i].z = fetch1(s + 2, in && left > 2);
                            x[b][i].w = fetch1(s + 3, in && left > 3);
                        }
                    }
                }
                // The next tile's mask is brought to L2 meanwhile, a row of this warp's columns by each lane: these fetches,
                // which nothing is ahead of, took a trip to memory per tile (64 -> 256 masked 139 us, 115 with it).
                {
                    const int64_t row = (int64_t)(tile + (int)gridDim.y) * 128 + quarter * 32 + lane;
                    const float* at = p.aux + row * p.ldaux + n0 + c_lo;
                    if (row < p.m && n0 + c_lo < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
                    if (row < p.m && n0 + c_lo + 32 < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 32));
                }
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    u32 bits = 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        // (a NaN lets the gradient through, as the backward of torch.relu does)
                        bits |= ((x[b][i].x <= 0.f ? 0u : 1u) | (x[b][i].y <= 0.f ? 0u : 2u) | (x[b][i].z <= 0.f ? 0u : 4u) |
                                 (x[b][i].w <= 0.f ? 0u : 8u))
                                << (4 * i);
                    keep[b] = bits;
                }
            }
            // The first step sets the sums, the others add to them (told apart at compile time: the sums must not
            // be live while the mask is fetched).
            constexpr int BLOCKS = PAIR ? 1 : 2;  // of 32 columns
            float acc[BLOCKS][32];
            auto collect = [&](auto first, bool second) -> bool {
                const u32 ds = it & 1, use = it >> 1;
                if (!warp_wait(d_full + 8 * ds, use & 1, gave_up, p.timeout)) return false;
                const u32 at = tmem + ds * D_COLS + c_lo + ((u32)(quarter * 32) << 16);
                // From `width` on nothing is fetched and what the registers held before is added once more: to sums that are
                // neither stored value by value nor, where a box is stored, within the result's columns.  (A half has 16 columns
                // at least, so both registers' 8 have been fetched.  Leaving the loop there is slower: 180 000 rows, 128 ->
                // 112 42 us, 45 with it; 64 -> 80 25 and 26.)
                float r[2][8];
                ld8(r[0], at);
#pragma unroll
                for (int q = 0; q < 8; ++q) {  // the next 8 columns are on their way while these are added
                    const bool more = PAIR ? (q != 3 || second) : 8 * (q + 1) < width;
                    if (PAIR && q == 4 && !second) break;
                    wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i) asm volatile("" : "+f"(r[q & 1][i]));  // not before the wait
                    if (q < 7 && more) ld8(r[(q + 1) & 1], PAIR && q >= 3 ? at + D_COLS / 2 + 8 * (q - 3) : at + 8 * (q + 1));
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        float &s = acc[PAIR ? 0 : q >> 2][8 * (q & 3) + i], &t = acc[PAIR ? 0 : q >> 2][8 * (q & 3) + i + 1];
                        if (decltype(first)::value && !(PAIR && q >= 4)) {
                            s = r[q & 1][i];
                            t = r[q & 1][i + 1];
                        } else {
                            add2(s, t, r[q & 1][i], r[q & 1][i + 1]);
                        }
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(d_empty + 8 * ds);
                ++it;
                return true;
            };
            if constexpr (PAIR) {
                if (!collect(std::true_type{}, p.steps > 1)) goto done;
                for (int s = 2; s < p.steps; s += 2)
                    if (!collect(std::false_type{}, s + 1 < p.steps)) goto done;
            } else {
                if (!collect(std::true_type{}, false)) goto done;
                for (int s = 1; s < p.steps; ++s)
                    if (!collect(std::false_type{}, false)) goto done;
            }
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                if (32 * b >= width) break;
                if (EXTRA == 0 && p.boxes) {
                    // A box that holds these columns only, or that the last column cuts off, goes out by one asynchronous copy.
                    // (What is cut off is cut at 16 bytes: a width that ends elsewhere leaves its last block value by value.)
                    // What lay in its place before may still be on its way out: the place is free once that has been read.
                    const bool whole = 32 * b + 32 <= width && n0 + c_lo + 32 * b + 32 <= p.n;
                    const bool box = whole || (p.n % 4 == 0 && n0 + c_lo + width >= p.n);
                    if (box && p.places == 2) {
                        mine = mine0 + (boxed & 1) * (TURN_BYTES / 16);
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    } else {
                        mine = mine0;
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    }
                    __syncwarp();
                    if (box) {
                        ++boxed;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float4 y = make_float4(acc[b][4 * j], acc[b][4 * j + 1], acc[b][4 * j + 2], acc[b][4 * j + 3]);
                            if (p.relu_out) y = relu(y);
                            mine[lane * 8 + (j ^ (lane & 7))] = y;
                        }
                        fence_async();
                        __syncwarp();
                        const int row = tile * 128 + quarter * 32;
                        if (lane == 0) {
                            if (row < p.m)
                                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&p.store),
                                             "r"(n0 + c_lo + 32 * b), "r"(row), "r"(smem_u32(mine))
                                             : "memory");
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                        continue;
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    mine[lane * 8 + (j ^ (lane & 7))] = make_float4(acc[b][4 * j], acc[b][4 * j + 1], acc[b][4 * j + 2], acc[b][4 * j + 3]);
                __syncwarp();
                const int col = 32 * b + col_in, left = col < c_lo + width ? p.n - n0 - col : 0;
                float* d0 = p.d + (int64_t)row0 * p.ldd + n0 + col;
                // A block that is all there and goes out in whole lines: nothing is asked about single values.
                if (EXTRA < 2 && p.d_vec && tile * 128 + 128 <= p.m && 32 * b + 32 <= width && n0 + c_lo + 32 * b + 32 <= p.n) {
                    const float4* from = mine + (lane >> 3) * 8 + ((lane & 7) ^ (lane >> 3));
                    const float4* odd = mine + (lane >> 3) * 8 + ((lane & 7) ^ (lane >> 3) ^ 4);
                    const int64_t step = 4 * p.ldd;
#pragma unroll
                    for (int i = 0; i < 8; ++i, d0 += step) {
                        float4 y = (i & 1 ? odd : from)[32 * i];
                        if constexpr (EXTRA) {
                            const u32 bits = keep[b] >> (4 * i);
                            y = make_float4(bits & 1 ? y.x : 0.f, bits & 2 ? y.y : 0.f, bits & 4 ? y.z : 0.f, bits & 8 ? y.w : 0.f);
                        }
                        if (p.relu_out) y = relu(y);
                        *reinterpret_cast<float4*>(d0) = y;
                    }
                    __syncwarp();
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = (lane >> 3) + 4 * i;
                    float4 y = mine[r * 8 + ((lane & 7) ^ (r & 7))];
                    float* d = d0 + 4 * i * p.ldd;
                    const int here = row0 + 4 * i < p.m ? left : 0;
                    if constexpr (EXTRA) {
                        if (EXTRA == 2 && p.add) {
                            if (here > 0) y.x += d[0];
                            if (here > 1) y.y += d[1];
                            if (here > 2) y.z += d[2];
                            if (here > 3) y.w += d[3];
                        }
                        const u32 bits = keep[b] >> (4 * i);
                        y = make_float4(bits & 1 ? y.x : 0.f, bits & 2 ? y.y : 0.f, bits & 4 ? y.z : 0.f, bits & 8 ? y.w : 0.f);
                    }
                    if (p.relu_out) y = relu(y);
                    if (p.d_vec && here >= 4) {
                        *reinterpret_cast<float4*>(d) = y;
                    } else {
                        if (here > 0) d[0] = y.x;
                        if (here > 1) d[1] = y.y;
                        if (here > 2) d[2] = y.z;
                        if (here > 3) d[3] = y.w;
                    }
                }
                __syncwarp();
            }
        }
    }
done:
    if (EXTRA == 0 && p.boxes) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // before the memory they read is given up
    __syncwarp();
    fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_free(tmem);
}

// The map of d for asynchronous stores; false where the driver has none to offer.
bool make_boxes(CUtensorMap* map, float* d, int64_t ldd, int m, int n) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult got;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &got) != cudaSuccess || got != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            fn = nullptr;
        }
        return reinterpret_cast<Encode>(fn);
    }();
    if (!encode || ldd * 4 >= (int64_t)1 << 40) return false;
    const cuuint64_t size[2] = {(cuuint64_t)n, (cuuint64_t)m}, pitch[1] = {(cuuint64_t)ldd * 4};
    const cuuint32_t box[2] = {32, 32}, step[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, d, size, pitch, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool aligned_rows(const void* p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0; }

int round_up(int v, int to) { return (v + to - 1) / to * to; }

int smem_of(int steps, int bn, int places) {
    return 3 * ((steps + 3) / 4) * bn * 128 + places * EPILOGUE_WARPS * TURN_BYTES + 1024;
}

template <bool B_TRANS, int EXTRA, bool PAIR>
int launch_form(const char* who, const MapParams& p, int sms, cudaStream_t stream) {
    if (!allow_smem<map_kernel<B_TRANS, EXTRA, PAIR>>(SMEM_ALL))
        return cbm::fail(CBM_B200_ERR_CUDA, std::string(who) + ": shared memory size refused");
    const int n_tiles = (p.n + p.bn - 1) / p.bn;
    const dim3 grid(n_tiles, std::max(1, std::min(p.row_tiles, sms / n_tiles)));
    // at least half of an SM's shared memory, so that two blocks, which both want all tensor memory, never share one
    const int smem = std::max(smem_of(p.steps, p.bn, p.places), 120 * 1024);
    cbm::launch_next(map_kernel<B_TRANS, EXTRA, PAIR>, grid, THREADS, smem, stream, p);
    if (cudaGetLastError() != cudaSuccess) return cbm::fail(CBM_B200_ERR_CUDA, std::string(who) + ": launch failed");
    return CBM_B200_OK;
}

template <bool B_TRANS, int EXTRA>
int launch(const char* who, const MapParams& p, int sms, cudaStream_t stream) {
    return p.bn <= 64 ? launch_form<B_TRANS, EXTRA, true>(who, p, sms, stream) : launch_form<B_TRANS, EXTRA, false>(who, p, sms, stream);
}

// d [m, n] = a [m, k] b^T, b [n, k] (b_trans: [k, n]).
int run_map(const char* who, const float* a, int64_t lda, const float* b, int64_t ldb, bool b_trans, float* d, int64_t ldd,
            const float* aux, int64_t ldaux, int m, int n, int k, bool relu_in, bool relu_out, cudaStream_t stream) {
    if (lda < k || ldb < (b_trans ? n : k) || ldd < n)
        return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": a leading dimension is smaller than its row");
    if (const int rc = check_timeout(who)) return rc;
    const int sms = sm_count();
    const int row_tiles = (m + 127) / 128;
    // Tile width: up to 128 columns (an epilogue warp keeps 32 x 64 sums in registers), less where their split
    // weights, up to 512 of the contraction, would not fit into shared memory (a longer contraction is cut into
    // passes that add to d).  Few row tiles: narrower, so that every SM has a tile, down to 32 columns.
    const int n16 = round_up(n, 16);
    const auto depth = [](int bn) { return SMEM_MAX / (384 * bn) * 64; };  // contraction that fits beside bn columns
    int bn = std::min(n16, 128);
    while (bn > 16 && depth(bn) < std::min(k, 512)) bn -= 16;
    const int want = std::max((n16 + bn - 1) / bn, std::min(sms / row_tiles, (n16 + 31) / 32));
    bn = round_up((n16 + want - 1) / want, 16);
    const int most = std::min(round_up(k, 16), depth(bn));
    const int passes = (k + most - 1) / most;
    const int seg = round_up((k + passes - 1) / passes, 16);
    for (int k0 = 0; k0 < k; k0 += seg) {
        MapParams p{};
        const bool last = k0 + seg >= k;
        p.a = a + k0;
        p.b = b_trans ? b + (int64_t)k0 * ldb : b + k0;
        p.d = d;
        p.lda = lda;
        p.ldb = ldb;
        p.ldd = ldd;
        p.m = m;
        p.n = n;
        p.k = std::min(seg, k - k0);
        p.bn = bn;
        p.row_tiles = row_tiles;
        p.steps = (p.k + 15) / 16;
        p.a_vec = aligned_rows(p.a, lda);
        p.d_vec = aligned_rows(d, ldd);
        p.relu_in = relu_in;
        p.relu_out = relu_out && last;
        p.add = k0 > 0;
        // (a map of the result takes the host 2 us, and a block that has one tile has nothing to go on to)
        p.boxes = p.d_vec && passes == 1 && !aux && row_tiles >= sms && make_boxes(&p.store, d, ldd, m, n);
        p.places = p.boxes && smem_of(p.steps, bn, 2) <= SMEM_BESIDE_L1 ? 2 : 1;
        if (aux) {
            p.aux = aux;
            p.ldaux = ldaux;
            p.aux_vec = aligned_rows(aux, ldaux);
        }
        p.timeout = timeout_word();
        const int rc = b_trans ? (p.add ? launch<true, 2>(who, p, sms, stream)
                                        : p.aux ? launch<true, 1>(who, p, sms, stream) : launch<true, 0>(who, p, sms, stream))
                               : (p.add ? launch<false, 2>(who, p, sms, stream) : launch<false, 0>(who, p, sms, stream));
        if (rc) return rc;
    }
    return CBM_B200_OK;
}

}  // namespace
}  // namespace cbm_map

using namespace cbm_map;

extern "C" int cbm_b200_dense_forward(const float* x, int64_t ldx, const float* w, int64_t ldw, float* y, int64_t ldy,
                                      int32_t n_rows, int32_t n_in, int32_t n_out, void* stream) {
    if (!x || !w || !y || n_rows < 0 || n_in <= 0 || n_out <= 0)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_forward: bad arguments");
    if (n_rows == 0) return CBM_B200_OK;
    return run_map("dense_forward", x, ldx, w, ldw, false, y, ldy, nullptr, 0, n_rows, n_out, n_in, false, false, (cudaStream_t)stream);
}

extern "C" int cbm_b200_dense_forward_relu(const float* x, int64_t ldx, const float* w, int64_t ldw, float* y,
                                           int64_t ldy, int32_t n_rows, int32_t n_in, int32_t n_out, void* stream) {
    if (!x || !w || !y || n_rows < 0 || n_in <= 0 || n_out <= 0)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_forward_relu: bad arguments");
    if (n_rows == 0) return CBM_B200_OK;
    return run_map("dense_forward_relu", x, ldx, w, ldw, false, y, ldy, nullptr, 0, n_rows, n_out, n_in, false, true, (cudaStream_t)stream);
}

extern "C" int cbm_b200_dense_forward_of_relu(const float* x, int64_t ldx, const float* w, int64_t ldw, float* y, int64_t ldy,
                                              int32_t n_rows, int32_t n_in, int32_t n_out, int32_t relu, void* stream) {
    if (!x || !w || !y || n_rows < 0 || n_in <= 0 || n_out <= 0)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_forward_of_relu: bad arguments");
    if (n_rows == 0) return CBM_B200_OK;
    return run_map("dense_forward_of_relu", x, ldx, w, ldw, false, y, ldy, nullptr, 0, n_rows, n_out, n_in, true, relu != 0,
                   (cudaStream_t)stream);
}

extern "C" int cbm_b200_dense_grad_input(const float* dy, int64_t lddy, const float* w, int64_t ldw, float* dx,
                                         int64_t lddx, int32_t n_rows, int32_t n_in, int32_t n_out, void* stream) {
    if (!dy || !w || !dx || n_rows < 0 || n_in <= 0 || n_out <= 0)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_grad_input: bad arguments");
    if (n_rows == 0) return CBM_B200_OK;
    return run_map("dense_grad_input", dy, lddy, w, ldw, true, dx, lddx, nullptr, 0, n_rows, n_in, n_out, false, false, (cudaStream_t)stream);
}

extern "C" int cbm_b200_dense_grad_input_relu(const float* dy, int64_t lddy, const float* w, int64_t ldw, const float* h,
                                              int64_t ldh, float* dx, int64_t lddx, int32_t n_rows, int32_t n_in,
                                              int32_t n_out, void* stream) {
    if (!dy || !w || !h || !dx || n_rows < 0 || n_in <= 0 || n_out <= 0)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_grad_input_relu: bad arguments");
    if (ldh < n_in) return cbm::fail(CBM_B200_ERR_ARG, "dense_grad_input_relu: rows of h must hold n_in floats");
    if (n_rows == 0) return CBM_B200_OK;
    return run_map("dense_grad_input_relu", dy, lddy, w, ldw, true, dx, lddx, h, ldh, n_rows, n_in, n_out, false, false,
                   (cudaStream_t)stream);
}
