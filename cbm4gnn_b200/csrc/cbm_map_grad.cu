// Weight gradient dW = dY^T X of the dense maps (see cbm_map.cuh for the arithmetic): a contraction over the
// N rows of the graph (hundreds of thousands) into a small [out, in] result, bound by reading dY and X.
//
// Each block takes one tile of the result (128 columns of one operand by 64 or 128 of the other) and one range of
// rows.  Both operands are needed with the rows as the contraction, that is transposed: a lane owns one column
// (or two) and reads it down 32 (8) rows, a warp's reads being 128-byte lines (two), splits, and has neighbours of the
// contraction in its own registers - written to tensor memory for the first operand, as 16-byte pieces of swizzled
// K-major rows to shared memory for the second.  8 + 7 warps do that, the next chunk's loads in flight, one warp
// issues the MMAs, 8 warps add the accumulators of every 64 rows to sums in registers.  The ranges' partial results
// are added in a fixed order by a second kernel, which also turns the tile round where the operands' roles were
// exchanged.
//
// A chunk's way through a block (load, split, store) is a chain that the memory's latency bounds, not its rate, so
// each warp of the second operand asks for its next task's rows before it works on this one's, and rows without gaps
// are brought to L2 AHEAD chunks early.  With three warps for the second operand they were what everyone waited for (the
// MMA warp 62 % of its time); seven that take its tasks in turn leave the chain of the first operand.  235 868 rows:
// 64 x 256 101 -> 92 us, 256 x 128 129 -> 110, 256 x 256 249 -> 202.
#include "cbm_launch.cuh"
#include "cbm_map.cuh"

namespace cbm_map {
namespace {

constexpr int A_WARPS = 8, B_WARPS = 7, SUM_WARPS = 8;
constexpr int MMA_WARP = A_WARPS + B_WARPS, FIRST_SUM_WARP = MMA_WARP + 1;
constexpr int GRAD_THREADS = (FIRST_SUM_WARP + SUM_WARPS) * 32;  // 24 warps, 80 registers a thread at launch ...
constexpr int LAUNCH_REGS = 80, A_REGS = 96, B_REGS = 64, SUM_REGS = 80;  // ... and after the split (the MMA warp has B's share)
static_assert(A_REGS > LAUNCH_REGS && SUM_REGS == LAUNCH_REGS && B_REGS < LAUNCH_REGS &&
                  32 * (A_WARPS * A_REGS + (B_WARPS + 1) * B_REGS + SUM_WARPS * SUM_REGS) <= GRAD_THREADS * LAUNCH_REGS,
              "setmaxnreg.inc and .dec only go up and down, within the registers of the launch");
// Chunks between a prefetch to L2 and the loads: 3 and 4 measure alike, 8 costs 5 % and 12 13 % (L2 evicts early).
constexpr int AHEAD = 4;
constexpr int MAX_PARTS = CBM_B200_DENSE_MAX_CHUNKS;
static_assert(FIRST_SUM_WARP % 4 == 0, "a warp reads the tensor-memory lanes of its number modulo 4");

struct GradParams {
    const float* a;  // [rows, m]
    const float* b;  // [rows, n]
    float* part;     // [gridDim.y] x [m, n]
    int64_t lda, ldb;
    int rows, m, n;
    int bn;          // columns of b in a tile, 64 or 128
    int n_tiles;     // tiles along n
    int chunks_per;  // 32-row chunks per block, even
    int relu_a, relu_b;  // max(., 0) first
    int b_vec;       // pairs of columns of b are 8-byte aligned
    int* timeout;
};

// Fetches without a condition, volatile for the same reason as fetch1.
__device__ __forceinline__ float fetch(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 fetch_pair(const float* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

__global__ void __launch_bounds__(GRAD_THREADS, 1) grad_kernel(const __grid_constant__ GradParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ u64 s_bar[2 * A_SLOTS + 5];  // full x4, empty x4, accumulator full x2, accumulator empty x2, drained
    __shared__ u32 s_tmem;
    __shared__ int s_gave_up;
    unsigned char* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const u32 bars = smem_u32(s_bar);
    const u32 full = bars, empty = bars + 8 * A_SLOTS, d_full = bars + 16 * A_SLOTS, d_empty = d_full + 16, drained = d_full + 32;
    const int m0 = (int)(blockIdx.x / (u32)p.n_tiles) * 128, n0 = (int)(blockIdx.x % (u32)p.n_tiles) * p.bn;
    const int total = (p.rows + CHUNK_K - 1) / CHUNK_K;
    const int first = (int)blockIdx.y * p.chunks_per;
    const int chunks = max(0, min(p.chunks_per, total - first));
    const int kblocks = (chunks + 1) / 2;
    const u32 term = (u32)p.bn * 128, stage = 3 * term;  // a stage holds two chunks side by side (64 values deep)

    if (warp == MMA_WARP) tmem_alloc(smem_u32(&s_tmem));
    if (threadIdx.x == 0) {
        for (int s = 0; s < A_SLOTS; ++s) {
            bar_init(full + 8 * s, 4 + p.bn / 64 * 4);  // four A warps, and every task of B
            bar_init(empty + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            bar_init(d_full + 8 * s, 1);
            bar_init(d_empty + 8 * s, SUM_WARPS);
        }
        bar_init(drained, 1);
        s_gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cbm::wait_before();
    fence_before();
    __syncthreads();
    fence_after();
    const u32 tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    volatile int* gave_up = &s_gave_up;

    if (warp < A_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(A_REGS));
        // lane = column; two groups of four warps, alternate chunks.  Lanes past the last column read it again: their
        // rows of the tile are not stored.
        const int quarter = warp & 3, group = warp >> 2;
        const float* src = p.a + min(m0 + quarter * 32 + lane, p.m - 1);
        float v[CHUNK_K];
        auto load = [&](int c) {
            const int r0 = (first + c) * CHUNK_K;
            const float* at = src + (int64_t)r0 * p.lda;
            if (r0 + CHUNK_K <= p.rows) {
#pragma unroll
                for (int i = 0; i < CHUNK_K; ++i, at += p.lda) v[i] = fetch(at);
            } else {
#pragma unroll
                for (int i = 0; i < CHUNK_K; ++i, at += p.lda) v[i] = fetch1(at, r0 + i < p.rows);
            }
        };
        // Rows that follow one another without a gap are also brought to L2 some chunks ahead, by one request each.
        auto ahead = [&](int c) {
            const int r0 = (first + c) * CHUNK_K, rows = min(CHUNK_K, p.rows - r0);
            if (blockIdx.x != 0 || warp != 0 || lane > 1 || c >= chunks || rows <= 0) return;
            const float* at = lane ? p.b + (int64_t)r0 * p.ldb : p.a + (int64_t)r0 * p.lda;
            const int width = lane ? p.n : p.m;
            const u32 bytes = (u32)(rows * width) * 4;
            if ((lane ? p.ldb : p.lda) == width && (((u64)at | bytes) & 15) == 0)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(bytes));
        };
        for (int c = 1; c < AHEAD; ++c) ahead(c);
        if (group < chunks) load(group);
        for (int c = group; c < chunks; c += 2) {
            ahead(c + AHEAD);
            ahead(c + AHEAD + 1);
            const u32 slot = (u32)c % A_SLOTS;
            u32 t[3][CHUNK_K / 2];
#pragma unroll
            for (int i = 0; i < CHUNK_K / 2; ++i) {
                float x = v[2 * i], y = v[2 * i + 1];
                if (p.relu_a) {
                    x = relu(x);
                    y = relu(y);
                }
                split2(x, y, t[0][i], t[1][i], t[2][i]);
            }
            if (c + 2 < chunks) load(c + 2);
            if (c >= A_SLOTS && !warp_wait(empty + 8 * slot, ((u32)c / A_SLOTS + 1) & 1, gave_up, p.timeout)) goto done;
            const u32 at = tmem + A_COL + slot * A_SLOT_COLS + ((u32)(quarter * 32) << 16);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                asm volatile(
                    "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
                    "%15, %16};" ::"r"(at + 16 * q),
                    "r"(t[q][0]), "r"(t[q][1]), "r"(t[q][2]), "r"(t[q][3]), "r"(t[q][4]), "r"(t[q][5]), "r"(t[q][6]),
                    "r"(t[q][7]), "r"(t[q][8]), "r"(t[q][9]), "r"(t[q][10]), "r"(t[q][11]), "r"(t[q][12]), "r"(t[q][13]),
                    "r"(t[q][14]), "r"(t[q][15])
                    : "memory");
            wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(full + 8 * slot);
        }
    } else if (warp < FIRST_SUM_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(B_REGS));
        if (warp == MMA_WARP) {
            const u32 idesc = idesc_of((u32)p.bn), b0 = smem_u32(smem);
            bool ok = true;
            for (int kb = 0; kb < kblocks; ++kb) {
                const u32 ds = kb & 1, use = kb >> 1;
                if (use > 0 && !(ok = warp_wait(d_empty + 8 * ds, (use + 1) & 1, gave_up, p.timeout))) break;
                const u32 d = tmem + ds * D_COLS;
                const int here = min(2, chunks - 2 * kb);
                for (int c = 0; c < here && ok; ++c) {
                    const u32 r = 2 * kb + c, slot = r % A_SLOTS;
                    if (!(ok = warp_wait(full + 8 * slot, (r / A_SLOTS) & 1, gave_up, p.timeout))) break;
#pragma unroll
                    for (int s = 0; s < 2; ++s)
                        mma_small(d, tmem + A_COL + slot * A_SLOT_COLS + 8 * s, b0 + (slot >> 1) * stage + (slot & 1) * 64 + 32 * s, term,
                                  idesc, c + s > 0);
                }
                if (!ok) break;
                for (int c = 0; c < here; ++c) {
                    const u32 slot = (2 * kb + c) % A_SLOTS;
#pragma unroll
                    for (int s = 0; s < 2; ++s)
                        mma(d, tmem + A_COL + slot * A_SLOT_COLS + 8 * s, desc_of(b0 + (slot >> 1) * stage + (slot & 1) * 64 + 32 * s), idesc, true);
                    commit(empty + 8 * slot);
                }
                commit(d_full + 8 * ds);
            }
            if (!ok) {  // the MMAs under way end before the block frees its tensor memory
                commit(drained);
                for (u32 spins = 0; spins < (1u << 20) && !bar_poll(drained, 0); ++spins) {
                }
                __syncwarp();
            }
            goto done;
        }
        // Task i of a chunk: 64 columns by 8 rows, of the (bn / 64) x 4 of them.  The warps take the tasks of all chunks in
        // turn, the next one's loads under way.  A lane has
        // columns 2 lane and 2 lane + 1 of the 64 and puts them into rows lane and lane + 32 of the operand tile, so
        // that its 16-byte stores fall into different banks; the sums' columns are put straight on the way out.
        const int lg = p.bn == 64 ? 2 : 3, tasks = chunks << lg;
        float2 v[2][8];
        auto load = [&](int buf, int t) {
            const int task = t & ((1 << lg) - 1);
            const int col = n0 + (task >> 2) * 64 + 2 * lane, r0 = (first + (t >> lg)) * CHUNK_K + (task & 3) * 8;
            const int c0 = min(col, (p.n - 1) & ~1), step = c0 + 1 < p.n ? 1 : 0;
            const float* at = p.b + (int64_t)r0 * p.ldb + c0;
            if (r0 + 8 <= p.rows && p.b_vec) {
#pragma unroll
                for (int j = 0; j < 8; ++j, at += p.ldb) v[buf][j] = fetch_pair(at);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j, at += p.ldb)
                    v[buf][j] = make_float2(fetch1(at, r0 + j < p.rows), fetch1(at + step, r0 + j < p.rows));
            }
        };
        int t = warp - A_WARPS;
        if (t < tasks) load(0, t);
        while (t < tasks) {
#pragma unroll
            for (int buf = 0; buf < 2; ++buf) {
                if (t >= tasks) break;
                if (t + B_WARPS < tasks) load(buf ^ 1, t + B_WARPS);
                const int c = t >> lg, task = t & ((1 << lg) - 1);
                const u32 slot = (u32)c % A_SLOTS;
                if (c >= A_SLOTS && !warp_wait(empty + 8 * slot, ((u32)c / A_SLOTS + 1) & 1, gave_up, p.timeout)) goto done;
                unsigned char* at = smem + (slot >> 1) * stage;
                const u32 row = (u32)((task >> 2) * 64 + lane), k8 = (slot & 1) * 4 + (u32)(task & 3);
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = p.relu_b ? relu(v[buf][j].x) : v[buf][j].x;
                store_split8(at + swizzled(row, k8), term, x);
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = p.relu_b ? relu(v[buf][j].y) : v[buf][j].y;
                store_split8(at + swizzled(row + 32, k8), term, x);
                fence_async();
                __syncwarp();
                if (lane == 0) bar_arrive(full + 8 * slot);
                t += B_WARPS;
            }
        }
    } else {
        // lane = row of the tile; accumulator column 32 j + i of this warp's 64 is column 2 i + j of the result
        const int quarter = warp & 3, c_lo = 64 * ((warp - FIRST_SUM_WARP) >> 2);
        float acc[2][32];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[j][i] = 0.f;
        for (int kb = 0; kb < kblocks; ++kb) {
            const u32 ds = kb & 1, use = kb >> 1;
            if (!warp_wait(d_full + 8 * ds, use & 1, gave_up, p.timeout)) goto done;
            if (c_lo < p.bn) {
                const u32 at = tmem + ds * D_COLS + c_lo + ((u32)(quarter * 32) << 16);
#pragma unroll
                for (int g = 0; g < 4; ++g) {  // 16 columns at a time
                    float r[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
                        "%15}, [%16];"
                        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                          "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                        : "r"(at + 16 * g));
                    wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        asm volatile("" : "+f"(r[i]));  // not before the wait
                        acc[g >> 1][16 * (g & 1) + i] += r[i];
                    }
                }
                fence_before();
            }
            __syncwarp();
            if (lane == 0) bar_arrive(d_empty + 8 * ds);
        }
        const int row = m0 + quarter * 32 + lane;
        if (row < p.m && c_lo < p.bn) {
            float* out = p.part + ((int64_t)blockIdx.y * p.m + row) * p.n + n0 + c_lo;
            const bool vec = p.n % 4 == 0;  // (n0 and the workspace are aligned)
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const int left = p.n - (n0 + c_lo + 2 * i);
                float* d = out + 2 * i;
                if (vec && left >= 4) {
                    *reinterpret_cast<float4*>(d) = make_float4(acc[0][i], acc[1][i], acc[0][i + 1], acc[1][i + 1]);
                } else {
                    if (left > 0) d[0] = acc[0][i];
                    if (left > 1) d[1] = acc[1][i];
                    if (left > 2) d[2] = acc[0][i + 1];
                    if (left > 3) d[3] = acc[1][i + 1];
                }
            }
        }
    }
done:
    __syncwarp();
    fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_free(tmem);
}

// out = sum of `parts` partial results [m, n], in a fixed order: 8 threads of a block add every eighth part of an
// element, the 8 sums are added in turn.  `turn`: out is [n, m].
__global__ void __launch_bounds__(256) reduce_parts_kernel(const float* part, int parts, int m, int n, float* out, int64_t ldo, int turn) {
    cbm::wait_before();
    __shared__ float s[8][32];
    const int64_t size = (int64_t)m * n, i = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const int g = threadIdx.x >> 5;
    float sum = 0.f;
    if (i < size) {
        int q = g;
        for (; q + 24 < parts; q += 32) {
            const float x0 = __ldcs(part + q * size + i), x1 = __ldcs(part + (q + 8) * size + i);
            const float x2 = __ldcs(part + (q + 16) * size + i), x3 = __ldcs(part + (q + 24) * size + i);
            sum += x0;
            sum += x1;
            sum += x2;
            sum += x3;
        }
        for (; q < parts; q += 8) sum += __ldcs(part + q * size + i);
    }
    s[g][threadIdx.x & 31] = sum;
    __syncthreads();
    if (g == 0 && i < size) {
#pragma unroll
        for (int k = 1; k < 8; ++k) sum += s[k][threadIdx.x];
        const int64_t r = i / n, c = i - r * n;
        out[turn ? c * ldo + r : r * ldo + c] = sum;
    }
}

// How the contraction is cut: orientation, tiles of the result, row ranges.
struct Split {
    bool turn;  // dW^T (M = in, N = out) instead of dW (M = out, N = in)
    int m_tiles, n_tiles, bn;
    int chunks_per, ranges;
};

Split split_of(int n_rows, int n_in, int n_out) {
    const auto tiling = [](int m, int n, Split& t) {
        t.m_tiles = (m + 127) / 128;
        t.n_tiles = (n + 127) / 128;
        t.bn = (n + t.n_tiles - 1) / t.n_tiles <= 64 ? 64 : 128;
        return (int64_t)t.n_tiles * m + (int64_t)t.m_tiles * n;  // columns read by all tiles of one row range
    };
    // the orientation that reads fewer operand columns, then the one that wastes fewer tile columns
    Split plain{}, turned{};
    const int64_t reads = tiling(n_out, n_in, plain), turned_reads = tiling(n_in, n_out, turned);
    turned.turn = true;
    Split t = turned_reads < reads || (turned_reads == reads && turned.bn * turned.m_tiles * turned.n_tiles <
                                                                    plain.bn * plain.m_tiles * plain.n_tiles)
                  ? turned
                  : plain;
    // one wave of blocks, each with at least four chunks to itself
    const int total = (int)(((int64_t)n_rows + CHUNK_K - 1) / CHUNK_K);
    const int parts = std::max(1, std::min({sm_count() / (t.m_tiles * t.n_tiles), (total + 3) / 4, MAX_PARTS}));
    t.chunks_per = std::max(2, ((total + parts - 1) / parts + 1) / 2 * 2);
    t.ranges = std::max(1, (total + t.chunks_per - 1) / t.chunks_per);
    return t;
}

}  // namespace
}  // namespace cbm_map

using namespace cbm_map;

extern "C" int64_t cbm_b200_dense_grad_weight_workspace(int32_t n_rows, int32_t n_in, int32_t n_out) {
    return (int64_t)split_of(n_rows, n_in, n_out).ranges * n_in * n_out * (int64_t)sizeof(float);
}

namespace {
int run_grad(const float* dy, int64_t lddy, const float* x, int64_t ldx, float* dw, int64_t lddw, int32_t n_rows, int32_t n_in,
             int32_t n_out, bool relu_x, void* workspace, int64_t workspace_bytes, void* stream) {
    if (!dy || !x || !dw || n_rows < 0 || n_in <= 0 || n_out <= 0)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_grad_weight: bad arguments");
    if (lddy < n_out || ldx < n_in || lddw < n_in)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_grad_weight: a leading dimension is smaller than its row");
    if (const int rc = check_timeout("dense_grad_weight")) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const Split t = split_of(n_rows, n_in, n_out);
    const int64_t need = (int64_t)t.ranges * n_in * n_out * (int64_t)sizeof(float);
    if (!workspace || workspace_bytes < need)
        return cbm::fail(CBM_B200_ERR_ARG, "dense_grad_weight: workspace of " + std::to_string(need) + " bytes needed");
    GradParams p{};
    p.a = t.turn ? x : dy;
    p.b = t.turn ? dy : x;
    p.lda = t.turn ? ldx : lddy;
    p.ldb = t.turn ? lddy : ldx;
    p.rows = n_rows;
    p.m = t.turn ? n_in : n_out;
    p.n = t.turn ? n_out : n_in;
    p.bn = t.bn;
    p.n_tiles = t.n_tiles;
    p.chunks_per = t.chunks_per;
    p.relu_a = t.turn && relu_x;
    p.relu_b = !t.turn && relu_x;
    p.b_vec = (reinterpret_cast<uintptr_t>(p.b) & 7) == 0 && p.ldb % 2 == 0;
    p.part = static_cast<float*>(workspace);
    p.timeout = timeout_word();
    // at least half of an SM's shared memory, so that two blocks, which both want all tensor memory, never share one
    const int smem = 120 * 1024;
    static_assert(2 * 3 * D_COLS * 128 + 1024 <= 120 * 1024, "two stages of B");
    if (!allow_smem<grad_kernel>(smem))
        return cbm::fail(CBM_B200_ERR_CUDA, "dense_grad_weight: shared memory size refused");
    cbm::launch_next(grad_kernel, dim3(t.m_tiles * t.n_tiles, t.ranges), GRAD_THREADS, smem, s, p);
    const int64_t size = (int64_t)n_in * n_out;
    cbm::launch_next(reduce_parts_kernel, (unsigned)((size + 31) / 32), 256, 0, s, p.part, t.ranges, p.m, p.n, dw, lddw, t.turn ? 1 : 0);
    if (cudaGetLastError() != cudaSuccess) return cbm::fail(CBM_B200_ERR_CUDA, "dense_grad_weight: launch failed");
    return CBM_B200_OK;
}
}  // namespace

extern "C" int cbm_b200_dense_grad_weight(const float* dy, int64_t lddy, const float* x, int64_t ldx, float* dw,
                                          int64_t lddw, int32_t n_rows, int32_t n_in, int32_t n_out, void* workspace,
                                          int64_t workspace_bytes, void* stream) {
    return run_grad(dy, lddy, x, ldx, dw, lddw, n_rows, n_in, n_out, false, workspace, workspace_bytes, stream);
}

extern "C" int cbm_b200_dense_grad_weight_of_relu(const float* dy, int64_t lddy, const float* x, int64_t ldx, float* dw,
                                                  int64_t lddw, int32_t n_rows, int32_t n_in, int32_t n_out,
                                                  void* workspace, int64_t workspace_bytes, void* stream) {
    return run_grad(dy, lddy, x, ldx, dw, lddw, n_rows, n_in, n_out, true, workspace, workspace_bytes, stream);
}
