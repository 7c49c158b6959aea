// Communities of rows by label propagation, for the order in which a plan works on its rows.
//
// Graphs with communities name, within one community, the same few columns over and over; but node
// numbers seldom follow communities, so rows in node order find nothing of one another in an SM's L1.
// Every row repeatedly takes the label that is most frequent among (up to 31 of) its columns.  One
// warp per row: one column per lane, and __match_any_sync counts the lanes that hold the same label.
// Half of the rows move in each round, so that two rows cannot swap labels for ever.  A round reads the labels of the
// round before from one array and writes its own to another: plans of one graph are the same.  A round over
// 400 000 rows of 22 entries is bound by the 9 M label fetches from L2 (well under 0.1 ms); bringing the
// pattern to the GPU takes longer than all rounds.
#include "cbm_cluster.h"

#include <cuda_runtime.h>

#include <utility>

namespace {

constexpr int ROUNDS = 12;

// The integer hash "lowbias32" (Chris Wellons, Hash Function Prospector).
__device__ __forceinline__ unsigned mix(unsigned v) {
    v ^= v >> 16;
    v *= 0x7feb352du;
    v ^= v >> 15;
    v *= 0x846ca68bu;
    return v ^ (v >> 16);
}

__global__ void __launch_bounds__(256) init_labels_kernel(int32_t n, int32_t* label) {
    const int32_t v = blockIdx.x * 256 + threadIdx.x;
    if (v < n) label[v] = v;
}

__global__ void __launch_bounds__(256) propagate_kernel(int32_t n, const int32_t* __restrict__ crow,
                                                        const int32_t* __restrict__ col, const int32_t* __restrict__ parent,
                                                        const int32_t* __restrict__ label, int32_t* __restrict__ next_label,
                                                        int round) {
    const int32_t v = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (v >= n) return;
    const int32_t mine = label[v];
    if (((mix((unsigned)v) + (unsigned)round) & 1u) != 0) {
        if (lane == 0) next_label[v] = mine;
        return;
    }
    const int32_t beg = crow[v], len = crow[v + 1] - beg;
    const int32_t par = parent[v];
    // the last lane looks at the parent: what a row shares with its parent is not among its delta columns
    const int32_t have = min(31, len);
    int32_t u = -1;
    if (lane < have) u = col[beg + (len <= 31 ? lane : (int32_t)((int64_t)lane * len / 31))];
    else if (lane == 31) u = par;
    const int32_t l = u >= 0 && u < n && u != v ? __ldg(label + u) : -1 - lane;  // lanes without a row match nobody
    const unsigned same = __match_any_sync(0xffffffffu, l);
    // most frequent label; the row's own wins ties, then an arbitrary but fixed order of the labels
    const unsigned score =
        l < 0 ? 0u : ((unsigned)__popc(same) << 9) | (l == mine ? 256u : 0u) | (mix((unsigned)l) & 255u);
    const unsigned best = __reduce_max_sync(0xffffffffu, score);
    const int from = __ffs(__ballot_sync(0xffffffffu, score == best)) - 1;
    const int32_t next = __shfl_sync(0xffffffffu, l, from);
    if (lane == 0) next_label[v] = best == 0 ? mine : next;
}

struct Buffers {
    int32_t *crow = nullptr, *col = nullptr, *parent = nullptr, *label = nullptr, *other = nullptr;
    ~Buffers() {
        cudaFree(crow);
        cudaFree(col);
        cudaFree(parent);
        cudaFree(label);
        cudaFree(other);
    }
};

}  // namespace

bool cbm::cluster_rows(int32_t n, const int32_t* crow, const int32_t* col, const int32_t* parent, int device,
                       int32_t* label) {
    int prev = 0;
    if (n <= 0 || cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return false;
    bool ok = false;
    {
        Buffers b;
        const size_t rows = (size_t)n * sizeof(int32_t), entries = (size_t)crow[n] * sizeof(int32_t);
        if (cudaMalloc((void**)&b.crow, rows + sizeof(int32_t)) == cudaSuccess &&
            cudaMalloc((void**)&b.col, entries + sizeof(int32_t)) == cudaSuccess &&
            cudaMalloc((void**)&b.parent, rows) == cudaSuccess && cudaMalloc((void**)&b.label, rows) == cudaSuccess &&
            cudaMalloc((void**)&b.other, rows) == cudaSuccess &&
            cudaMemcpy(b.crow, crow, rows + sizeof(int32_t), cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(b.col, col, entries, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(b.parent, parent, rows, cudaMemcpyHostToDevice) == cudaSuccess) {
            init_labels_kernel<<<(n + 255) / 256, 256>>>(n, b.label);
            for (int r = 0; r < ROUNDS; ++r) {
                propagate_kernel<<<(n + 7) / 8, 256>>>(n, b.crow, b.col, b.parent, b.label, b.other, r);
                std::swap(b.label, b.other);
            }
            ok = cudaGetLastError() == cudaSuccess &&
                 cudaMemcpy(label, b.label, rows, cudaMemcpyDeviceToHost) == cudaSuccess;
            for (int32_t v = 0; ok && v < n; ++v) ok = label[v] >= 0 && label[v] < n;  // the caller counts by them
        }
        if (!ok) cudaGetLastError();
    }
    cudaSetDevice(prev);
    return ok;
}
