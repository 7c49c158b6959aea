// Candidate search of the CBM builder on the GPU.
//
// The builder's first step finds, for every row u, the rows v that share more than (|u| + alpha) / 2
// columns with it (the candidate rule of cbm/cbm_extensions.cpp:75-102, which the reference evaluates
// on all of A * A^T).  The host search (cbm_builder.cpp) walks, for every u, the column lists of u's
// rarest columns and counts hits per row; on a high-degree graph that is billions of random counter
// increments and 97 % of the build.  Here the same filter runs with one thread block per parent
// row: warps stream the column lists of the prefix and count with atomics into a per-block array of
// 16-bit counters that stays in L2, rows that reach the required number of hits get their exact
// intersection from a bitmap of u's columns, and survivors of the rule are appended to one output
// list.  The filter is lossless (see cbm_builder.cpp), so the set of candidates — and with it the
// structure the builder emits — is identical to the host search's; only the order of the output
// differs, and the caller sorts it.
//
// What the search reads - the columns in order of frequency, each row's columns in that order, each column's rows - is
// made here too, from the pattern alone: counts by atomics, places by a scan, rows put in order by a warp, a block or, where
// they are long, through a bitmap.  Which of two equally frequent columns comes first, and in which order a column's rows
// stand, is left to chance: the set of candidates does not depend on it.  100 000 rows, 3.1 M entries: the transposed
// pattern, the order of the columns and the sorted rows took 16 threads 15 ms of a build of 23; the whole build is 15 ms now.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "cbm_candidates.h"

namespace {

using i32 = int32_t;
using i64 = int64_t;
using u32 = uint32_t;
using u64 = unsigned long long;

struct SearchParams {
    i32 n, alpha;
    const i64* row_ptr;   // rows of the pattern, columns replaced by their rank (rare = small), ascending
    const i32* row_rank;
    const i64* col_ptr;   // each column's rows, by its rank
    const i32* col_rows;
    u32* hits;            // per block: (n + 1) / 2 words, two 16-bit counters each
    i32* touched;         // per block: n entries
    u32* bitmap;          // per block: (n + 31) / 32 words, bit per rank id
    i64 hits_stride, touched_stride, bitmap_stride;
    cbm::CandTriple* out;
    u64* out_count;       // [0] entries appended, [1] next parent row to claim
    i64 out_cap;
    i32* skipped;         // parents left to the host (prefix too long for 16-bit counters)
    i32* n_skipped;
    i32* large;           // parents whose prefix lists more rows than a warp's table takes
    i32* n_large;
    i32 n_blocks_of;      // parents in `large`, for the block's search
};

constexpr int kThreads = 512;
constexpr int kMaxPrefix = 65000;

// Shared columns that an edge u -> v needs, and the prefix of u's columns that guarantees `hits` of them.  More hits make
// a longer prefix to count and leave fewer rows to intersect, the candidates are the same: 100 000 copy-model rows of 31
// entries list 978 rows each with at least 8 hits and 640 with 4, and 0.4 and 2 of them pass; from 64 shared columns
// on an eighth of them measured best.
struct Need {
    i32 need, hits, prefix;
    bool none;  // no row can have that many
};
__device__ __forceinline__ Need need_of(i32 nu, i32 alpha) {
    const i64 sum = (i64)nu + alpha;
    const i64 half_floor = sum >= 0 ? sum / 2 : -((-sum + 1) / 2);
    const i64 need64 = max(half_floor + 1, (i64)1);
    Need r;
    r.none = need64 > nu;
    r.need = (i32)min(need64, (i64)INT32_MAX);
    r.hits = min(r.need, max(4, min(32, r.need / 8)));
    r.prefix = nu - r.need + r.hits;
    return r;
}

// The search for a parent whose prefix lists few rows, by one warp: the rows are counted in a table in shared memory.  A
// block to a parent spends its time between barriers there: 100 000 rows of 31 entries 2.5 ms, 1.1 for the nine tenths of them
// that go here and 0.6 for the others, which are put on a list.
constexpr int TABLE_BITS = 10, TABLE = 1 << TABLE_BITS, TABLE_TAKES = 704, TABLE_WARPS = 8;
constexpr int TABLE_BYTES = TABLE * 4 + TABLE * 2;  // a row and a 16-bit count each

__global__ void __launch_bounds__(TABLE_WARPS * 32) candidate_warp_kernel(const SearchParams p) {
    constexpr int EACH = 4;
    extern __shared__ i32 s_table[];
    const int lane = threadIdx.x & 31;
    i32* key = s_table + (threadIdx.x >> 5) * (TABLE_BYTES / 4);  // -1: free
    u32* count = reinterpret_cast<u32*>(key + TABLE);             // two to a word
    for (int i = lane; i < TABLE; i += 32) key[i] = -1;
    for (int i = lane; i < TABLE / 2; i += 32) count[i] = 0;
    __syncwarp();
    for (;;) {
        i32 u = 0;
        if (lane == 0) u = (i32)min((u64)p.n, atomicAdd(p.out_count + 1, 1ULL));
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= p.n) return;
        const i64 ub = p.row_ptr[u];
        const i32 nu = (i32)(p.row_ptr[u + 1] - ub);
        const Need want = need_of(nu, p.alpha);
        if (want.none) continue;
        i64 listed = 0;
        for (i32 i = lane; i < want.prefix && listed <= TABLE_TAKES; i += 32) {
            const i32 c = p.row_rank[ub + i];
            listed += p.col_ptr[c + 1] - p.col_ptr[c];
        }
        for (int d = 16; d; d >>= 1) listed += __shfl_xor_sync(0xffffffffu, listed, d);
        if (listed > TABLE_TAKES) {
            if (lane == 0) p.large[atomicAdd(p.n_large, 1)] = u;
            continue;
        }
        // 32 lists at a time, end to end: lane k holds where the k-th begins and how much lies before it
        for (i32 i0 = 0; i0 < want.prefix; i0 += 32) {
            i64 qb = 0;
            i32 len = 0;
            if (i0 + lane < want.prefix) {
                const i32 c = p.row_rank[ub + i0 + lane];
                qb = p.col_ptr[c];
                len = (i32)(p.col_ptr[c + 1] - qb);
            }
            i32 upto = len;
            for (int d = 1; d < 32; d <<= 1) {
                const i32 up = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += up;
            }
            const i32 total = __shfl_sync(0xffffffffu, upto, 31);
            for (i32 t0 = 0; t0 < total; t0 += 32 * EACH) {
                i32 v[EACH];
#pragma unroll
                for (int e = 0; e < EACH; ++e) {  // all fetches before the first count
                    const i32 t = t0 + 32 * e + lane;
                    int k = 0;  // lists that end at or before t
#pragma unroll
                    for (int d = 16; d; d >>= 1)
                        if (__shfl_sync(0xffffffffu, upto, k + d - 1) <= t) k += d;
                    const i64 b = __shfl_sync(0xffffffffu, qb, k);
                    const i32 before = __shfl_sync(0xffffffffu, upto - len, k);
                    v[e] = t < total ? __ldg(p.col_rows + b + (t - before)) : -1;
                }
#pragma unroll
                for (int e = 0; e < EACH; ++e) {
                    if (v[e] < 0) continue;
                    unsigned h = ((unsigned)v[e] * 2654435761u) >> (32 - TABLE_BITS);
                    for (;;) {  // (there are free places)
                        const i32 was = atomicCAS(key + h, -1, v[e]);
                        if (was == -1 || was == v[e]) break;
                        h = (h + 1) & (TABLE - 1);
                    }
                    atomicAdd(count + (h >> 1), (h & 1) ? 0x10000u : 1u);
                }
            }
        }
        __syncwarp();
        const bool has_tail = want.prefix < nu;
        for (int i = lane; i < TABLE; i += 32) {
            const i32 mine = key[i], hits = (i32)((count[i >> 1] >> (16 * (i & 1))) & 0xffffu);
            __syncwarp();  // (two lanes share a word of counts)
            key[i] = -1;
            if ((i & 1) == 0) count[i >> 1] = 0;
            bool pass = mine >= 0 && mine != u && hits >= want.hits;
            pass = pass && p.row_ptr[mine + 1] - p.row_ptr[mine] >= want.need;
            for (unsigned m = __ballot_sync(0xffffffffu, pass); m; m &= m - 1) {
                const int from = __ffs(m) - 1;
                const i32 v = __shfl_sync(0xffffffffu, mine, from);
                i32 both = __shfl_sync(0xffffffffu, hits, from);
                const i64 vb = p.row_ptr[v];
                const i32 nv = (i32)(p.row_ptr[v + 1] - vb);
                if (has_tail) {  // the whole intersection: each of v's columns is looked for among u's
                    i32 found = 0;
                    for (i32 k = lane; k < nv; k += 32) {
                        const i32 r = p.row_rank[vb + k];
                        i32 lo = 0, hi = nu;
                        while (lo < hi) {
                            const i32 mid = (lo + hi) >> 1;
                            if (p.row_rank[ub + mid] < r) lo = mid + 1;
                            else hi = mid;
                        }
                        found += lo < nu && p.row_rank[ub + lo] == r;
                    }
                    both = (i32)__reduce_add_sync(0xffffffffu, (unsigned)found);
                }
                const i32 h = nu + nv - 2 * both;
                if (h < nv - p.alpha && lane == 0) {  // cbm/cbm_extensions.cpp:93-101
                    const u64 pos = atomicAdd(p.out_count, 1ULL);
                    if ((i64)pos < p.out_cap) p.out[pos] = cbm::CandTriple{u, v, h};
                }
            }
        }
        __syncwarp();
    }
}

// The search for the parents on the list, a block to each.
__global__ void __launch_bounds__(kThreads) candidate_kernel(const SearchParams p) {
    __shared__ i32 s_u, s_touched, s_passed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = kThreads / 32;
    u32* hits = p.hits + (i64)blockIdx.x * p.hits_stride;
    i32* touched = p.touched + (i64)blockIdx.x * p.touched_stride;
    u32* bitmap = p.bitmap + (i64)blockIdx.x * p.bitmap_stride;
    for (;;) {
        if (tid == 0) {
            const u64 t = atomicAdd(p.out_count + 1, 1ULL);
            s_u = t < (u64)p.n_blocks_of ? p.large[t] : -1;
            s_touched = s_passed = 0;
        }
        __syncthreads();
        const i32 u = s_u;
        if (u < 0) return;
        const i64 ub = p.row_ptr[u];
        const i32 nu = (i32)(p.row_ptr[u + 1] - ub);
        const Need want = need_of(nu, p.alpha);
        const i32 need = want.need, j_hits = want.hits, plen = want.prefix;
        bool skip = want.none;
        if (!skip && plen > kMaxPrefix) {
            if (tid == 0) p.skipped[atomicAdd(p.n_skipped, 1)] = u;
            skip = true;
        }
        if (skip) {
            __syncthreads();
            continue;
        }
        // 1. count hits of every row through the column lists of the prefix
        for (i32 i = warp; i < plen; i += n_warps) {
            const i32 c = p.row_rank[ub + i];
            const i64 qb = p.col_ptr[c], qe = p.col_ptr[c + 1];
            for (i64 q = qb + lane; q < qe; q += 32) {
                const i32 v = p.col_rows[q];
                const u32 old = atomicAdd(hits + (v >> 1), (v & 1) ? 0x10000u : 1u);
                if ((((v & 1) ? (old >> 16) : old) & 0xffffu) == 0) touched[atomicAdd(&s_touched, 1)] = v;
            }
        }
        const bool has_tail = plen < nu;
        if (has_tail)
            for (i32 i = tid; i < nu; i += kThreads) {
                const i32 r = p.row_rank[ub + i];
                atomicOr(bitmap + (r >> 5), 1u << (r & 31));
            }
        __syncthreads();
        // 2. rows with enough hits in the prefix: exact intersection, then the rule
        const i32 n_touched = s_touched;
        // Every lane looks at one touched row: nearly all fall at the number of hits, and a warp that took them one by
        // one spent its time waiting for that counter (100 000 rows: 7.8 ms the whole search, 2.5 so).  Those that
        // pass are gathered at the front of the list and dealt out to the warps one at a time: where many pass, a
        // warp that dealt with its own 32 kept the block waiting (132 534 rows of 265 entries: 2.6 s, 0.93 so).
        for (i32 t0 = 0; t0 < n_touched; t0 += kThreads) {
            i32 v = u;
            bool pass = false;
            if (t0 + tid < n_touched) {
                v = touched[t0 + tid];
                const u32 mine = (v & 1) ? 0xffff0000u : 0x0000ffffu;
                const i32 in_prefix = (i32)((__ldcg(hits + (v >> 1)) & mine) >> ((v & 1) * 16));
                pass = v != u && in_prefix >= j_hits && p.row_ptr[v + 1] - p.row_ptr[v] >= need;
                if (!pass) atomicAnd(hits + (v >> 1), ~mine);
            }
            __syncthreads();  // all of this stretch is read: the list may grow into it
            if (pass) touched[atomicAdd(&s_passed, 1)] = v;
        }
        __syncthreads();
        const i32 n_passed = s_passed;
        for (i32 t = warp; t < n_passed; t += n_warps) {
            const i32 v = touched[t];
            i32 both = 0;
            if (lane == 0) {
                const u32 w = atomicAnd(hits + (v >> 1), (v & 1) ? 0x0000ffffu : 0xffff0000u);  // read and clear
                both = (i32)(((v & 1) ? (w >> 16) : w) & 0xffffu);
            }
            both = __shfl_sync(0xffffffffu, both, 0);
            const i64 vb = p.row_ptr[v];
            const i32 nv = (i32)(p.row_ptr[v + 1] - vb);
            if (has_tail) {
                i32 cnt = 0;
                for (i32 k = lane; k < nv; k += 32) {
                    const i32 r = p.row_rank[vb + k];
                    cnt += (i32)((bitmap[r >> 5] >> (r & 31)) & 1u);
                }
                both = (i32)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
            }
            const i32 h = nu + nv - 2 * both;
            if (h < nv - p.alpha && lane == 0) {  // cbm/cbm_extensions.cpp:93-101
                const u64 pos = atomicAdd(p.out_count, 1ULL);
                if ((i64)pos < p.out_cap) p.out[pos] = cbm::CandTriple{u, v, h};
            }
        }
        __syncthreads();
        if (has_tail)
            for (i32 i = tid; i < nu; i += kThreads) bitmap[p.row_rank[ub + i] >> 5] = 0;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- what the search reads, from the pattern
__global__ void __launch_bounds__(256) count_columns_kernel(i64 nnz, const i32* __restrict__ col, i32* __restrict__ count) {
    for (i64 i = (i64)blockIdx.x * 256 + threadIdx.x; i < nnz; i += (i64)gridDim.x * 256) atomicAdd(count + col[i], 1);
}

// How many columns occur how often.
__global__ void __launch_bounds__(256) count_counts_kernel(i32 n, const i32* __restrict__ count, i32* __restrict__ often) {
    const i32 c = blockIdx.x * 256 + threadIdx.x;
    if (c < n) atomicAdd(often + count[c], 1);
}

// Exclusive sums: a block takes SCAN_TILE values, adds them up here and hands its total on, one block adds up the totals,
// and the third kernel adds them to the tiles.
constexpr int SCAN_THREADS = 256, SCAN_EACH = 8, SCAN_TILE = SCAN_THREADS * SCAN_EACH;

// The exclusive sum of `mine` over the block's threads, and the block's total.
__device__ __forceinline__ i64 block_scan(i64 mine, i64* s_warp, i64& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    i64 sum = mine;
    for (int d = 1; d < 32; d <<= 1) {
        const i64 up = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += up;
    }
    __syncthreads();  // (s_warp may still be read from the round before)
    if (lane == 31) s_warp[warp] = sum;
    __syncthreads();
    i64 before = 0;
    total = 0;
    for (int w = 0; w < warps; ++w) {
        if (w < warp) before += s_warp[w];
        total += s_warp[w];
    }
    return before + sum - mine;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_tiles_kernel(i64 n, const i32* __restrict__ in, i64* __restrict__ out,
                                                                  i64* __restrict__ totals) {
    __shared__ i64 s_warp[SCAN_THREADS / 32];
    const i64 first = (i64)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_EACH;
    i64 v[SCAN_EACH], mine = 0, total;
    for (int k = 0; k < SCAN_EACH; ++k) {
        v[k] = mine;
        if (first + k < n) mine += in[first + k];
    }
    const i64 before = block_scan(mine, s_warp, total);
    for (int k = 0; k < SCAN_EACH; ++k)
        if (first + k < n) out[first + k] = before + v[k];
    if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_totals_kernel(i32 tiles, i64* totals) {
    __shared__ i64 s_warp[SCAN_THREADS / 32];
    i64 before = 0;
    for (i32 t = 0; t < tiles; t += SCAN_THREADS) {
        const i32 i = t + (i32)threadIdx.x;
        i64 total;
        const i64 sum = block_scan(i < tiles ? totals[i] : 0, s_warp, total);
        if (i < tiles) totals[i] = before + sum;
        before += total;
    }
}

// out[n] receives the sum of all.
__global__ void __launch_bounds__(256) scan_add_kernel(i64 n, const i32* __restrict__ in, i64* __restrict__ out,
                                                       const i64* __restrict__ totals) {
    const i64 i = (i64)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const i64 sum = out[i] + totals[i / SCAN_TILE];
    out[i] = sum;
    if (i == n - 1) out[n] = sum + in[i];
}

// Ranks of the columns, rare ones first, and their counts in that order; `taken` is zero before.
__global__ void __launch_bounds__(256) rank_columns_kernel(i32 n, const i32* __restrict__ count, const i64* __restrict__ first,
                                                           i32* __restrict__ taken, i32* __restrict__ rank,
                                                           i32* __restrict__ count_of_rank) {
    const i32 c = blockIdx.x * 256 + threadIdx.x;
    if (c >= n) return;
    const i32 r = (i32)first[count[c]] + atomicAdd(taken + count[c], 1);
    rank[c] = r;
    count_of_rank[r] = count[c];
}

// A warp to a row: its columns become ranks, and the row enters their lists; `taken` is zero before.
__global__ void __launch_bounds__(256) list_rows_kernel(i32 n, const i64* __restrict__ row_ptr, i32* __restrict__ row_rank,
                                                        const i32* __restrict__ rank, const i64* __restrict__ col_ptr,
                                                        i32* __restrict__ taken, i32* __restrict__ col_rows) {
    const i32 u = (i32)(((i64)blockIdx.x * 256 + threadIdx.x) >> 5);
    if (u >= n) return;
    for (i64 k = row_ptr[u] + (threadIdx.x & 31); k < row_ptr[u + 1]; k += 32) {
        const i32 r = rank[row_rank[k]];
        row_rank[k] = r;
        col_rows[col_ptr[r] + atomicAdd(taken + r, 1)] = u;
    }
}

// Bitonic sort of s[0, size), a power of two, by `threads` threads that call sync() between the steps.
template <class Sync>
__device__ __forceinline__ void bitonic(i32* s, int size, int me, int threads, Sync sync) {
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            sync();
            for (int t = me; t < size / 2; t += threads) {
                const int a = 2 * t - (t & (j - 1)), b = a + j;
                const i32 x = s[a], y = s[b];
                if ((x > y) == ((a & k) == 0)) {
                    s[a] = y;
                    s[b] = x;
                }
            }
        }
    sync();
}

constexpr int WARP_ROW = 256, BLOCK_ROW = 4096;  // longest rows that a warp and a block sort in shared memory

__global__ void __launch_bounds__(256) sort_rows_warp_kernel(i32 n, const i64* __restrict__ row_ptr, i32* __restrict__ row_rank) {
    __shared__ i32 s_all[8][WARP_ROW];
    const int lane = threadIdx.x & 31;
    const i32 u = (i32)(((i64)blockIdx.x * 256 + threadIdx.x) >> 5);
    if (u >= n) return;
    const i64 b = row_ptr[u], len = row_ptr[u + 1] - b;
    if (len < 2 || len > WARP_ROW) return;
    if (len <= 32) {
        i32 x = lane < len ? row_rank[b + lane] : INT32_MAX;
        for (int k = 2; k <= 32; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                const i32 y = __shfl_xor_sync(0xffffffffu, x, j);
                const bool low = (lane & j) == 0, up = (lane & k) == 0;
                x = low == up ? min(x, y) : max(x, y);
            }
        if (lane < len) row_rank[b + lane] = x;
        return;
    }
    i32* s = s_all[threadIdx.x >> 5];
    const int size = 1 << (32 - __clz((int)len - 1));
    for (int i = lane; i < size; i += 32) s[i] = i < len ? row_rank[b + i] : INT32_MAX;
    bitonic(s, size, lane, 32, [] { __syncwarp(); });
    for (int i = lane; i < len; i += 32) row_rank[b + i] = s[i];
}

// The rows that no warp takes: up to BLOCK_ROW entries in shared memory, longer ones by the block's bitmap, whose bits
// are read off in order.  Bitmaps are zero before and after.
__global__ void __launch_bounds__(512) sort_rows_block_kernel(i32 n, const i64* __restrict__ row_ptr, i32* __restrict__ row_rank,
                                                              u32* bitmaps, i64 bitmap_stride) {
    __shared__ i32 s[BLOCK_ROW];
    __shared__ i64 s_warp[512 / 32];
    u32* bitmap = bitmaps + (i64)blockIdx.x * bitmap_stride;
    for (i32 u = blockIdx.x; u < n; u += gridDim.x) {
        const i64 b = row_ptr[u], len = row_ptr[u + 1] - b;
        if (len <= WARP_ROW) continue;
        if (len <= BLOCK_ROW) {
            const int size = 1 << (32 - __clz((int)len - 1));
            __syncthreads();
            for (int i = threadIdx.x; i < size; i += 512) s[i] = i < len ? row_rank[b + i] : INT32_MAX;
            bitonic(s, size, threadIdx.x, 512, [] { __syncthreads(); });
            for (int i = threadIdx.x; i < len; i += 512) row_rank[b + i] = s[i];
            continue;
        }
        for (i64 i = threadIdx.x; i < len; i += 512) {
            const i32 r = row_rank[b + i];
            atomicOr(bitmap + (r >> 5), 1u << (r & 31));
        }
        __syncthreads();
        i64 before = 0;
        for (i32 w0 = 0; w0 < (n + 31) / 32; w0 += 512) {
            const i32 w = w0 + (i32)threadIdx.x;
            u32 bits = 0;
            if (w < (n + 31) / 32) {
                bits = __ldcg(bitmap + w);
                bitmap[w] = 0;
            }
            i64 total;
            i64 at = b + before + block_scan(__popc(bits), s_warp, total);
            for (; bits; bits &= bits - 1) row_rank[at++] = 32 * w + __ffs(bits) - 1;
            before += total;
        }
        __syncthreads();
    }
}

// Pieces of one allocation: a cudaMalloc and cudaFree take 0.3 ms each, whatever their size up to some 100 MB, and for each
// array took longer than the search of a small graph.
struct Arena {
    unsigned char* base = nullptr;
    size_t used = 0;
    template <class T>
    size_t plan(size_t count) {
        const size_t at = used;
        used += (std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
        return at;
    }
    template <class T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(base + offset);
    }
    ~Arena() { cudaFree(base); }
};

}  // namespace

namespace cbm {

int gpu_candidates(int device, int32_t n, int32_t alpha, const int64_t* row_ptr, const int32_t* col, std::vector<CandTriple>& out,
                   std::vector<int32_t>& left_to_host, std::string& err) {
    out.clear();
    left_to_host.clear();
    if (n <= 0) return 0;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        err = std::string("gpu_candidates: cudaSetDevice: ") + cudaGetErrorString(e);
        return 1;
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int blocks = (int)std::min<int64_t>((int64_t)sms * 2, n);
    const int64_t nnz = row_ptr[n];
    SearchParams p{};
    p.n = n;
    p.alpha = alpha;
    p.hits_stride = ((int64_t)n + 1) / 2 + 1;
    p.touched_stride = n;
    p.bitmap_stride = ((int64_t)n + 31) / 32 + 1;
    // Room for the candidates: a list that turns out too short costs a second search, a needlessly long one its
    // allocation.  Rows that resemble one another closely have the more candidates the more entries they have (132 534
    // rows of 265 entries, 16 a row were too few: 4.7 s instead of 1.9).
    p.out_cap = std::max<int64_t>({1ll << 20, 16ll * n, nnz / 2});
    Arena mem;
    CandTriple* longer = nullptr;  // the list, where the first one was too short
    const size_t o_row_ptr = mem.plan<i64>((size_t)n + 1), o_col_ptr = mem.plan<i64>((size_t)n + 1);
    const size_t o_row_rank = mem.plan<i32>((size_t)nnz), o_rank = mem.plan<i32>((size_t)n), o_count_of_rank = mem.plan<i32>((size_t)n);
    const size_t tiles = ((size_t)n + 1 + SCAN_TILE - 1) / SCAN_TILE, o_totals = mem.plan<i64>(tiles), o_first = mem.plan<i64>((size_t)n + 2);
    const size_t o_col_rows = mem.plan<i32>((size_t)nnz), o_skipped = mem.plan<i32>((size_t)n);
    const size_t o_large = mem.plan<i32>((size_t)n), o_out = mem.plan<CandTriple>((size_t)p.out_cap);
    const size_t o_touched = mem.plan<i32>((size_t)blocks * p.touched_stride), o_hits = mem.plan<u32>((size_t)blocks * p.hits_stride);
    const size_t o_zero = mem.used;  // cleared together: counters, counts, bitmaps
    const size_t o_count = mem.plan<u64>(2), o_n_skipped = mem.plan<i32>(1), o_n_large = mem.plan<i32>(1);
    const size_t o_columns = mem.plan<i32>((size_t)n), o_often = mem.plan<i32>((size_t)n + 1);
    const size_t o_taken = mem.plan<i32>((size_t)n + 1), o_listed = mem.plan<i32>((size_t)n);
    const size_t o_bitmap = mem.plan<u32>((size_t)blocks * p.bitmap_stride);
    const size_t zero_bytes = mem.used - o_zero;
    auto cleanup = [&]() {
        cudaFree(longer);
        if (prev >= 0) cudaSetDevice(prev);
    };
    auto fail = [&](const char* what, cudaError_t ce) {
        err = std::string("gpu_candidates: ") + what + ": " + cudaGetErrorString(ce);
        cleanup();
        return 1;
    };
    if ((e = cudaMalloc((void**)&mem.base, mem.used)) != cudaSuccess) return fail("device memory", e);
    auto send = [&](size_t offset, const void* src, size_t bytes) {
        return bytes ? cudaMemcpyAsync(mem.base + offset, src, bytes, cudaMemcpyHostToDevice) : cudaSuccess;
    };
    if ((e = cudaMemsetAsync(mem.base + o_zero, 0, zero_bytes)) != cudaSuccess ||
        (e = send(o_row_ptr, row_ptr, ((size_t)n + 1) * sizeof(i64))) != cudaSuccess ||
        (e = send(o_row_rank, col, (size_t)nnz * sizeof(i32))) != cudaSuccess)
        return fail("copy to the device", e);
    {
        const auto over = [](i64 count) { return (unsigned)((count + 255) / 256); };
        i64 *d_row_ptr = mem.at<i64>(o_row_ptr), *d_col_ptr = mem.at<i64>(o_col_ptr), *d_first = mem.at<i64>(o_first);
        i64* d_totals = mem.at<i64>(o_totals);
        i32 *d_row_rank = mem.at<i32>(o_row_rank), *d_columns = mem.at<i32>(o_columns), *d_often = mem.at<i32>(o_often);
        i32 *d_rank = mem.at<i32>(o_rank), *d_count_of_rank = mem.at<i32>(o_count_of_rank);
        const auto scan = [&](i64 count, const i32* in, i64* sums) {
            const i32 t = (i32)((count + SCAN_TILE - 1) / SCAN_TILE);
            scan_tiles_kernel<<<t, SCAN_THREADS>>>(count, in, sums, d_totals);
            scan_totals_kernel<<<1, SCAN_THREADS>>>(t, d_totals);
            scan_add_kernel<<<over(count), 256>>>(count, in, sums, d_totals);
        };
        if (nnz) count_columns_kernel<<<std::min<unsigned>(over(nnz), 8u * sms), 256>>>(nnz, d_row_rank, d_columns);
        count_counts_kernel<<<over(n), 256>>>(n, d_columns, d_often);
        scan((i64)n + 1, d_often, d_first);
        rank_columns_kernel<<<over(n), 256>>>(n, d_columns, d_first, mem.at<i32>(o_taken), d_rank, d_count_of_rank);
        scan(n, d_count_of_rank, d_col_ptr);
        list_rows_kernel<<<over((i64)n * 32), 256>>>(n, d_row_ptr, d_row_rank, d_rank, d_col_ptr, mem.at<i32>(o_listed), mem.at<i32>(o_col_rows));
        sort_rows_warp_kernel<<<over((i64)n * 32), 256>>>(n, d_row_ptr, d_row_rank);
        sort_rows_block_kernel<<<blocks, 512>>>(n, d_row_ptr, d_row_rank, mem.at<u32>(o_bitmap), p.bitmap_stride);
        if ((e = cudaGetLastError()) != cudaSuccess) return fail("launch", e);
    }
    u64* d_count = mem.at<u64>(o_count);
    i32 *d_n_skipped = mem.at<i32>(o_n_skipped), *d_skipped = mem.at<i32>(o_skipped);
    p.hits = mem.at<u32>(o_hits);
    p.touched = mem.at<i32>(o_touched);
    p.out = mem.at<CandTriple>(o_out);
    p.large = mem.at<i32>(o_large);
    p.n_large = mem.at<i32>(o_n_large);
    p.bitmap = mem.at<u32>(o_bitmap);
    p.row_ptr = mem.at<i64>(o_row_ptr);
    p.row_rank = mem.at<i32>(o_row_rank);
    p.col_ptr = mem.at<i64>(o_col_ptr);
    p.col_rows = mem.at<i32>(o_col_rows);
    p.out_count = d_count;
    p.skipped = d_skipped;
    p.n_skipped = d_n_skipped;
    for (int attempt = 0; attempt < 2; ++attempt) {  // a second pass only if the output list was too small
        if (attempt > 0) {
            if ((e = cudaMalloc((void**)&longer, (size_t)p.out_cap * sizeof(CandTriple))) != cudaSuccess) return fail("out", e);
            p.out = longer;
        }
        cudaMemset(d_count, 0, 2 * sizeof(u64));
        cudaMemset(d_n_skipped, 0, sizeof(i32));
        cudaMemset(p.n_large, 0, sizeof(i32));
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        const bool trace = std::getenv("CBM_B200_BUILD_TRACE") != nullptr;
        if (trace) {
            cudaEventCreate(&e0);
            cudaEventCreate(&e1);
            cudaEventRecord(e0);
        }
        const int table_bytes = TABLE_WARPS * TABLE_BYTES;
        if ((e = cudaFuncSetAttribute(candidate_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, table_bytes)) != cudaSuccess)
            return fail("shared memory", e);
        candidate_warp_kernel<<<std::min<int64_t>((int64_t)sms * 4, ((int64_t)n + TABLE_WARPS - 1) / TABLE_WARPS), TABLE_WARPS * 32, table_bytes>>>(p);
        if ((e = cudaGetLastError()) != cudaSuccess) return fail("launch", e);
        if ((e = cudaMemcpy(&p.n_blocks_of, p.n_large, sizeof(i32), cudaMemcpyDeviceToHost)) != cudaSuccess) return fail("kernel", e);
        if (p.n_blocks_of > 0) {
            if ((e = cudaMemsetAsync(p.hits, 0, (size_t)blocks * p.hits_stride * sizeof(u32))) != cudaSuccess) return fail("device memory", e);
            cudaMemsetAsync(d_count + 1, 0, sizeof(u64));
            candidate_kernel<<<blocks, kThreads>>>(p);
            if ((e = cudaGetLastError()) != cudaSuccess) return fail("launch", e);
        }
        if (trace) cudaEventRecord(e1);
        if ((e = cudaDeviceSynchronize()) != cudaSuccess) return fail("kernel", e);
        if (trace) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            std::fprintf(stderr, "[cbm build] candidate kernel %.3f ms\n", ms);
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
        }
        u64 h_count[2] = {0, 0};
        cudaMemcpy(h_count, d_count, sizeof(h_count), cudaMemcpyDeviceToHost);
        if ((int64_t)h_count[0] <= p.out_cap) {
            out.resize((size_t)h_count[0]);
            if (h_count[0])
                cudaMemcpy(out.data(), p.out, (size_t)h_count[0] * sizeof(CandTriple), cudaMemcpyDeviceToHost);
            i32 ns = 0;
            cudaMemcpy(&ns, d_n_skipped, sizeof(ns), cudaMemcpyDeviceToHost);
            left_to_host.resize((size_t)ns);
            if (ns) cudaMemcpy(left_to_host.data(), d_skipped, (size_t)ns * sizeof(i32), cudaMemcpyDeviceToHost);
            cleanup();
            return 0;
        }
        p.out_cap = (int64_t)h_count[0] + 1024;  // the kernel counted every survivor: now it fits
    }
    err = "gpu_candidates: output list overflowed twice";
    cleanup();
    return 1;
}

}  // namespace cbm
