// CUDA engine (sm_100a) for the CBM product: plans, kernels and the compute half of the C ABI.
//
// What the reference does in two steps per call — an MKL sparse product dst = deltas * rhs
// (cbm/cbm_extensions.cpp:694-704) followed by a depth-first walk that adds every finished parent
// row into its children (cbm/cbm_extensions.cpp:1166-1218; normalized form :1285-1373) — is done
// here by ONE kernel.  Rows are issued to warps in a topological order of the tree.  A warp
//   1. gathers the signed rows of X named by its row's delta entries into registers,
//   2. waits (bounded) until its parent's finished row is published, reads it from L2,
//   3. applies the row scale, stores the finished row once, and publishes it.
// Step 1 does not depend on the parent, so the wait in step 2 is normally already satisfied.
// Rows whose parent saves them little are gathered whole and wait for nobody (cbm_lift.cpp).
// The dense operand is processed in column slabs so that one slab of X stays resident in the
// 126 MB L2 while every row gathers from it.
//
// Forward progress: work items are claimed in increasing order from one counter, and an item only
// ever waits for an item with a smaller index.  Whoever holds that smaller item is already running
// and, by induction, never blocked on anything unclaimed, so the kernel cannot deadlock however
// many thread blocks are resident.  Every wait is bounded all the same: when the bound runs out
// the warp raises the plan's status word and all warps drain.

#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

#include "cbm_b200.h"
#include "cbm_cluster.h"
#include "cbm_common.h"
#include "cbm_launch.cuh"
#include "cbm_lift.h"

namespace cbm {
std::string& last_error_slot() {
    static thread_local std::string slot;
    return slot;
}
}  // namespace cbm

extern "C" const char* cbm_b200_last_error(void) { return cbm::last_error_slot().c_str(); }
extern "C" const char* cbm_b200_version(void) { return "cbm_b200 0.1 sm_100a"; }

namespace {

using i32 = int32_t;
using i64 = int64_t;
using u64 = unsigned long long;

#define CBM_CUDA(call)                                                                      \
    do {                                                                                    \
        cudaError_t e__ = (call);                                                           \
        if (e__ != cudaSuccess)                                                             \
            return cbm::fail(CBM_B200_ERR_CUDA, std::string(#call) + ": " +                 \
                                                    cudaGetErrorString(e__));               \
    } while (0)

// One work item of the schedule, in processing order.  32 bytes, read as two 16-byte loads.
//
// A row with many delta entries is cut into segments: all but the last become PARTIAL items that
// leave their share of the gather in a scratch slot (slot index = the item's own position); the
// last segment is the row's finishing item, which adds those slots to its own share.
//
// The schedule has two parts.  Positions [0, n_prefix) hold the items that wait for nobody — first
// every PARTIAL item, then the unsplit children of the virtual root, longest first.  Positions
// [n_prefix, n_items) hold the items that may wait: finishing items of split rows and every row
// below the first level, in breadth-first order, so that whatever an item waits for has a smaller
// position.  Delta entries are stored in item order, hence consecutive items own consecutive
// entry ranges.
struct __align__(16) RowDesc {
    i32 out_row;      // row of y this item produces (local to the shard); unused if PARTIAL
    i32 parent_row;   // row of y holding the parent's finished row, -1 under the virtual root
    i32 parent_pos;   // parent's position in processing order (index of its ready flag)
    i32 info;         // bits 0-1 ITEM_* flags, bits 8-15 number of delta entries (<= 255),
                      // bits 16-31 number of PARTIAL items of this row (finishing items only)
    i32 beg;          // first delta entry of the item in the plan's col/val arrays
    i32 first_part;   // position of the row's first PARTIAL item (when there are any)
    float scale;      // s_v  = D^-1/2 of this row (1 when the plan has no multiplier)
    float inv_parent; // 1/s_u of the parent (1 when none)
};
enum : int { ITEM_PUBLISH = 1, ITEM_PARTIAL = 2, ITEM_LEN_SHIFT = 8, ITEM_NPART_SHIFT = 16 };

// A delta entry: the column and the value to multiply it with.
struct __align__(8) Entry {
    i32 col;
    float val;
};

// Clustered plans (see cbm_chunks.cuh): a run of consecutive items that a block brings into shared memory
// together.  There every item's first entry stands at an even position.
struct __align__(16) Chunk {
    i32 first, count;  // items
    i32 e0, ne;        // their entries, both even
};

enum Mode : int { MODE_FUSED = 0, MODE_DELTA_ONLY = 1, MODE_UPDATE_ONLY = 2 };

struct KParams {
    const RowDesc* desc;
    const Entry* ent;
    const float* x;
    float* y;
    i64 ldx, ldy;
    i32 f;
    i32 y_vec;       // rows of y are 16-byte aligned
    i32 in_turn;     // entries are added strictly one after the other, also in narrow slabs
    const Chunk* chunks;   // clustered plans: chunks ...
    unsigned ldx_bytes;    // ... and 4 * ldx
    i32 slab_w;      // columns per slab
    i32 n_items;     // work items per slab
    i32 n_prefix;    // items that never wait (claimed `group` at a time)
    i32 group;       // prefix items per claim
    i32 n_pclaims;   // ceil(n_prefix / group)
    i32 claims_per_slab;  // n_pclaims + (n_items - n_prefix)
    i64 n_claims;    // claims_per_slab * n_slabs
    float* scratch;  // n_slabs * n_partial * slab_w floats: partial sums of long rows
    i32 n_partial;   // PARTIAL items (positions [0, n_partial))
    u64* counter;    // next claim; 0 between launches
    u64 n_warps;     // claimers in this launch: warps, or the blocks of a clustered plan's kernel
    i32* flags;      // n_slabs * n_items ready flags holding the epoch of the launch that set them
    i32 epoch;
    i32* status;     // 0 ok; non-zero: a wait gave up
    i32 mode;
    i32 use_scale;
    u64 wait_ns;
    // Broadcast epilogue (multi-GPU): every finished row is also written, after the optional
    // ReLU, to n_bcast further buffers with the layout of y — the slices that this shard occupies
    // in the gathered layer output of each GPU (peer memory mapped into this process, reached
    // by ordinary stores over NVLink).  y itself keeps the row as the tree needs it.
    float* bcast[CBM_B200_MAX_BCAST];
    i32 n_bcast;
    i32 bcast_relu;
};

__device__ __forceinline__ i32 ld_acquire(const i32* p) {
    i32 v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(i32* p, i32 v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ i32 ld_relaxed(const i32* p) {
    i32 v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ u64 global_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for `*flag == epoch`.  All lanes of the warp call it together.
__device__ __forceinline__ bool wait_ready(const i32* flag, i32 epoch, i32* status, u64 wait_ns) {
    if (ld_acquire(flag) == epoch) return true;
    const u64 t0 = global_ns();
    unsigned spins = 0;
    for (;;) {
        if (ld_acquire(flag) == epoch) return true;
        ++spins;
        if ((spins & 31u) == 0) {
            if (ld_relaxed(status) != 0) return false;  // someone else gave up: drain
            if (global_ns() - t0 > wait_ns) {
                atomicExch(status, CBM_B200_ERR_TIMEOUT);
                return false;
            }
        }
        __nanosleep(spins < 16 ? 20 : 200);
    }
}

template <bool V4>
struct Vec;
template <>
struct Vec<true> {
    using T = float4;
    static constexpr int E = 4;
    static __device__ __forceinline__ T zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    // Fetch of the operand that is skipped (giving zeros) when `on` is false.  Written as volatile asm
    // so that a batch of fetches stays a batch: the compiler may not sink one below its use.  (Not ld.global.nc: see cbm_launch.cuh.)
    static __device__ __forceinline__ T ld_ro_if(const float* p, bool on) {
        T v;
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
            "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
            "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
            "@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
            : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
            : "l"(p), "r"((int)on));
        return v;
    }
    // The same fetch without the predicate, for slabs in which every lane has columns.
    static __device__ __forceinline__ T ld_ro(const float* p) {
        T v;
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "l"(p));
        return v;
    }
    static __device__ __forceinline__ T ld_l2(const float* p) { return __ldcg((const float4*)p); }
    // L2-only fetch (data written earlier in the same launch), zeros when `on` is false; volatile
    // asm for the same reason as ld_ro_if.
    static __device__ __forceinline__ T ld_l2_if(const float* p, bool on) {
        T v;
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
            "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
            "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
            "@q ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
            : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
            : "l"(p), "r"((int)on)
            : "memory");
        return v;
    }
    static __device__ __forceinline__ void st(float* p, T v) { *(float4*)p = v; }
    static __device__ __forceinline__ void st_stream(float* p, T v) { __stcs((float4*)p, v); }
    static __device__ __forceinline__ T fma(float w, T a, T c) {
        c.x = fmaf(w, a.x, c.x);
        c.y = fmaf(w, a.y, c.y);
        c.z = fmaf(w, a.z, c.z);
        c.w = fmaf(w, a.w, c.w);
        return c;
    }
    static __device__ __forceinline__ T mul(float w, T a) {
        a.x *= w;
        a.y *= w;
        a.z *= w;
        a.w *= w;
        return a;
    }
    static __device__ __forceinline__ T relu(T a) {
        a.x = fmaxf(a.x, 0.f);
        a.y = fmaxf(a.y, 0.f);
        a.z = fmaxf(a.z, 0.f);
        a.w = fmaxf(a.w, 0.f);
        return a;
    }
    static __device__ __forceinline__ T add_xor(T a, int d) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, d);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, d);
        a.z += __shfl_xor_sync(0xffffffffu, a.z, d);
        a.w += __shfl_xor_sync(0xffffffffu, a.w, d);
        return a;
    }
    // Rows whose vectors are not 16-byte aligned, or a vector that reaches past the row's end: the
    // `n` columns that exist, one by one.
    static __device__ __forceinline__ void st_some(float* p, T v, int n) {
        if (n > 0) p[0] = v.x;
        if (n > 1) p[1] = v.y;
        if (n > 2) p[2] = v.z;
        if (n > 3) p[3] = v.w;
    }
    static __device__ __forceinline__ T ld_some_l2(const float* p, int n) {
        T v = zero();
        if (n > 0) v.x = __ldcg(p);
        if (n > 1) v.y = __ldcg(p + 1);
        if (n > 2) v.z = __ldcg(p + 2);
        if (n > 3) v.w = __ldcg(p + 3);
        return v;
    }
};
template <>
struct Vec<false> {
    using T = float;
    static constexpr int E = 1;
    static __device__ __forceinline__ T zero() { return 0.f; }
    static __device__ __forceinline__ T ld_ro_if(const float* p, bool on) {
        T v;
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "@q ld.global.f32 %0, [%1];\n\t}"
            : "=f"(v)
            : "l"(p), "r"((int)on));
        return v;
    }
    static __device__ __forceinline__ T ld_ro(const float* p) {
        T v;
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
        return v;
    }
    static __device__ __forceinline__ T ld_l2(const float* p) { return __ldcg(p); }
    static __device__ __forceinline__ T ld_l2_if(const float* p, bool on) {
        T v;
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
            "@q ld.global.cg.f32 %0, [%1];\n\t}"
            : "=f"(v)
            : "l"(p), "r"((int)on)
            : "memory");
        return v;
    }
    static __device__ __forceinline__ void st(float* p, T v) { *p = v; }
    static __device__ __forceinline__ void st_stream(float* p, T v) { __stcs(p, v); }
    static __device__ __forceinline__ T fma(float w, T a, T c) { return fmaf(w, a, c); }
    static __device__ __forceinline__ T mul(float w, T a) { return w * a; }
    static __device__ __forceinline__ T relu(T a) { return fmaxf(a, 0.f); }
    static __device__ __forceinline__ T add_xor(T a, int d) { return a + __shfl_xor_sync(0xffffffffu, a, d); }
    static __device__ __forceinline__ void st_some(float* p, T v, int n) {
        if (n > 0) *p = v;
    }
    static __device__ __forceinline__ T ld_some_l2(const float* p, int n) { return n > 0 ? __ldcg(p) : 0.f; }
};

// Where the entries of a row come from: a plan's array of pairs, or a caller's two CSR arrays.
struct PairEntries {
    const Entry* e;
    __device__ __forceinline__ void get(i32 i, i32& c, float& w) const {
        const int2 q = __ldg(reinterpret_cast<const int2*>(e) + i);
        c = q.x;
        w = __int_as_float(q.y);
    }
};
struct CsrEntries {
    const i32* __restrict__ col;
    const float* __restrict__ val;
    __device__ __forceinline__ void get(i32 i, i32& c, float& w) const {
        c = __ldg(col + i);
        w = __ldg(val + i);
    }
};

// acc[v] += sum over entries [beg,end) of val * X[col, slab columns of this lane].
// The 32 lanes fetch 32 (col, val) pairs at once and pass them round by shuffle.  Row fetches are
// issued UNROLL at a time so that several independent loads per lane are in flight; the weights
// are picked up after the fetches have been issued.
template <int NV, bool V4, int UNROLL, bool FULL = false, class Entries>
__device__ __forceinline__ void gather_row(const Entries ent, i32 beg, i32 end,
                                           const float* __restrict__ xs, i64 ldx,
                                           const bool (&ok)[NV], typename Vec<V4>::T (&acc)[NV],
                                           int lane) {
    using V = Vec<V4>;
    using T = typename V::T;
    constexpr int STEP = 32 * V::E;
    for (i32 b = beg; b < end; b += 32) {
        const i32 n_here = min(32, end - b);
        i32 mc = 0;
        float mw = 0.f;
        if (lane < n_here) ent.get(b + lane, mc, mw);
        i32 j = 0;
        for (; j + UNROLL <= n_here; j += UNROLL) {
            T t[UNROLL][NV];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) {
                const i32 c = __shfl_sync(0xffffffffu, mc, j + k);
                const float* r = xs + (i64)c * ldx;
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    if constexpr (FULL) t[k][v] = V::ld_ro(r + v * STEP);  // every lane has columns
                    else t[k][v] = V::ld_ro_if(r + v * STEP, ok[v]);
                }
            }
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) {
                const float w = __shfl_sync(0xffffffffu, mw, j + k);
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[v] = V::fma(w, t[k][v], acc[v]);
            }
        }
        if (j < n_here) {  // the last, shorter batch: same code with the surplus fetches switched off
            T t[UNROLL][NV];
            const i32 live = n_here - j;
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) {
                const i32 c = __shfl_sync(0xffffffffu, mc, (j + k) & 31);
                const float* r = xs + (i64)c * ldx;
#pragma unroll
                for (int v = 0; v < NV; ++v) t[k][v] = V::ld_ro_if(r + v * STEP, ok[v] && k < live);
            }
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) {
                const float w = __shfl_sync(0xffffffffu, mw, (j + k) & 31);  // 0 past the end
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[v] = V::fma(k < live ? w : 0.f, t[k][v], acc[v]);
            }
        }
    }
}

// The same sum for slabs that 2^lg < 32 lanes cover with one vector each: 32 >> lg delta entries are fetched side by
// side, one per group of lanes, and the groups' sums are combined by shuffles at the end, so that every lane
// holds the total of its column group.
template <bool V4, int UNROLL, class Entries>
__device__ __forceinline__ void gather_row_narrow(const Entries ent, i32 beg, i32 end, const float* __restrict__ x_slab,
                                                  i64 ldx, i32 wcols, int lg, typename Vec<V4>::T& acc, int lane) {
    using V = Vec<V4>;
    const int li = lane & ((1 << lg) - 1), group = lane >> lg, side = 32 >> lg;
    const bool okh = li * V::E < wcols;
    const float* xs = x_slab + li * V::E;
    for (i32 b = beg; b < end; b += 32) {
        const i32 n_here = min(32, end - b);
        i32 mc = 0;
        float mw = 0.f;
        if (lane < n_here) ent.get(b + lane, mc, mw);
        for (i32 j = 0; j < n_here; j += side * UNROLL) {
            typename V::T t[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) {
                const i32 idx = j + k * side + group;
                const i32 c = __shfl_sync(0xffffffffu, mc, idx & 31);
                t[k] = V::ld_ro_if(xs + (i64)c * ldx, okh && idx < n_here);
            }
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) {
                const i32 idx = j + k * side + group;
                const float w = __shfl_sync(0xffffffffu, mw, idx & 31);
                acc = V::fma(idx < n_here ? w : 0.f, t[k], acc);
            }
        }
    }
    for (int d = 1 << lg; d < 32; d <<= 1) acc = V::add_xor(acc, d);
}

// Lanes (as a power of two) that cover `wcols` columns with one vector of E floats each.
template <int E>
__device__ __forceinline__ int lanes_log2(i32 wcols) {
    const i32 lanes = (wcols + E - 1) / E;
    return lanes <= 1 ? 0 : 32 - __clz(lanes - 1);
}

// Claims are drawn from one counter, and every claimer draws until it gets one past the last: together they draw
// n_claims + n_warps, and whoever draws the last of these rewinds the counter for the next launch.
__device__ __forceinline__ void draw_last(const KParams& p, u64 t) {
    if (t == (u64)p.n_claims + p.n_warps - 1) *p.counter = 0;
}

// A claimer that gives up draws what is left without working on it, so that the counter is rewound after a failed wait
// too and a plan stays usable after a timeout.  (Whoever waits for such an item sees the status word.)
__device__ __forceinline__ void drain(const KParams& p, int lane) {
    if (lane != 0) return;
    u64 t;
    do t = atomicAdd(p.counter, 1ULL);
    while (t < (u64)p.n_claims);
    draw_last(p, t);
}

// The first claims of a block's 8 warps, drawn as one: the draws of all warps at the start of a launch meet at one address,
// one after the other, and 7 104 of them take 4 us.  In one round (see LaunchCfg) there are no others.  (The shuffle tells
// the compiler that the number is the same in all lanes: it is kept out of the 40 registers then.)
template <bool ONE_ROUND>
__device__ __forceinline__ u64 first_claim(const KParams& p) {
    __shared__ u64 s_first;
    if (threadIdx.x == 0) {
        s_first = atomicAdd(p.counter, 8ULL);
        if (ONE_ROUND && s_first + 8 == p.n_warps) *p.counter = 0;
    }
    __syncthreads();
    return __shfl_sync(0xffffffffu, s_first + (threadIdx.x >> 5), 0);
}

__device__ __forceinline__ u64 draw_claim(const KParams& p, int lane) {
    u64 t = 0;
    if (lane == 0) t = atomicAdd(p.counter, 1ULL);
    return __shfl_sync(0xffffffffu, t, 0);
}

// Maps a claim number to (slab, first item, end of its items): inside a slab the prefix is handed out
// `group` items at a time, the rest one item at a time.  Only items that never wait are grouped:
// a warp that sits on an item waiting for a neighbour would starve the items behind it in its
// group, which others in turn wait for (measured: 16x slower with 4 mixed items per claim).
// In one round a claim's items of the prefix lie n_pclaims apart: they stand in order of length, and every warp is to have
// as much to do as the others.
template <bool ONE_ROUND = false>
__device__ __forceinline__ void decode_claim(const KParams& p, u64 t, i32& slab, i32& first, i32& end) {
    const unsigned u = (unsigned)t;  // the host refuses launches of 2^31 claims or more
    slab = (i32)(u / (unsigned)p.claims_per_slab);
    const i32 r = (i32)(u - (unsigned)slab * (unsigned)p.claims_per_slab);
    if (r >= p.n_pclaims) {
        first = p.n_prefix + (r - p.n_pclaims);
        end = first + 1;
    } else if (ONE_ROUND) {
        first = r;
        end = p.n_prefix;
    } else {
        first = r * p.group;
        end = min(first + p.group, p.n_prefix);
    }
}

// Everything that happens to an item once its own gather is in `acc`: park a PARTIAL share, or
// collect the row's parked shares, add the parent's finished row, scale, store and publish.
// Returns false when a bounded wait ran out.
template <int NV, bool V4, bool RAGGED = false>
__device__ __forceinline__ bool finish_item(const KParams& p, i32 slab, i32 pos, i32 out_row,
                                            i32 parent_row, i32 parent_pos, i32 info,
                                            i32 first_part, float scale, float inv_parent,
                                            typename Vec<V4>::T (&acc)[NV], const bool (&ok)[NV],
                                            i32 c0, int lane) {
    using V = Vec<V4>;
    constexpr int STEP = 32 * V::E;
    i32* slab_flags = p.flags + (i64)slab * p.n_items;
    if (info & ITEM_PARTIAL) {
        float* slot = p.scratch + ((i64)slab * p.n_partial + pos) * p.slab_w + lane * V::E;
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (ok[v]) V::st(slot + v * STEP, acc[v]);
        // the warp barrier orders every lane's stores before lane 0's release store, whose
        // gpu-scope release then covers them all: no per-lane fence is needed
        __syncwarp();
        if (lane == 0) st_release(slab_flags + pos, p.epoch);
        return true;
    }
    const i32 n_part = (i32)((unsigned)info >> ITEM_NPART_SHIFT);
    if (n_part > 0 && p.mode != MODE_UPDATE_ONLY) {
        // A row can have hundreds of parked shares; taking them one memory round trip at a time
        // would serialise the whole product behind the longest row.  The 32 lanes wait for 32
        // flags at once, then the shares are fetched PART_BATCH at a time and added in slot order
        // (a fixed order, so results do not depend on timing).
        bool mine = true;
        for (i32 k = lane; k < n_part; k += 32)
            mine = mine && wait_ready(slab_flags + first_part + k, p.epoch, p.status, p.wait_ns);
        if (!__all_sync(0xffffffffu, mine)) return false;
        // lane k acquired flag k; the warp barrier extends that ordering to the lanes that did not
        __syncwarp();
        constexpr int PART_BATCH = NV == 1 ? 8 : 4;
        const float* slot0 = p.scratch + ((i64)slab * p.n_partial + first_part) * p.slab_w + lane * V::E;
        for (i32 k = 0; k < n_part; k += PART_BATCH) {
            typename V::T t[PART_BATCH][NV];
#pragma unroll
            for (int j = 0; j < PART_BATCH; ++j)
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    t[j][v] = V::ld_l2_if(slot0 + (i64)(k + j) * p.slab_w + v * STEP, ok[v] && (k + j) < n_part);
#pragma unroll
            for (int j = 0; j < PART_BATCH; ++j)
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[v] = V::fma(1.0f, t[j][v], acc[v]);
        }
    }
    const i32 lane_col = c0 + lane * V::E;
    // RAGGED: rows of y that are not 16-byte aligned, or a last vector that reaches past column f; the columns
    // of vector v that exist are then accessed one by one
    auto some = [&](int v) { return p.f - (lane_col + v * STEP); };
    auto whole = [&](int v) { return !RAGGED || (p.y_vec && some(v) >= V::E); };
    if (p.mode != MODE_DELTA_ONLY) {
        if (parent_row >= 0) {
            if (!wait_ready(slab_flags + parent_pos, p.epoch, p.status, p.wait_ns)) return false;
            const float* prow = p.y + (i64)parent_row * p.ldy + lane_col;
            const float ip = p.use_scale ? inv_parent : 1.0f;
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (ok[v])
                    acc[v] = V::fma(ip, whole(v) ? V::ld_l2(prow + v * STEP) : V::ld_some_l2(prow + v * STEP, some(v)),
                                    acc[v]);
        }
        if (p.use_scale) {
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[v] = V::mul(scale, acc[v]);
        }
    }
    float* yrow = p.y + (i64)out_row * p.ldy + lane_col;
    if (info & ITEM_PUBLISH) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (ok[v]) {
                if (whole(v)) V::st(yrow + v * STEP, acc[v]);
                else V::st_some(yrow + v * STEP, acc[v], some(v));
            }
    } else {
        // nobody reads this row again during the product: a streaming store keeps it from
        // pushing slabs of X out of L2
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (ok[v]) {
                if (whole(v)) V::st_stream(yrow + v * STEP, acc[v]);
                else V::st_some(yrow + v * STEP, acc[v], some(v));
            }
    }
    if ((info & ITEM_PUBLISH) && p.mode != MODE_DELTA_ONLY) {
        __syncwarp();
        if (lane == 0) st_release(slab_flags + pos, p.epoch);
    }
    if (p.n_bcast > 0) {
        if (p.bcast_relu) {
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[v] = V::relu(acc[v]);
        }
        const i64 off = (i64)out_row * p.ldy + lane_col;
        for (int k = 0; k < p.n_bcast; ++k) {
            float* dst = p.bcast[k] + off;
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (ok[v]) {
                    if (whole(v)) V::st(dst + v * STEP, acc[v]);
                    else V::st_some(dst + v * STEP, acc[v], some(v));
                }
        }
    }
    return true;
}

// Several whole rows that wait for nobody (prefix items, positions [first, end), none of them PARTIAL) by one warp, 2^lg
// lanes for each: for slabs of at most 16 vectors, where a row's fixed costs - descriptor, entries, store, each a trip to
// memory - outweigh its fetches.  Neighbours in the prefix are of about equal length.  A row's entries are summed as
// gather_row_narrow sums them, in 32 >> lg interleaved shares: which of the two a row gets depends on where its claim
// falls, its bits do not.  Four entries of each row are on their way at a time, without conditions as long as all rows have
// them (two, each with its own: 50 000 rows of 31 entries, 64 columns 44.2 us, 43.0 now).
template <bool V4, bool RAGGED, int LG>
__device__ __forceinline__ void rows_narrow(const KParams& p, i32 slab, i32 first, i32 end, i32 c0, i32 wcols, int lane) {
    using V = Vec<V4>;
    using T = typename V::T;
    constexpr int width = 1 << LG, SHARES = 32 >> LG, UNROLL = 4;
    const int li = lane & (width - 1);
    const bool has = li * V::E < wcols;
    const float* xs = p.x + c0 + li * V::E;
    for (i32 base = first; base < end; base += SHARES) {
        const i32 pos = base + (lane >> LG);
        const bool on = pos < end;
        const int4 da = __ldg((const int4*)(p.desc + min(pos, end - 1)));
        const int4 db = __ldg((const int4*)(p.desc + min(pos, end - 1)) + 1);
        const i32 len = on ? (da.w >> ITEM_LEN_SHIFT) & 0xff : 0;
        const i32 most = (i32)__reduce_max_sync(0xffffffffu, (unsigned)len), least = (i32)__reduce_min_sync(0xffffffffu, (unsigned)len);
        T acc[SHARES];
#pragma unroll
        for (int s = 0; s < SHARES; ++s) acc[s] = V::zero();
        for (i32 b = 0; b < most; b += width) {
            i32 mc = 0;
            float mw = 0.f;
            if (b + li < len) PairEntries{p.ent}.get(db.x + b + li, mc, mw);
            const i32 here = min(width, most - b);
            for (i32 j = 0; j < here; j += UNROLL) {
                T t[UNROLL];
                if (b + j + UNROLL <= least) {  // all rows have these entries
#pragma unroll
                    for (int k = 0; k < UNROLL; ++k) {
                        const i32 c = __shfl_sync(0xffffffffu, mc, j + k, width);
                        t[k] = V::ld_ro_if(xs + (i64)c * p.ldx, has);
                    }
#pragma unroll
                    for (int k = 0; k < UNROLL; ++k)
                        acc[k % SHARES] = V::fma(__shfl_sync(0xffffffffu, mw, j + k, width), t[k], acc[k % SHARES]);
                } else {
#pragma unroll
                    for (int k = 0; k < UNROLL; ++k) {
                        const i32 c = __shfl_sync(0xffffffffu, mc, j + k, width);
                        t[k] = V::ld_ro_if(xs + (i64)c * p.ldx, has && b + j + k < len);
                    }
#pragma unroll
                    for (int k = 0; k < UNROLL; ++k) {
                        const float w = __shfl_sync(0xffffffffu, mw, j + k, width);
                        acc[k % SHARES] = V::fma(b + j + k < len ? w : 0.f, t[k], acc[k % SHARES]);
                    }
                }
            }
        }
#pragma unroll
        for (int d = 1; d < SHARES; d <<= 1)
#pragma unroll
            for (int s = 0; s < SHARES; s += 2 * d) acc[s] = V::fma(1.0f, acc[s + d], acc[s]);
        if (p.use_scale && p.mode != MODE_DELTA_ONLY) acc[0] = V::mul(__int_as_float(db.z), acc[0]);
        if (on && has) {
            const i32 col = c0 + li * V::E, some = p.f - col;
            float* y = p.y + (i64)da.x * p.ldy + col;
            if (RAGGED && !(p.y_vec && some >= V::E)) V::st_some(y, acc[0], some);
            else if (da.w & ITEM_PUBLISH) V::st(y, acc[0]);
            else V::st_stream(y, acc[0]);
        }
        if (p.mode != MODE_DELTA_ONLY) {
            __syncwarp();
            if (on && li == 0 && (da.w & ITEM_PUBLISH)) st_release(p.flags + (i64)slab * p.n_items + pos, p.epoch);
        }
    }
}

// The same for claims of 8 rows, community order: all descriptors are fetched at once, and then all entries, which follow one another,
// into the warp's piece of shared memory (400 000 rows of 22 entries, 47 columns 247 us without, 232 with it).
// Works on as many rows as have room for their entries, and returns the first one after them.
constexpr int NARROW_ROWS = 8, NARROW_ENTRIES = 256;  // of a claim, that a warp's shared memory takes
struct NarrowClaim {
    int4 desc[2 * NARROW_ROWS];
    int2 ent[NARROW_ENTRIES];
};

template <bool V4, bool RAGGED, int LG>
__device__ __forceinline__ i32 rows_narrow_staged(const KParams& p, NarrowClaim& my, i32 slab, i32 first, i32 end, i32 c0, i32 wcols, int lane) {
    using V = Vec<V4>;
    using T = typename V::T;
    constexpr int width = 1 << LG, SHARES = 32 >> LG, UNROLL = 4;
    const int li = lane & (width - 1);
    const bool has = li * V::E < wcols;
    const float* xs = p.x + c0 + li * V::E;
    i32 e0;
    {
        int4 q = make_int4(0, 0, 0, 0);
        if (lane < 2 * (end - first)) q = __ldg((const int4*)(p.desc + first) + lane);
        e0 = __shfl_sync(0xffffffffu, q.x, 1);
        // row r's entries end, counted from the first row's, at what lane 2 r holds
        const i32 upto = __shfl_down_sync(0xffffffffu, q.x, 1) + ((q.w >> ITEM_LEN_SHIFT) & 0xff) - e0;
        const i32 rows = __popc(__ballot_sync(0xffffffffu, lane % 2 == 0 && lane < 2 * (end - first) && upto <= NARROW_ENTRIES));
        if (rows < end - first) end = first + rows / SHARES * SHARES;
        if (end == first) return first;
        const i32 n_ent = __shfl_sync(0xffffffffu, upto, 2 * (end - first - 1));
        __syncwarp();  // (all lanes are done with the claim before)
        if (lane < 2 * NARROW_ROWS) my.desc[lane] = q;
        for (i32 i = lane; i < n_ent; i += 32) my.ent[i] = __ldg(reinterpret_cast<const int2*>(p.ent) + e0 + i);
        __syncwarp();
    }
    for (i32 base = first; base < end; base += SHARES) {
        const i32 pos = base + (lane >> LG);
        const bool on = pos < end;
        const int at = 2 * (min(pos, end - 1) - first);
        const i32 len = on ? (my.desc[at].w >> ITEM_LEN_SHIFT) & 0xff : 0;
        const i32 most = (i32)__reduce_max_sync(0xffffffffu, (unsigned)len), least = (i32)__reduce_min_sync(0xffffffffu, (unsigned)len);
        T acc[SHARES];
#pragma unroll
        for (int s = 0; s < SHARES; ++s) acc[s] = V::zero();
        const int2* e = my.ent + (my.desc[at + 1].x - e0);
        i32 j = 0;
        for (; j + UNROLL <= least; j += UNROLL) {  // all rows have these entries
            T t[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) t[k] = V::ld_ro_if(xs + (i64)e[j + k].x * p.ldx, has);
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) acc[k % SHARES] = V::fma(__int_as_float(e[j + k].y), t[k], acc[k % SHARES]);
        }
        for (; j < most; j += UNROLL) {
            T t[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k) t[k] = V::ld_ro_if(xs + (i64)(j + k < len ? e[j + k].x : 0) * p.ldx, has && j + k < len);
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                acc[k % SHARES] = V::fma(j + k < len ? __int_as_float(e[j + k].y) : 0.f, t[k], acc[k % SHARES]);
        }
#pragma unroll
        for (int d = 1; d < SHARES; d <<= 1)
#pragma unroll
            for (int s = 0; s < SHARES; s += 2 * d) acc[s] = V::fma(1.0f, acc[s + d], acc[s]);
        const int4 da = my.desc[at];
        if (p.use_scale && p.mode != MODE_DELTA_ONLY) acc[0] = V::mul(__int_as_float(my.desc[at + 1].z), acc[0]);
        if (on && has) {
            const i32 col = c0 + li * V::E, some = p.f - col;
            float* y = p.y + (i64)da.x * p.ldy + col;
            if (RAGGED && !(p.y_vec && some >= V::E)) V::st_some(y, acc[0], some);
            else if (da.w & ITEM_PUBLISH) V::st(y, acc[0]);
            else V::st_stream(y, acc[0]);
        }
        if (p.mode != MODE_DELTA_ONLY) {
            __syncwarp();
            if (on && li == 0 && (da.w & ITEM_PUBLISH)) st_release(p.flags + (i64)slab * p.n_items + pos, p.epoch);
        }
    }
    return end;
}

// Product kernel, register form: one warp per (item, column slab), the gather held in registers.
// Serves operands the bulk-copy form cannot take (width not a multiple of 4 floats, unaligned
// pointers) and the update-only mode, which gathers nothing; it is also the default form.
// UNROLL = row fetches in flight per lane, MINB = thread blocks the register budget must allow
// per SM.
// NARROW: every slab is at most 64 columns wide; STAGED: and claims are of up to 8 rows in community order.
template <int NV, bool V4, int UNROLL, int MINB, bool RAGGED = false, bool NARROW = false, bool ONE_ROUND = false, bool STAGED = false>
__global__ void __launch_bounds__(256, MINB) cbm_items_kernel(const __grid_constant__ KParams p) {
    cbm::wait_before();
    using V = Vec<V4>;
    using T = typename V::T;
    constexpr int STEP = 32 * V::E;
    __shared__ NarrowClaim s_narrow[STAGED ? 8 : 1];
    const int lane = threadIdx.x & 31;
    for (u64 t = first_claim<ONE_ROUND>(p);; t = draw_claim(p, lane)) {
        if (t >= (u64)p.n_claims) {
            if (!ONE_ROUND && lane == 0) draw_last(p, t);
            return;
        }
        i32 slab, first, end;
        decode_claim<ONE_ROUND>(p, t, slab, first, end);
        const i32 c0 = slab * p.slab_w;
        const i32 wcols = min(p.slab_w, p.f - c0);
        bool ok[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) ok[v] = (lane * V::E + v * STEP) < wcols;
        if constexpr (NARROW) {
            const int lg = lanes_log2<V::E>(wcols);
            if (!ONE_ROUND && lg >= 3 && end - first > 1 && end - first <= NARROW_ROWS && first >= p.n_partial && end <= p.n_prefix && p.n_bcast == 0) {
                if constexpr (STAGED) {
                    NarrowClaim& my = s_narrow[threadIdx.x >> 5];
                    for (i32 from = -1; from != first && first < end;) {
                        from = first;
                        first = lg == 4 ? rows_narrow_staged<V4, RAGGED, 4>(p, my, slab, first, end, c0, wcols, lane)
                                        : rows_narrow_staged<V4, RAGGED, 3>(p, my, slab, first, end, c0, wcols, lane);
                    }
                } else {
                    if (lg == 4) rows_narrow<V4, RAGGED, 4>(p, slab, first, end, c0, wcols, lane);
                    else rows_narrow<V4, RAGGED, 3>(p, slab, first, end, c0, wcols, lane);
                    continue;
                }
            }
        }
        for (i32 pos = first; pos < end; pos += ONE_ROUND ? p.n_pclaims : 1) {
            const int4 da = __ldg((const int4*)(p.desc + pos));
            const int4 db = __ldg((const int4*)(p.desc + pos) + 1);
            const i32 info = da.w;
            if ((info & ITEM_PARTIAL) && p.mode == MODE_UPDATE_ONLY) continue;  // nothing to gather
            T acc[NV];
            if (p.mode == MODE_UPDATE_ONLY) {
                const float* yrow = p.y + (i64)da.x * p.ldy + c0 + lane * V::E;
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[v] = ok[v] ? V::ld_l2(yrow + v * STEP) : V::zero();  // (y_vec here)
            } else {
#pragma unroll
                for (int v = 0; v < NV; ++v) acc[v] = V::zero();
                const i32 len = (info >> ITEM_LEN_SHIFT) & 0xff;
                if constexpr (NARROW) {
                    gather_row_narrow<V4, UNROLL>(PairEntries{p.ent}, db.x, db.x + len, p.x + c0, p.ldx, wcols,
                                                  lanes_log2<V::E>(wcols), acc[0], lane);
                } else if constexpr (NV == 1) {
                    if (wcols <= 16 * V::E && !p.in_turn)
                        gather_row_narrow<V4, UNROLL>(PairEntries{p.ent}, db.x, db.x + len, p.x + c0, p.ldx, wcols,
                                                      lanes_log2<V::E>(wcols), acc[0], lane);
                    else if (V4 && wcols == 128)  // a complete slab: no per-lane predicate on the fetches
                        gather_row<NV, V4, UNROLL, true>(PairEntries{p.ent}, db.x, db.x + len, p.x + c0 + lane * V::E,
                                                         p.ldx, ok, acc, lane);
                    else
                        gather_row<NV, V4, UNROLL>(PairEntries{p.ent}, db.x, db.x + len, p.x + c0 + lane * V::E,
                                                   p.ldx, ok, acc, lane);
                } else {
                    gather_row<NV, V4, UNROLL>(PairEntries{p.ent}, db.x, db.x + len, p.x + c0 + lane * V::E, p.ldx,
                                               ok, acc, lane);
                }
            }
            if (!finish_item<NV, V4, RAGGED>(p, slab, pos, da.x, da.y, da.z, info, db.y, __int_as_float(db.z),
                                             __int_as_float(db.w), acc, ok, c0, lane)) {
                if (!ONE_ROUND) drain(p, lane);
                return;
            }
        }
        if (ONE_ROUND) return;
    }
}

// The register form for products that may park only the partial sums of the longest rows (the fixed scratch array, see
// cbm_b200_spmm_update_static): the PARTIAL items from position `kept` on are left out, and the finishing items they
// belong to gather those segments themselves, one after the other and in the same order, so that the results are the
// same bits.  Positions, flags and slots are numbered without the `out` items left out; p holds the counts so numbered.
template <int NV, bool V4>
__global__ void __launch_bounds__(256, NV == 1 ? 4 : 2) cbm_items_frugal_kernel(const KParams p, i32 out, i32 segment) {
    using V = Vec<V4>;
    using T = typename V::T;
    constexpr int STEP = 32 * V::E, UNROLL = 4;
    const int lane = threadIdx.x & 31;
    const i32 kept = p.n_partial;
    for (u64 t = first_claim<false>(p);; t = draw_claim(p, lane)) {
        if (t >= (u64)p.n_claims) {
            if (lane == 0) draw_last(p, t);
            return;
        }
        i32 slab, first, end;
        decode_claim(p, t, slab, first, end);
        const i32 c0 = slab * p.slab_w;
        const i32 wcols = min(p.slab_w, p.f - c0);
        bool ok[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) ok[v] = (lane * V::E + v * STEP) < wcols;
        auto gather = [&](i32 beg, i32 len, T(&acc)[NV]) {
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[v] = V::zero();
            if (NV == 1 && wcols <= 16 * V::E)
                gather_row_narrow<V4, UNROLL>(PairEntries{p.ent}, beg, beg + len, p.x + c0, p.ldx, wcols, lanes_log2<V::E>(wcols),
                                              acc[0], lane);
            else
                gather_row<NV, V4, UNROLL>(PairEntries{p.ent}, beg, beg + len, p.x + c0 + lane * V::E, p.ldx, ok, acc, lane);
        };
        for (i32 pos = first; pos < end; ++pos) {
            const i32 item = pos < kept ? pos : pos + out;
            const int4 da = __ldg((const int4*)(p.desc + item));
            const int4 db = __ldg((const int4*)(p.desc + item) + 1);
            i32 info = da.w;
            T acc[NV];
            gather(db.x, (info >> ITEM_LEN_SHIFT) & 0xff, acc);
            const i32 n_part = (i32)((unsigned)info >> ITEM_NPART_SHIFT);
            if (n_part > 0 && db.y >= kept) {
                const i32 beg = __ldg(&p.desc[db.y].beg);
                for (i32 k = 0; k < n_part; ++k) {
                    T part[NV];
                    gather(beg + k * segment, segment, part);
#pragma unroll
                    for (int v = 0; v < NV; ++v) acc[v] = V::fma(1.0f, part[v], acc[v]);
                }
                info &= (1 << ITEM_NPART_SHIFT) - 1;
            }
            if (!finish_item<NV, V4, V4>(p, slab, pos, da.x, da.y, da.z - out, info, db.y, __int_as_float(db.z),
                                         __int_as_float(db.w), acc, ok, c0, lane)) {
                drain(p, lane);
                return;
            }
        }
    }
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Bounded: gives up after `limit_ns` (each poll itself blocks for a hardware-defined slice), or, where
// `heed` is set, as soon as another wait of the launch has given up.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, i32* status, u64 limit_ns = 2000000000ULL,
                                          bool heed = false) {
    if (mbar_try_wait(bar, parity)) return true;
    const u64 t0 = global_ns();
    for (unsigned spins = 0; spins < (1u << 24); ++spins) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spins & 63u) == 63u) {
            if (heed && ld_relaxed(status) != 0) return false;
            if (global_ns() - t0 > limit_ns) break;
        }
    }
    atomicExch(status, CBM_B200_ERR_TIMEOUT);
    return false;
}
// Global -> shared; src, dst and bytes are multiples of 16 (the host checks).
__device__ __forceinline__ void bulk_copy_g2s(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void fence_async_proxy() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

#include "cbm_chunks.cuh"

// ------------------------------------------------------------------------------------------
// Bulk-copy form of the product kernel.
//
// The register form keeps at most UNROLL row fetches per lane in flight, so a typical row of 20-30
// delta entries costs several memory round trips in a row, on top of the round trips for the
// claim, the descriptor and the indices.  Here each lane issues ONE bulk asynchronous copy
// (cp.async.bulk, the untiled TMA path) that brings a whole slab-wide piece of one operand row
// into shared memory, so up to NB rows per stage are in flight per warp and complete on an
// mbarrier; stages alternate so the next batch is on its way while the current one is summed out
// of shared memory.  Items of the never-waiting prefix are claimed `group` at a time and their
// consecutive entry ranges are streamed as one sequence of batches, which amortises the claim and
// keeps short rows from leaving the pipeline empty.
//
// Measured on B200 (100 000-row product, F = 500): the copy engine retires about 7 G bulk copies
// per second whatever their size between 512 B and 1 KB, so 512-byte pieces reach 3.5 TB/s and
// 1 KB pieces 7 TB/s, against 12.8 TB/s for the register form.  Row pieces of a few hundred bytes
// are too small for this path; it is kept as an opt-in form (cbm_b200_plan_tune, form = 1) and the
// register form is the default.
// ------------------------------------------------------------------------------------------
template <int SLABW, int NB, int STAGES>
struct TmaLayout {
    static constexpr int SLABB = SLABW * 4;                   // bytes of one row piece
    static constexpr int STAGE_BYTES = NB * SLABB;            // NB row pieces
    // rounded up so that every warp's area starts 128-byte aligned (bulk copies need 16)
    static constexpr int WARP_BYTES = (STAGES * STAGE_BYTES + STAGES * NB * 4 + STAGES * 8 + 127) / 128 * 128;
    static __host__ __device__ constexpr int smem_bytes(int warps) { return warps * WARP_BYTES; }
};

template <int SLABW, int NB, int STAGES, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) cbm_items_tma_kernel(const KParams p) {
    using V = Vec<true>;
    using T = float4;
    using L = TmaLayout<SLABW, NB, STAGES>;
    constexpr int NV = SLABW / 128;
    constexpr int STEP = 128;
    static_assert(NB <= 32 && SLABW % 128 == 0, "one lane per staged row; slabs of 128 floats");
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    unsigned char* my = smem + (size_t)warp * L::WARP_BYTES;
    unsigned char* rows = my;                                               // [STAGES][NB][SLABB]
    float* wts = reinterpret_cast<float*>(my + STAGES * L::STAGE_BYTES);    // [STAGES][NB]
    const unsigned bar0 = smem_addr(my + STAGES * L::STAGE_BYTES + STAGES * NB * 4);
    if (lane == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_init(bar0 + 8 * s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_async_proxy();
    __syncwarp();
    unsigned parity = 0;  // bit s = phase the next wait on stage s looks for

    for (;;) {
        const u64 t = draw_claim(p, lane);
        if (t >= (u64)p.n_claims) {
            if (lane == 0) draw_last(p, t);
            return;
        }
        i32 slab, first, end;
        decode_claim(p, t, slab, first, end);
        const i32 count = end - first;
        const i32 c0 = slab * SLABW;
        const i32 wcols = min(SLABW, p.f - c0);
        const unsigned piece = (unsigned)wcols * 4u;
        bool ok[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) ok[v] = (lane * 4 + v * STEP) < wcols;

        // lane i keeps the descriptor of item first + i
        int4 da = make_int4(0, -1, -1, 0), db = make_int4(0, 0, 0, 0);
        if (lane < count) {
            da = __ldg((const int4*)(p.desc + first + lane));
            db = __ldg((const int4*)(p.desc + first + lane) + 1);
        }
        const i32 my_end = db.x + ((da.w >> ITEM_LEN_SHIFT) & 0xff);
        const i32 e_begin = __shfl_sync(0xffffffffu, db.x, 0);
        const i32 e_end = __shfl_sync(0xffffffffu, my_end, count - 1);
        const i32 n_batches = (e_end - e_begin + NB - 1) / NB;
        const float* xs = p.x + c0;

        // indices of batch q, one entry per lane
        auto load_idx = [&](i32 q, i32& c, float& w) {
            const i32 e = e_begin + q * NB + lane;
            c = -1;
            w = 0.f;
            if (lane < NB && e < e_end) {
                PairEntries{p.ent}.get(e, c, w);
            }
        };
        // start the copies of batch q into its stage
        auto issue = [&](i32 q, i32 c, float w) {
            const int s = q % STAGES;
            const i32 cnt = min(NB, e_end - (e_begin + q * NB));
            const unsigned bar = bar0 + 8 * s;
            __syncwarp();         // every lane has finished reading this stage
            fence_async_proxy();  // ... before the copies of the async proxy may land in it
            if (lane == 0) mbar_expect_tx(bar, (unsigned)cnt * piece);
            if (lane < NB) wts[s * NB + lane] = w;
            __syncwarp();
            if (lane < cnt)
                bulk_copy_g2s(smem_addr(rows + (size_t)s * L::STAGE_BYTES + (size_t)lane * L::SLABB),
                              xs + (i64)c * p.ldx, piece, bar);
        };

        T acc[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] = V::zero();
        i32 cur = 0;  // item being accumulated
        i32 cur_end = __shfl_sync(0xffffffffu, my_end, 0);
        bool alive = true;
        auto flush = [&](i32 i) {  // finish item first + i with what is in acc, then clear acc
            const i32 o = __shfl_sync(0xffffffffu, da.x, i), pr = __shfl_sync(0xffffffffu, da.y, i);
            const i32 pp = __shfl_sync(0xffffffffu, da.z, i), inf = __shfl_sync(0xffffffffu, da.w, i);
            const i32 fp = __shfl_sync(0xffffffffu, db.y, i);
            const float sc = __int_as_float(__shfl_sync(0xffffffffu, db.z, i));
            const float ip = __int_as_float(__shfl_sync(0xffffffffu, db.w, i));
            alive = finish_item<NV, true>(p, slab, first + i, o, pr, pp, inf, fp, sc, ip, acc, ok, c0, lane);
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[v] = V::zero();
        };

        i32 c_nx = -1;
        float w_nx = 0.f;
        i32 issued = 0;
        if (n_batches > 0) {
            load_idx(0, c_nx, w_nx);
            issue(0, c_nx, w_nx);
            issued = 1;
            if (n_batches > 1) load_idx(1, c_nx, w_nx);
        }
        i32 waited = 0;  // batches whose arrival has been consumed
        for (i32 q = 0; q < n_batches && alive; ++q) {
            while (issued < n_batches && issued - q < STAGES) {  // keep the other stages busy
                issue(issued, c_nx, w_nx);
                ++issued;
                if (issued < n_batches) load_idx(issued, c_nx, w_nx);
            }
            const int s = q % STAGES;
            if (!mbar_wait(bar0 + 8 * s, (parity >> s) & 1u, p.status)) {
                alive = false;
                break;
            }
            parity ^= 1u << s;
            waited = q + 1;
            const i32 e0 = e_begin + q * NB;
            const i32 cnt = min(NB, e_end - e0);
            const unsigned char* st = rows + (size_t)s * L::STAGE_BYTES + lane * 16;
            const float* wq = wts + s * NB;
            for (i32 l = 0; l < cnt && alive; ++l) {
                while (e0 + l == cur_end && cur < count - 1 && alive) {  // entry belongs to a later item
                    flush(cur);
                    ++cur;
                    cur_end = __shfl_sync(0xffffffffu, my_end, cur);
                }
                const float w = wq[l];
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    if (ok[v])
                        acc[v] = V::fma(w, *reinterpret_cast<const float4*>(st + (size_t)l * L::SLABB + v * 512),
                                        acc[v]);
            }
        }
        if (!alive) {
            // A wait ran out: the status word is set.  Copies already issued into this warp's
            // shared-memory stages must land before the block may retire and its shared memory
            // be handed on, so every outstanding stage is waited for (bounded) and discarded.
            for (i32 qq = waited; qq < issued; ++qq) {
                const int s2 = qq % STAGES;
                mbar_wait(bar0 + 8 * s2, (parity >> s2) & 1u, p.status);
                parity ^= 1u << s2;
            }
            drain(p, lane);
            return;
        }
        while (cur < count && alive) {  // the last item, and any empty items behind it
            flush(cur);
            ++cur;
        }
        if (!alive) {
            drain(p, lane);
            return;
        }
    }
}

// Plain CSR product (no tree): rows in natural order, one warp per (row, slab), grid-stride.
template <int NV, bool V4>
__global__ void __launch_bounds__(256, (NV >= 4 ? 2 : 3))
    csr_rows_kernel(i32 n_rows, const i32* __restrict__ row_b, const i32* __restrict__ row_e,
                    const i32* __restrict__ col, const float* __restrict__ val,
                    const float* __restrict__ x, i64 ldx, float* __restrict__ y, i64 ldy, i32 f,
                    i32 slab_w, i64 n_units) {
    using V = Vec<V4>;
    using T = typename V::T;
    constexpr int STEP = 32 * V::E;
    const int lane = threadIdx.x & 31;
    const i64 warp = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const i64 n_warps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 u = warp; u < n_units; u += n_warps) {
        const i32 slab = (i32)(u / n_rows);
        const i32 row = (i32)(u - (i64)slab * n_rows);
        const i32 c0 = slab * slab_w;
        const i32 wcols = min(slab_w, f - c0);
        const i32 lane_col = c0 + lane * V::E;
        bool ok[NV];
        T acc[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            ok[v] = (lane * V::E + v * STEP) < wcols;
            acc[v] = V::zero();
        }
        gather_row<NV, V4, (NV == 1 ? 8 : 4)>(CsrEntries{col, val}, __ldg(row_b + row), __ldg(row_e + row), x + lane_col, ldx, ok,
                           acc, lane);
        float* yrow = y + (i64)row * ldy + lane_col;
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (ok[v]) V::st(yrow + v * STEP, acc[v]);
    }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Picks the widest vector form the operands allow and the slab width it covers.
struct Shape {
    bool v4;
    int nv;
    i32 slab_w;
    i32 n_slabs;
};
// Default slab width of the 128-bit path: 128 columns, one 16-byte vector per lane.  One slab of the
// operand (n_labels rows of slab_w floats) is what every row gathers from while that slab is
// processed, and it should stay in L2.  B200's 126 MB L2 is two partitions that each keep their own
// copy of lines read from both dies, so about half of it holds such an operand: at 100 000 rows a
// 256-column slab (102 MB) does not stay, a 128-column slab (51 MB) does, and DRAM traffic halves.
// Measured on B200, 128 columns also win where no slab can stay resident (200 000 - 400 000 rows:
// 0.55 / 0.71 ms against 0.63 / 0.77 ms for 256 columns; 236 000 rows, width 256: 0.307 against
// 0.324 ms): the one-vector form holds eight row fetches per lane in 56 registers and keeps 32 warps
// per SM, the two-vector form four fetches in 72 registers and 24 warps.
constexpr i32 DEFAULT_SLAB = 128;

Shape pick_shape(i32 f, i32 want_slab, bool can_v4) {
    Shape s{};
    s.v4 = can_v4;
    const i32 lane_w = s.v4 ? 128 : 32;  // columns covered by one vector per lane
    i32 slab = want_slab > 0 ? want_slab : (s.v4 ? DEFAULT_SLAB : 64);
    if (s.v4 && (want_slab == 64 || want_slab == 32)) {  // narrow slabs on request: half-warp gather
        s.nv = 1;
        s.slab_w = want_slab;
        s.n_slabs = (f + want_slab - 1) / want_slab;
        return s;
    }
    slab = std::max(lane_w, (slab / lane_w) * lane_w);
    slab = std::min(slab, lane_w * 4);
    const i32 f_up = ((f + lane_w - 1) / lane_w) * lane_w;
    slab = std::min(slab, f_up);
    s.nv = slab / lane_w;
    if (s.nv == 3) {
        s.nv = 2;
        slab = 2 * lane_w;
    }
    s.slab_w = slab;
    s.n_slabs = (f + slab - 1) / slab;
    return s;
}

}  // namespace

// ------------------------------------------------------------------------------------------
// A schedule on the device.
struct DeviceSchedule {
    i32 n_items = 0;   // work items per slab (rows + extra segments of long rows); 0: there is none
    i32 n_prefix = 0;  // items that never wait
    i32 n_partial = 0; // PARTIAL items = scratch slots per slab
    i32 segment = 0;   // entries of a PARTIAL item
    i32 n_chunks = 0;  // 0: not clustered
    i32 n_waits = 0;   // rows with a parent
    i32 depth = 0;
    i64 n_entries = 0;
    std::vector<i32> part_ends;  // see Schedule
    i32 n_partial_coarse = 0;
    RowDesc* d_desc = nullptr;
    Entry* d_ent = nullptr;
    Chunk* d_chunks = nullptr;
};

void free_schedule(const DeviceSchedule& d) {
    cudaFree(d.d_desc);
    cudaFree(d.d_ent);
    cudaFree(d.d_chunks);
}

struct cbm_b200_plan {
    int device = 0;
    i32 n = 0;
    i32 n_labels = 0;  // rows of the dense right-hand side
    i32 n_out = 0;     // rows of the output shard (owned label range)
    i32 n_rows = 0;    // rows actually computed
    // The structure's own schedule, and the one with rows lifted out of the tree (cbm_lift.cpp), which the product in
    // one pass goes by where there is one that pays at `f` columns.  The halves of the product (delta product, update) need
    // the tree itself.
    DeviceSchedule tree, lifted;
    const DeviceSchedule& schedule_for(i32 mode, i32 f) const {
        return mode == MODE_FUSED && lifted.n_items > 0 && !tree_pays(f) ? lifted : tree;
    }
    // Rows are lifted by what entries, waits and levels cost at 128 columns (cbm_lift.cpp).  The more columns, the more the
    // entries count, and a level as much as before: 5 000 rows of 156 entries, of which the tree saves a quarter, 128 columns
    // lifted 30 us, by the tree 37, 256 columns 60 and 51, 1 024 columns 198 and 152; 20 000 rows of 74, a sixth saved, 128
    // columns 56 and 52, 256 113 and 91.  Where rows are short, they have too little to gather while they wait (8 000 rows of 65 in
    // communities, 40 by the tree, 1 024 columns 126 and 187; 5 000 of 37, 13 by the tree, 57 and 82; 100 000 of 40, 36 by the
    // tree, 256 columns 238 and 255), and in community order lifted rows are faster at all widths (17 000 rows of 59, 32
    // by the tree, 1 024 columns 198 and 295).
    bool long_rows() const { return tree.n_entries >= 48 * (i64)n_rows; }
    bool tree_pays(i32 f) const {
        if (lifted.n_chunks > 0 || !long_rows()) return false;
        const i64 slabs = (f + 127) / 128;
        const auto cost = [&](const DeviceSchedule& d) {
            return (d.n_entries + 4 * (i64)d.n_waits) * slabs + (d.depth > 1 ? 25000 * (i64)d.depth : 0);
        };
        return cost(tree) < cost(lifted);
    }
    float* d_scratch = nullptr;
    i64 scratch_cap = 0;
    i64 n_delta = 0;
    i32 n_root_children = 0;
    i32 depth = 0;
    bool normalized = false;
    float* d_pack = nullptr;     // the operand copied to 16-byte aligned rows (when the caller's are not)
    i64 pack_cap = 0;
    i32* d_flags = nullptr;
    i64 flags_cap = 0;
    bool in_pool = false;  // counted among the plans that share the device's workspace pool
    bool captured = false;       // a graph may hold the workspaces' addresses:
    std::vector<void*> retired;  // those that larger ones have replaced since are kept for it
    u64* d_counter = nullptr;
    i32* d_status = nullptr;
    i32 epoch = 0;
    i32 slab_width = 0;
    i32 n_blocks = 0;
    i32 sm_count = 148;
    i64 device_bytes = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    std::vector<cudaEvent_t> events;
    i32 host_chunk = 0;
    i32 form = 0;      // 0 register form, 1 bulk-copy form
    unsigned char* bounce = nullptr;  // page-locked slots that pageable operands pass through
    float* stage_x = nullptr;
    float* stage_y = nullptr;
    i64 stage_x_cap = 0, stage_y_cap = 0;
};

namespace {

struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) ok = cudaSetDevice(dev) == cudaSuccess;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

template <class T>
int upload(T** dst, const T* src, size_t count, i64& bytes) {
    *dst = nullptr;
    const size_t sz = std::max<size_t>(count, 1) * sizeof(T);
    CBM_CUDA(cudaMalloc((void**)dst, sz));
    bytes += (i64)sz;
    if (count) CBM_CUDA(cudaMemcpy(*dst, src, count * sizeof(T), cudaMemcpyHostToDevice));
    return CBM_B200_OK;
}

}  // namespace

namespace {

// The flags, parked sums and packed operands of all plans of a device come from one stream-ordered pool.  A plan
// finds out at its first product how much it needs, and cudaMalloc and cudaFree then take longer than the product
// (50 000 rows of 300 columns: first product on a new plan 0.9 ms with them, 0.2 with the pool).  The pool keeps at most
// POOL_KEEPS bytes that no plan uses, and nothing once the device's last plan is gone.
constexpr u64 POOL_KEEPS = (u64)256 << 20;
constexpr int MAX_POOLS = 64;
struct WorkspacePool {
    cudaMemPool_t pool = nullptr;
    int plans = 0;
};
WorkspacePool g_pools[MAX_POOLS];
std::mutex g_pools_lock;

int pool_enter(int device) {
    if (device < 0 || device >= MAX_POOLS) return cbm::fail(CBM_B200_ERR_ARG, "plan_create: device number out of range");
    std::lock_guard<std::mutex> hold(g_pools_lock);
    WorkspacePool& w = g_pools[device];
    if (!w.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        CBM_CUDA(cudaMemPoolCreate(&pool, &props));
        u64 keeps = POOL_KEEPS;
        const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keeps);
        if (e != cudaSuccess) cudaMemPoolDestroy(pool);
        CBM_CUDA(e);
        w.pool = pool;
    }
    ++w.plans;
    return CBM_B200_OK;
}

void pool_leave(int device) {
    std::lock_guard<std::mutex> hold(g_pools_lock);
    WorkspacePool& w = g_pools[device];
    if (--w.plans == 0) cudaMemPoolTrimTo(w.pool, 0);
}

// Makes a workspace hold `need` elements, its contents lost (zero if `zeroed`).  Any stream may use it afterwards.
template <class T>
int grow(cbm_b200_plan* p, T*& at, i64& cap, i64 need, bool zeroed, cudaStream_t s) {
    if (need <= cap) return CBM_B200_OK;
    if (at && p->captured) {
        try {
            p->retired.push_back(at);
        } catch (const std::bad_alloc&) {
            return cbm::fail(CBM_B200_ERR_ALLOC, "out of host memory");
        }
    } else {
        if (at) {  // a launch in flight may still read the old one, on whatever stream
            CBM_CUDA(cudaDeviceSynchronize());
            CBM_CUDA(cudaFreeAsync(at, s));
        }
        p->device_bytes -= cap * (i64)sizeof(T);
    }
    at = nullptr;
    cap = 0;
    void* fresh = nullptr;
    CBM_CUDA(cudaMallocFromPoolAsync(&fresh, (size_t)need * sizeof(T), g_pools[p->device].pool, s));
    at = (T*)fresh;
    cap = need;
    p->device_bytes += need * (i64)sizeof(T);
    if (zeroed) CBM_CUDA(cudaMemsetAsync(at, 0, (size_t)need * sizeof(T), s));
    CBM_CUDA(cudaStreamSynchronize(s));
    return CBM_B200_OK;
}

}  // namespace

extern "C" void cbm_b200_plan_destroy(cbm_b200_plan* p) {
    if (!p) return;
    DeviceGuard g(p->device);
    if (p->in_pool) {
        cudaDeviceSynchronize();
        for (void* at : {(void*)p->d_pack, (void*)p->d_flags, (void*)p->d_scratch})
            if (at) cudaFreeAsync(at, p->own_stream);
        for (void* at : p->retired) cudaFreeAsync(at, p->own_stream);
        cudaStreamSynchronize(p->own_stream);
        pool_leave(p->device);
    }
    free_schedule(p->tree);
    free_schedule(p->lifted);
    cudaFree(p->d_counter);
    cudaFree(p->d_status);
    cudaFreeHost(p->bounce);
    cudaFree(p->stage_x);
    cudaFree(p->stage_y);
    if (p->own_stream) cudaStreamDestroy(p->own_stream);
    if (p->copy_in) cudaStreamDestroy(p->copy_in);
    if (p->copy_out) cudaStreamDestroy(p->copy_out);
    for (cudaEvent_t e : p->events) cudaEventDestroy(e);
    delete p;
}

namespace {

// The host-side schedule of one plan, before anything touches the device.
struct Schedule {
    std::vector<RowDesc> desc;
    std::unique_ptr<Entry[]> ent;  // not cleared first: the threads that fill it touch its pages
    i64 n_ent = 0;
    std::vector<i64> source;    // per item: its first entry in the delta arrays, or ~ its first in those of the lifted rows
    std::vector<Chunk> chunks;  // clustered plans
    bool clustered = false;
    i32 segment = 0;  // delta entries of a PARTIAL item
    std::vector<i32> part_ends;  // where each split row's PARTIAL items end
    i32 n_partial_coarse = 0;    // how many there would be with rows of more than 192 entries cut at 128
    i64 n_delta = 0;
    i32 n_prefix = 0, n_partial = 0, n_rows_owned = 0, depth = 0, n_root_children = 0, n_labels = 0;
};

// Checks, before any launch, the properties the kernels rely on: items wait only for smaller
// positions (so the in-order claiming cannot deadlock), whoever is waited for publishes, entry
// ranges are consecutive, every output row is produced exactly once and every parked share is
// collected exactly once.
int validate_schedule(const Schedule& sch, i32 n_out) {
    const i32 n_items = (i32)sch.desc.size();
    auto bad = [](const char* what) { return cbm::fail(CBM_B200_ERR_FORMAT, std::string("schedule check: ") + what); };
    if (sch.n_partial > sch.n_prefix || sch.n_prefix > n_items) return bad("prefix bounds");
    std::vector<char> produced((size_t)std::max(n_out, 0), 0), collected((size_t)sch.n_partial, 0);
    i64 cursor = 0;
    for (i32 pos = 0; pos < n_items; ++pos) {
        const RowDesc& d = sch.desc[pos];
        const i32 len = (d.info >> ITEM_LEN_SHIFT) & 0xff;
        const i32 n_part = (i32)((unsigned)d.info >> ITEM_NPART_SHIFT);
        const bool partial = (d.info & ITEM_PARTIAL) != 0;
        if (d.beg != cursor) return bad("entry ranges are not consecutive");
        cursor += sch.clustered ? (len + 1) / 2 * 2 : len;
        if (partial != (pos < sch.n_partial)) return bad("PARTIAL items must fill positions [0, n_partial)");
        if (partial) {
            if (!(d.info & ITEM_PUBLISH) || d.parent_row >= 0 || n_part != 0) return bad("malformed PARTIAL item");
            continue;
        }
        if (d.out_row < 0 || d.out_row >= n_out || produced[d.out_row]) return bad("output row missing or produced twice");
        produced[d.out_row] = 1;
        if (pos < sch.n_prefix && (d.parent_row >= 0 || n_part != 0)) return bad("a prefix item would have to wait");
        if (d.parent_row >= 0) {
            if (d.parent_pos < 0 || d.parent_pos >= pos) return bad("an item waits for a later position");
            const RowDesc& q = sch.desc[d.parent_pos];
            if ((q.info & ITEM_PARTIAL) || !(q.info & ITEM_PUBLISH) || q.out_row != d.parent_row)
                return bad("parent item does not publish the row its child reads");
        }
        if (n_part > 0) {
            if (pos < sch.n_prefix || d.first_part < 0 || d.first_part + n_part > sch.n_partial)
                return bad("parked shares out of range");
            for (i32 k = 0; k < n_part; ++k) {
                if (collected[d.first_part + k]) return bad("a parked share is collected twice");
                collected[d.first_part + k] = 1;
            }
        }
    }
    if (cursor != sch.n_ent) return bad("entries not covered exactly once");
    i32 at = 0;
    for (const Chunk& c : sch.chunks) {
        if (c.first != at || c.count <= 0 || c.count > MAX_CHUNK_ITEMS) return bad("chunks do not follow one another");
        at += c.count;
        const i64 end = at < n_items ? sch.desc[at].beg : cursor;
        if (at > n_items || c.e0 != sch.desc[c.first].beg || c.e0 + c.ne != end || c.ne > CHUNK_ENTRIES)
            return bad("a chunk does not hold its items' entries");
    }
    if (at != (sch.clustered ? n_items : 0)) return bad("items not covered by chunks");
    for (char c : collected)
        if (!c) return bad("a parked share is never collected");
    i32 rows = 0;
    for (char c : produced) rows += c;
    if (rows != sch.n_rows_owned) return bad("owned rows and produced rows differ");
    return CBM_B200_OK;
}

// Cuts a clustered schedule into the chunks that blocks claim.
void make_chunks(Schedule& sch, i32 n_prefix) {
    const i32 n_items = (i32)sch.desc.size();
    auto end_of = [&](i32 i) { return i + 1 < n_items ? sch.desc[i + 1].beg : (i32)sch.n_ent; };
    Chunk c{0, 0, 0, 0};
    for (i32 i = 0; i < n_items; ++i) {
        const i32 most = i < n_prefix ? MAX_CHUNK_ITEMS : MAX_CHUNK_ITEMS / 2;
        if (c.count > 0 && (c.count >= most || i == n_prefix || end_of(i) - c.e0 > CHUNK_ENTRIES)) {
            sch.chunks.push_back(c);
            c.count = 0;
        }
        if (c.count == 0) c = Chunk{i, 0, sch.desc[i].beg, 0};
        ++c.count;
        c.ne = end_of(i) - c.e0;
    }
    if (c.count > 0) sch.chunks.push_back(c);
}

// What a plan is made from, checked: the arrays as the caller has them, and the tree they describe.
struct Structure {
    i32 n = 0, n_labels = 0, own_begin = 0, own_end = 0;
    bool csr = false, square = false;
    const i32 *crow = nullptr, *col = nullptr, *perm = nullptr;
    const float *val = nullptr, *multiplier = nullptr;
    std::vector<i32> parent, level;  // of every row; parent n: the virtual root
    std::vector<i32> rows;           // those the plan computes, breadth-first
    i32 label(i32 v) const { return perm ? perm[v] : v; }
};

// How a schedule is cut and ordered.  As a plan on a GPU is: long rows cut finer where the mean row is short, communities
// looked for on `device` or, for a check without a GPU, given as `labels` (row v belongs to community labels[v]).
struct Rules {
    bool as_plan = false;
    int device = -1;
    const i32* labels = nullptr;
};

// Sorts the rows of a graph with communities by community (rank[v] = place of row v).  Returns false, and leaves
// the rows as they are, where that would not bring row pieces into reach of an SM's L1: in a small graph (X is
// fetched from L2 anyway and a launch is bound by latency), and where about 1 000 consecutive entries of
// the sorted rows still name mostly different columns.  On B200, width 128: rows of 22 entries in
// communities of 55 (ratio 0.4) gain 40 %, rows of 11 in communities of 118 (0.5) gain 15 %; copy-model graphs
// (0.75 - 0.95), whose common columns are few hubs, gain nothing.  Only for square matrices: the search takes a column for the
// row of that number.
bool cluster_order(const Structure& st, const Rules& rules, std::vector<i32>& rank) {
    if (!st.square) return false;
    const i32 n = st.n;
    const i32 *crow = st.crow, *col = st.col;
    std::vector<i32> label;
    if (rules.labels) {
        label.assign(rules.labels, rules.labels + n);
    } else {
        if (rules.device < 0 || n < 16384 || crow[n] < 4 * (i64)n || crow[n] > INT32_MAX - n - 1024) return false;
        label.resize((size_t)n);
        if (!cbm::cluster_rows(n, crow, col, st.parent.data(), rules.device, label.data())) return false;
    }
    // counting sort by label, stable in v
    std::vector<i32> start((size_t)n + 1, 0), sorted((size_t)n);
    for (i32 v = 0; v < n; ++v) ++start[(size_t)label[v] + 1];
    for (i32 l = 0; l < n; ++l) start[l + 1] += start[l];
    for (i32 v = 0; v < n; ++v) sorted[start[label[v]]++] = v;
    // distinct columns among the entries of runs of about 1 000 entries, sampled over the rows
    i64 entries = 0, distinct = 0;
    std::vector<i32> cols;
    const i32 samples = 128;
    for (i32 k = 0; k < samples; ++k) {
        cols.clear();
        for (i64 i = (i64)n * k / samples; i < n && cols.size() < 1024; ++i) {
            const i32 v = sorted[i];
            cols.insert(cols.end(), col + crow[v], col + crow[v + 1]);
        }
        entries += (i64)cols.size();
        std::sort(cols.begin(), cols.end());
        distinct += std::unique(cols.begin(), cols.end()) - cols.begin();
    }
    if (!rules.labels && distinct * 10 > entries * 7) return false;
    rank.resize((size_t)n);
    for (i32 i = 0; i < n; ++i) rank[sorted[i]] = i;
    return true;
}

// csr_cols > 0: a plain CSR matrix with that many columns (no tree: every row hangs off
// the virtual root, mst_row / mst_col / perm are not read); csr_cols == 0: a CBM structure.
int read_structure(int32_t n, const int32_t* mst_row, const int32_t* mst_col, const int32_t* delta_crow,
                   const int32_t* delta_col, const float* delta_val, const float* multiplier,
                   const int32_t* perm, int32_t n_labels, int32_t own_begin, int32_t own_end, int32_t csr_cols, Structure& st) {
    std::vector<i32> flat_row, flat_col;
    if (csr_cols > 0) {
        if (n < 0 || !delta_crow) return cbm::fail(CBM_B200_ERR_ARG, "csr_plan_create: NULL row pointers");
        flat_row.assign((size_t)n + 2, 0);
        flat_row[(size_t)n + 1] = n;
        flat_col.resize((size_t)n);
        for (i32 v = 0; v < n; ++v) flat_col[v] = v;
        mst_row = flat_row.data();
        mst_col = flat_col.data();
        perm = nullptr;
        n_labels = n;  // labels of the rows; the column bound is csr_cols
        own_begin = 0;
        own_end = n;
    }
    if (n < 0 || !mst_row || !delta_crow || (n > 0 && !mst_col))
        return cbm::fail(CBM_B200_ERR_ARG, "plan_create: NULL tree or delta arrays");
    if (n_labels == 0) n_labels = n;
    if (n_labels < n || (!perm && n_labels != n))
        return cbm::fail(CBM_B200_ERR_ARG, "plan_create: n_labels must be >= n (== n without perm)");
    if (own_begin < 0 || own_end > n_labels || own_begin > own_end)
        return cbm::fail(CBM_B200_ERR_ARG, "plan_create: bad owned range");
    const i64 nd_all = delta_crow[n];
    if (nd_all > 0 && (!delta_col || !delta_val))
        return cbm::fail(CBM_B200_ERR_ARG, "plan_create: NULL delta col/val");
    const i32 col_bound = csr_cols > 0 ? csr_cols : n;

    // ---- validate the tree: every row exactly once, reachable from the virtual root ----
    if (mst_row[0] != 0 || mst_row[n + 1] != n)
        return cbm::fail(CBM_B200_ERR_FORMAT, "plan_create: mst_row must run from 0 to n");
    std::vector<i32>& parent = st.parent;
    parent.assign((size_t)n, -1);
    for (i32 u = 0; u <= n; ++u) {
        if (mst_row[u] > mst_row[u + 1])
            return cbm::fail(CBM_B200_ERR_FORMAT, "plan_create: mst_row not monotone");
        for (i32 k = mst_row[u]; k < mst_row[u + 1]; ++k) {
            const i32 v = mst_col[k];
            if (v < 0 || v >= n || parent[v] != -1 || v == u)
                return cbm::fail(CBM_B200_ERR_FORMAT,
                                 "plan_create: mst_col is not a tree over the rows");
            parent[v] = u;
        }
    }
    std::vector<i32> order;  // breadth-first from the virtual root
    order.reserve((size_t)n);
    std::vector<i32>& level = st.level;
    level.assign((size_t)n + 1, 0);
    {
        std::vector<i32> q;
        q.reserve((size_t)n + 1);
        q.push_back(n);
        for (size_t h = 0; h < q.size(); ++h) {
            const i32 u = q[h];
            for (i32 k = mst_row[u]; k < mst_row[u + 1]; ++k) {
                level[mst_col[k]] = level[u] + 1;
                q.push_back(mst_col[k]);
            }
        }
        if ((i32)q.size() != n + 1)
            return cbm::fail(CBM_B200_ERR_FORMAT, "plan_create: tree has a cycle or unreachable rows");
        order.assign(q.begin() + 1, q.end());
    }
    for (i32 v = 0; v < n; ++v) {
        if (delta_crow[v] > delta_crow[v + 1] || delta_crow[v] < 0)
            return cbm::fail(CBM_B200_ERR_FORMAT, "plan_create: delta_crow not monotone");
    }
    for (i64 k = 0; k < nd_all; ++k)
        if (delta_col[k] < 0 || delta_col[k] >= col_bound)
            return cbm::fail(CBM_B200_ERR_FORMAT, "plan_create: delta column out of range");
    if (perm) {
        std::vector<char> seen((size_t)n_labels, 0);
        for (i32 v = 0; v < n; ++v) {
            if (perm[v] < 0 || perm[v] >= n_labels || seen[perm[v]])
                return cbm::fail(CBM_B200_ERR_ARG, "plan_create: perm labels not distinct / in range");
            seen[perm[v]] = 1;
        }
    }
    auto label = [&](i32 v) { return perm ? perm[v] : v; };
    auto owned = [&](i32 v) {
        const i32 l = label(v);
        return l >= own_begin && l < own_end;
    };
    st.rows.reserve((size_t)std::min<i64>(n, own_end - own_begin));
    for (i32 v : order)
        if (owned(v)) {
            const i32 u = parent[v];
            if (u != n && !owned(u))
                return cbm::fail(CBM_B200_ERR_ARG,
                                 "plan_create: owned range cuts a subtree (parent of an owned row "
                                 "is not owned)");
            st.rows.push_back(v);
        }
    st.n = n;
    st.n_labels = csr_cols > 0 ? csr_cols : n_labels;
    st.own_begin = own_begin;
    st.own_end = own_end;
    st.square = col_bound == n;
    st.csr = csr_cols > 0;
    st.crow = delta_crow;
    st.col = delta_col;
    st.val = delta_val;
    st.multiplier = multiplier;
    st.perm = perm;
    return CBM_B200_OK;
}

// The schedule (layout described at RowDesc), its entries aside, of the structure's rows, or with `lift` of the tree with some
// of them lifted; `rank`: their order by community, empty where the graph has none.
int lay_out(const Structure& st, const cbm::Lifted* lift, const std::vector<i32>& rank, const Rules& rules, Schedule& sch) {
    const i32 n = st.n, own_begin = st.own_begin, own_end = st.own_end;
    const std::vector<i32>&parent = lift ? lift->parent : st.parent, &level = lift ? lift->level : st.level;
    const std::vector<i32>& owned_rows = st.rows;
    const float* multiplier = st.multiplier;
    auto label = [&](i32 v) { return st.label(v); };
    auto row_len = [&](i32 v) { return lift ? lift->len[v] : st.crow[v + 1] - st.crow[v]; };
    const i64 nd_all = lift ? lift->n_entries : st.crow[n], nd_rows = lift ? (i64)owned_rows.size() : n;
    // Delta entries per item of a split row, and the length from which rows are split.  Rows of a plan are cut finer where
    // the mean row is short: a long row is then what a product ends on (100 000 rows of 31 entries, 500 columns: 397 us with
    // segments of 128, 390 with 64, 429 with 32; 50 000 rows, 64 columns: 56, 48, 50); where long rows are the rule, finer
    // segments only add parked sums (40 000 rows of 152 entries: 194 us, 201, 234).
    i32 longest = 0;
    for (i32 v = 0; v < n; ++v) longest = std::max(longest, row_len(v));
    const bool fine = rules.as_plan && nd_all <= 64 * nd_rows && longest <= 64 * 0xffff;
    const i32 SEG = fine ? 64 : 128, SPLIT_OVER = fine ? 96 : 192;
    auto is_split = [&](i32 v) { return row_len(v) > SPLIT_OVER; };
    std::vector<RowDesc>& desc = sch.desc;
    sch.clustered = !rank.empty();
    sch.segment = SEG;
    // items get their entry ranges only: the entries are filled in afterwards
    sch.source.reserve((size_t)n);
    auto append_entries = [&](i32 v, i32 from, i32 to) {  // entries [from, to) of row v
        const i32 beg = (i32)sch.n_ent;
        const i64 at = (lift ? lift->at[v] : st.crow[v]) + from;
        sch.source.push_back(lift && lift->lifted[v] ? ~at : at);
        sch.n_ent += to - from;
        if (sch.clustered) sch.n_ent += sch.n_ent % 2;
        return beg;
    };
    for (i32 v : owned_rows) sch.n_delta += row_len(v);
    // 1. PARTIAL items of every split row, the rows with most of them first (a product that cannot park all of them parks
    // those of the longest rows)
    std::vector<i32> first_part((size_t)n, -1), split_rows;
    for (i32 v : owned_rows)
        if (is_split(v)) split_rows.push_back(v);
    std::stable_sort(split_rows.begin(), split_rows.end(), [&](i32 a, i32 b) { return (row_len(a) - 1) / SEG > (row_len(b) - 1) / SEG; });
    for (i32 v : split_rows) {
        if (row_len(v) > 192) sch.n_partial_coarse += (row_len(v) - 1) / 128;
        const i32 n_part = (row_len(v) + SEG - 1) / SEG - 1;
        if (n_part > 0xffff)
            return cbm::fail(CBM_B200_ERR_ARG, "plan_create: a row has more than 8388480 delta entries");
        first_part[v] = (i32)desc.size();
        for (i32 k = 0; k < n_part; ++k) {
            RowDesc q{};
            q.out_row = 0;
            q.parent_row = -1;
            q.parent_pos = -1;
            q.info = ITEM_PARTIAL | ITEM_PUBLISH | (SEG << ITEM_LEN_SHIFT);
            q.beg = append_entries(v, k * SEG, (k + 1) * SEG);
            q.first_part = -1;
            q.scale = 1.0f;
            q.inv_parent = 1.0f;
            desc.push_back(q);
        }
        sch.part_ends.push_back((i32)desc.size());
    }
    const i32 n_partial = (i32)desc.size();
    // 2. unsplit children of the virtual root, longest first
    std::vector<i32> pos_of((size_t)n, -1);
    i32 depth = 0, n_root_children = 0;
    auto add_row_item = [&](i32 v) {
        const i32 u = parent[v];
        const i32 len = row_len(v);
        const i32 n_part = is_split(v) ? (len + SEG - 1) / SEG - 1 : 0;
        RowDesc d{};
        d.out_row = label(v) - own_begin;
        d.parent_row = (u == n) ? -1 : label(u) - own_begin;
        d.parent_pos = (u == n) ? -1 : pos_of[u];
        d.beg = append_entries(v, n_part * SEG, len);
        d.info = ((len - n_part * SEG) << ITEM_LEN_SHIFT) | (n_part << ITEM_NPART_SHIFT);
        d.first_part = first_part[v];
        d.scale = multiplier ? multiplier[v] : 1.0f;
        d.inv_parent = (multiplier && u != n) ? 1.0f / multiplier[u] : 1.0f;
        pos_of[v] = (i32)desc.size();
        if (u != n) desc[pos_of[u]].info |= ITEM_PUBLISH;
        else ++n_root_children;
        depth = std::max(depth, level[v]);
        desc.push_back(d);
    };
    {
        std::vector<i32> easy;
        for (i32 v : owned_rows)
            if (parent[v] == n && !is_split(v)) easy.push_back(v);
        if (sch.clustered)  // the few long rows first, then community by community
            std::sort(easy.begin(), easy.end(), [&](i32 a, i32 b) {
                const i32 la = row_len(a) > 64 ? row_len(a) : 0, lb = row_len(b) > 64 ? row_len(b) : 0;
                return la != lb ? la > lb : rank[a] < rank[b];
            });
        else
            {   // counting sort, stable
                std::vector<i32> place((size_t)SPLIT_OVER + 2, 0), sorted(easy.size());
                for (i32 v : easy) ++place[(size_t)(SPLIT_OVER - row_len(v)) + 1];
                for (i32 l = 0; l <= SPLIT_OVER; ++l) place[l + 1] += place[l];
                for (i32 v : easy) sorted[(size_t)place[(size_t)(SPLIT_OVER - row_len(v))]++] = v;
                easy.swap(sorted);
            }
        for (i32 v : easy) add_row_item(v);
    }
    const i32 n_prefix = (i32)desc.size();
    // 3. everything that may wait, breadth-first: finishing items of split rows, rows with a parent
    std::vector<i32> rest;
    for (i32 v : owned_rows)
        if (parent[v] != n || is_split(v)) rest.push_back(v);
    if (sch.clustered)  // level by level, so that parents stay in front of their children
        std::sort(rest.begin(), rest.end(), [&](i32 a, i32 b) {
            return level[a] != level[b] ? level[a] < level[b] : rank[a] < rank[b];
        });
    else if (lift)  // (lifting has changed levels)
        std::stable_sort(rest.begin(), rest.end(), [&](i32 a, i32 b) { return level[a] < level[b]; });
    for (i32 v : rest) add_row_item(v);
    if (sch.clustered) make_chunks(sch, n_prefix);
    sch.n_rows_owned = (i32)owned_rows.size();
    sch.n_prefix = n_prefix;
    sch.n_partial = n_partial;
    sch.depth = depth;
    sch.n_root_children = n_root_children;
    sch.n_labels = st.n_labels;
    return validate_schedule(sch, own_end - own_begin);
}

// The entries of a schedule, on several threads.
void fill_entries(const Structure& st, const cbm::Lifted* lift, Schedule& sch) {
    sch.ent.reset(new Entry[(size_t)std::max<i64>(sch.n_ent, 1)]);
    const i32 n_items = (i32)sch.desc.size();
    // (half of the threads: those that have finished spin for a while, beside the caller's first product)
    const int threads = (int)std::max<i64>(1, std::min<i64>(omp_get_max_threads() / 2, sch.n_ent / 100000));
#pragma omp parallel for schedule(static) num_threads(threads)
    for (i32 i = 0; i < n_items; ++i) {
        const i32 len = (sch.desc[i].info >> ITEM_LEN_SHIFT) & 0xff;
        Entry* e = sch.ent.get() + sch.desc[i].beg;
        const bool own = sch.source[i] >= 0;
        const i32* col = own ? st.col + sch.source[i] : lift->col.data() + ~sch.source[i];
        const float* val = own ? st.val + sch.source[i] : lift->val.data() + ~sch.source[i];
        for (i32 k = 0; k < len; ++k) e[k] = Entry{st.label(col[k]), val[k]};
        if (sch.clustered && len % 2) e[len] = Entry{0, 0.0f};
    }
    std::vector<i64>().swap(sch.source);
}

int build_schedule(const Structure& st, const cbm::Lifted* lift, const std::vector<i32>& rank, const Rules& rules, Schedule& sch) {
    const int rc = lay_out(st, lift, rank, rules, sch);
    if (rc == CBM_B200_OK) fill_entries(st, lift, sch);
    return rc;
}

// Runs both, side by side if `wide` and a thread can be had, and lets the first one's exception out before the other's.
// The second one opens no team of threads: OpenMP would keep another for it, and ends the process where it cannot.
template <class F, class G>
void run_both(bool wide, F first, G second) {
    std::exception_ptr first_thrown, second_thrown;
    const auto guarded_second = [&] {
        try {
            second();
        } catch (...) {
            second_thrown = std::current_exception();
        }
    };
    std::thread beside;
    if (wide) {
        try {
            beside = std::thread(guarded_second);
        } catch (const std::system_error&) {  // no thread to be had
        }
    }
    try {
        first();
    } catch (...) {
        first_thrown = std::current_exception();
    }
    if (beside.joinable()) beside.join();
    else if (!first_thrown) guarded_second();
    if (first_thrown) std::rethrow_exception(first_thrown);
    if (second_thrown) std::rethrow_exception(second_thrown);
}

int build_both(const Structure& st, const Rules& rules, Schedule& tree, Schedule& lifted) {
    cbm::Lifted lift;
    std::vector<i32> rank;
    const bool wide = st.crow[st.n] > 1000000;  // steps of milliseconds
    // A thread begins on the first device: it goes to the caller's, which it leaves as the current one, so that no other
    // GPU gets a context.
    int current = -1;
    if (rules.device >= 0 && cudaGetDevice(&current) != cudaSuccess) current = -1;
    run_both(
        wide,
        [&] {
            if (!st.csr) cbm::lift_rows(st.n, st.rows, st.parent, st.level, st.crow, st.col, st.val, lift);
        },
        [&] {
            if (current >= 0) cudaSetDevice(current);
            cluster_order(st, rules, rank);
        });
    if (lift.n_lifted == 0) return build_schedule(st, nullptr, rank, rules, tree);
    int rc = CBM_B200_OK, rc_lifted = CBM_B200_OK;
    run_both(
        wide, [&] { rc = build_schedule(st, nullptr, rank, rules, tree); },
        [&] { rc_lifted = lay_out(st, &lift, rank, rules, lifted); });
    if (rc) return rc;
    if (rc_lifted) lifted = Schedule();
    else fill_entries(st, &lift, lifted);
    return CBM_B200_OK;
}

// The structure's own schedule, and the one with rows lifted out of the tree where that pays, can be made and has memory:
// the product can do without it.
int build_schedules(const Structure& st, const Rules& rules, Schedule& tree, Schedule& lifted) {
    try {
        return build_both(st, rules, tree, lifted);
    } catch (const std::bad_alloc&) {
    } catch (const std::length_error&) {
    }
    tree = Schedule();
    lifted = Schedule();
    std::vector<i32> rank;
    cluster_order(st, rules, rank);
    return build_schedule(st, nullptr, rank, rules, tree);
}

}  // namespace

namespace {
// Runs what may allocate host memory: no exception leaves the library.
template <class F>
int guarded(const char* who, F run) {
    try {
        return run();
    } catch (const std::bad_alloc&) {
        return cbm::fail(CBM_B200_ERR_ALLOC, std::string(who) + ": out of host memory");
    } catch (const std::length_error&) {
        return cbm::fail(CBM_B200_ERR_ALLOC, std::string(who) + ": out of host memory");
    }
}
}  // namespace

extern "C" int cbm_b200_schedule_info(int32_t n, const int32_t* mst_row, const int32_t* mst_col,
                                      const int32_t* delta_crow, const int32_t* delta_col,
                                      const float* delta_val, const float* multiplier,
                                      const int32_t* perm, int32_t n_labels, int32_t own_begin,
                                      int32_t own_end, int32_t* n_items, int32_t* n_prefix,
                                      int32_t* n_partial, int32_t* n_rows) {
    Schedule sch;
    const int rc = guarded("schedule_info", [&] {
        Structure st;
        const int bad = read_structure(n, mst_row, mst_col, delta_crow, delta_col, delta_val, multiplier, perm, n_labels, own_begin,
                                       own_end, 0, st);
        return bad ? bad : build_schedule(st, nullptr, {}, Rules(), sch);
    });
    if (rc) return rc;
    if (n_items) *n_items = (i32)sch.desc.size();
    if (n_prefix) *n_prefix = sch.n_prefix;
    if (n_partial) *n_partial = sch.n_partial;
    if (n_rows) *n_rows = sch.n_rows_owned;
    return CBM_B200_OK;
}

namespace {
// FNV-1a over the items in their order, 8 bytes at a time.
uint64_t fingerprint_of(const RowDesc* desc, size_t n) {
    static_assert(sizeof(RowDesc) == 32, "four words an item");
    uint64_t h = 0xcbf29ce484222325ull;
    for (size_t i = 0; i < n; ++i) {
        uint64_t w[4];
        std::memcpy(w, desc + i, sizeof(w));
        for (uint64_t v : w) h = (h ^ v) * 0x100000001b3ull;
    }
    return h;
}
}  // namespace

namespace {
// The schedule of a whole matrix in its own order by the rules of a plan; csr_cols as for read_structure.
int schedule_as_planned(const char* who, int32_t n, const int32_t* mst_row, const int32_t* mst_col, const int32_t* crow,
                        const int32_t* col, const float* val, const float* multiplier, int32_t csr_cols, const int32_t* labels,
                        int32_t* n_items, int32_t* n_prefix, int32_t* n_partial, int32_t* n_chunks, int32_t* segment,
                        uint64_t* fingerprint) {
    for (i32 v = 0; labels && v < n; ++v)
        if (labels[v] < 0 || labels[v] >= n) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": label out of range");
    Schedule sch;
    const int rc = guarded(who, [&] {
        Structure st;
        const int bad = read_structure(n, mst_row, mst_col, crow, col, val, multiplier, nullptr, 0, 0, n, csr_cols, st);
        if (bad) return bad;
        const Rules rules{true, -1, labels};
        std::vector<i32> rank;
        cluster_order(st, rules, rank);
        return build_schedule(st, nullptr, rank, rules, sch);
    });
    if (rc) return rc;
    if (n_items) *n_items = (i32)sch.desc.size();
    if (n_prefix) *n_prefix = sch.n_prefix;
    if (n_partial) *n_partial = sch.n_partial;
    if (n_chunks) *n_chunks = (i32)sch.chunks.size();
    if (segment) *segment = sch.segment;
    if (fingerprint) *fingerprint = fingerprint_of(sch.desc.data(), sch.desc.size());
    return CBM_B200_OK;
}
}  // namespace

extern "C" int cbm_b200_schedule_as_planned(int32_t n, const int32_t* mst_row, const int32_t* mst_col,
                                            const int32_t* delta_crow, const int32_t* delta_col,
                                            const float* delta_val, const float* multiplier,
                                            const int32_t* labels, int32_t* n_items, int32_t* n_prefix,
                                            int32_t* n_partial, int32_t* n_chunks, int32_t* segment,
                                            uint64_t* fingerprint) {
    return schedule_as_planned("schedule_as_planned", n, mst_row, mst_col, delta_crow, delta_col, delta_val, multiplier, 0, labels,
                               n_items, n_prefix, n_partial, n_chunks, segment, fingerprint);
}

extern "C" int cbm_b200_csr_schedule_as_planned(int32_t n_rows, int32_t n_cols, const int32_t* crow, const int32_t* col,
                                                const float* val, const int32_t* labels, int32_t* n_items,
                                                int32_t* n_prefix, int32_t* n_partial, int32_t* n_chunks,
                                                int32_t* segment, uint64_t* fingerprint) {
    if (n_cols <= 0) return cbm::fail(CBM_B200_ERR_ARG, "csr_schedule_as_planned: n_cols must be positive");
    return schedule_as_planned("csr_schedule_as_planned", n_rows, nullptr, nullptr, crow, col, val, nullptr, n_cols, labels, n_items,
                               n_prefix, n_partial, n_chunks, segment, fingerprint);
}

extern "C" int cbm_b200_schedule_lifted(int32_t n, const int32_t* mst_row, const int32_t* mst_col, const int32_t* delta_crow,
                                        const int32_t* delta_col, const float* delta_val, const float* multiplier,
                                        const int32_t* labels, int32_t* n_lifted, int32_t* parent, int64_t* crow,
                                        int64_t capacity, int32_t* col, float* val) {
    for (i32 v = 0; labels && v < n; ++v)
        if (labels[v] < 0 || labels[v] >= n) return cbm::fail(CBM_B200_ERR_ARG, "schedule_lifted: label out of range");
    if (capacity > 0 && (!crow || !col || !val)) return cbm::fail(CBM_B200_ERR_ARG, "schedule_lifted: NULL array");
    return guarded("schedule_lifted", [&] {
        Structure st;
        Schedule tree, lifted;
        int rc = read_structure(n, mst_row, mst_col, delta_crow, delta_col, delta_val, multiplier, nullptr, 0, 0, n, 0, st);
        if (rc == CBM_B200_OK) rc = build_schedules(st, Rules{true, -1, labels}, tree, lifted);
        if (rc) return rc;
        // read back from the items, as a product walks over them
        const Schedule& sch = lifted.desc.empty() ? tree : lifted;
        std::vector<const RowDesc*> item((size_t)n, nullptr);
        for (size_t i = (size_t)sch.n_partial; i < sch.desc.size(); ++i) item[sch.desc[i].out_row] = &sch.desc[i];
        const auto len_of = [](const RowDesc& d) { return (d.info >> ITEM_LEN_SHIFT) & 0xff; };
        i64 at = 0;
        i32 differ = 0;
        for (i32 v = 0; v < n; ++v) {
            const RowDesc& d = *item[v];
            const i32 parts = (i32)((unsigned)d.info >> ITEM_NPART_SHIFT);
            if (parent) parent[v] = d.parent_row < 0 ? n : d.parent_row;
            differ += (d.parent_row < 0 ? n : d.parent_row) != st.parent[v];
            if (crow) crow[v] = at;
            for (i32 k = 0; k <= parts; ++k) {
                const RowDesc& q = k < parts ? sch.desc[d.first_part + k] : d;
                for (i32 e = 0; e < len_of(q); ++e, ++at)
                    if (at < capacity) {
                        col[at] = sch.ent[(size_t)q.beg + e].col;
                        val[at] = sch.ent[(size_t)q.beg + e].val;
                    }
            }
        }
        if (crow) crow[n] = at;
        if (n_lifted) *n_lifted = differ;
        return (int)CBM_B200_OK;
    });
}

namespace {
int plan_from_schedules(Schedule& tree, Schedule& lifted, int32_t n, int32_t n_out, bool normalized, int32_t device,
                        cbm_b200_plan** out);
}

extern "C" int cbm_b200_plan_create(int32_t n, const int32_t* mst_row, const int32_t* mst_col,
                                    const int32_t* delta_crow, const int32_t* delta_col,
                                    const float* delta_val, const float* multiplier,
                                    const int32_t* perm, int32_t n_labels, int32_t own_begin,
                                    int32_t own_end, int32_t device, cbm_b200_plan** out) {
    if (!out) return cbm::fail(CBM_B200_ERR_ARG, "plan_create: out is NULL");
    *out = nullptr;
    Schedule tree, lifted;
    const int rc0 = guarded("plan_create", [&] {
        Structure st;
        const int bad = read_structure(n, mst_row, mst_col, delta_crow, delta_col, delta_val, multiplier, perm, n_labels, own_begin,
                                       own_end, 0, st);
        return bad ? bad : build_schedules(st, Rules{true, device, nullptr}, tree, lifted);
    });
    if (rc0) return rc0;
    return plan_from_schedules(tree, lifted, n, own_end - own_begin, multiplier != nullptr, device, out);
}

extern "C" int cbm_b200_csr_plan_create(int32_t n_rows, int32_t n_cols, const int32_t* crow,
                                        const int32_t* col, const float* val, int32_t device,
                                        cbm_b200_plan** out) {
    if (!out) return cbm::fail(CBM_B200_ERR_ARG, "csr_plan_create: out is NULL");
    *out = nullptr;
    if (n_cols <= 0) return cbm::fail(CBM_B200_ERR_ARG, "csr_plan_create: n_cols must be positive");
    Schedule rows, none;
    const int rc0 = guarded("csr_plan_create", [&] {
        Structure st;
        const int bad = read_structure(n_rows, nullptr, nullptr, crow, col, val, nullptr, nullptr, 0, 0, 0, n_cols, st);
        return bad ? bad : build_schedules(st, Rules{true, device, nullptr}, rows, none);
    });
    if (rc0) return rc0;
    return plan_from_schedules(rows, none, n_rows, n_rows, false, device, out);
}

namespace {
int upload_schedule(Schedule& sch, DeviceSchedule& d, i64& bytes) {
    d.n_items = (i32)sch.desc.size();
    d.n_prefix = sch.n_prefix;
    d.n_partial = sch.n_partial;
    d.segment = sch.segment;
    d.part_ends.swap(sch.part_ends);
    d.n_partial_coarse = sch.n_partial_coarse;
    d.n_entries = sch.n_delta;
    d.n_waits = sch.n_rows_owned - sch.n_root_children;
    d.depth = sch.depth;
    d.n_chunks = (i32)sch.chunks.size();
    int rc = upload(&d.d_desc, sch.desc.data(), sch.desc.size(), bytes);
    if (rc == CBM_B200_OK) rc = upload(&d.d_ent, sch.ent.get(), (size_t)sch.n_ent, bytes);
    if (rc == CBM_B200_OK && sch.clustered) rc = upload(&d.d_chunks, sch.chunks.data(), sch.chunks.size(), bytes);
    return rc;
}

int plan_from_schedules(Schedule& tree, Schedule& lifted, int32_t n, int32_t n_out, bool normalized, int32_t device,
                        cbm_b200_plan** out) {
    int n_dev = 0;
    CBM_CUDA(cudaGetDeviceCount(&n_dev));
    if (device < 0 || device >= n_dev)
        return cbm::fail(CBM_B200_ERR_ARG, "plan_create: no such CUDA device");
    DeviceGuard guard(device);
    if (!guard.ok) return cbm::fail(CBM_B200_ERR_CUDA, "plan_create: cudaSetDevice failed");

    cbm_b200_plan* p = new (std::nothrow) cbm_b200_plan();
    if (!p) return cbm::fail(CBM_B200_ERR_ALLOC, "plan_create: out of host memory");
    p->device = device;
    p->n = n;
    p->n_labels = tree.n_labels;
    p->n_out = n_out;
    p->n_rows = tree.n_rows_owned;
    p->n_delta = tree.n_delta;
    p->n_root_children = tree.n_root_children;
    p->depth = tree.depth;
    p->normalized = normalized;
    int sms = 0;  // (the one attribute: all properties together take milliseconds)
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess) p->sm_count = sms;
    int rc = upload_schedule(tree, p->tree, p->device_bytes);
    const i64 tree_bytes = p->device_bytes;
    const auto without_lifted = [&] {  // the plan does without that schedule where the device has no room for it
        free_schedule(p->lifted);
        cudaGetLastError();
        p->lifted = DeviceSchedule();
        p->device_bytes = tree_bytes;
    };
    if (rc == CBM_B200_OK && !lifted.desc.empty() && upload_schedule(lifted, p->lifted, p->device_bytes) != CBM_B200_OK) without_lifted();
    if (rc == CBM_B200_OK) {
        cudaError_t e = cudaMalloc((void**)&p->d_counter, sizeof(u64));
        if (e == cudaSuccess) e = cudaMemset(p->d_counter, 0, sizeof(u64));
        if (e == cudaSuccess) e = cudaMalloc((void**)&p->d_status, sizeof(i32));
        if (e == cudaSuccess) e = cudaMemset(p->d_status, 0, sizeof(i32));
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p->own_stream, cudaStreamNonBlocking);
        if (e != cudaSuccess)
            rc = cbm::fail(CBM_B200_ERR_CUDA, std::string("plan_create: ") + cudaGetErrorString(e));
        p->device_bytes += 16;
    }
    if (rc == CBM_B200_OK) {
        rc = pool_enter(device);
        p->in_pool = rc == CBM_B200_OK;
    }
    // ready flags for operands of up to 512 columns and parked sums for one slab: most products then allocate nothing
    const auto first_room = [&] {
        const int bad = grow(p, p->d_flags, p->flags_cap, 4 * (i64)std::max(p->tree.n_items, p->lifted.n_items), true, p->own_stream);
        return bad ? bad : grow(p, p->d_scratch, p->scratch_cap, (i64)std::max(p->tree.n_partial, p->lifted.n_partial) * DEFAULT_SLAB, false, p->own_stream);
    };
    if (rc == CBM_B200_OK) rc = first_room();
    if (rc != CBM_B200_OK && p->in_pool && p->lifted.n_items > 0) {
        const i64 beside = p->flags_cap * (i64)sizeof(i32) + p->scratch_cap * (i64)sizeof(float) + 16;
        without_lifted();
        p->device_bytes += beside;
        rc = first_room();
    }
    if (rc != CBM_B200_OK) {
        const std::string keep = cbm::last_error_slot();
        cbm_b200_plan_destroy(p);
        cbm::last_error_slot() = keep;
        return rc;
    }
    *out = p;
    return CBM_B200_OK;
}
}  // namespace

extern "C" int cbm_b200_plan_info(const cbm_b200_plan* p, int32_t* n_rows, int64_t* n_delta,
                                  int32_t* n_root_children, int32_t* depth,
                                  int64_t* device_bytes) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, "plan_info: NULL plan");
    if (n_rows) *n_rows = p->n_rows;
    if (n_delta) *n_delta = p->n_delta;
    if (n_root_children) *n_root_children = p->n_root_children;
    if (depth) *depth = p->depth;
    if (device_bytes) *device_bytes = p->device_bytes;
    return CBM_B200_OK;
}

namespace {
int schedule_of(const cbm_b200_plan* p, const DeviceSchedule& d, int32_t* n_items, int32_t* n_prefix, int32_t* n_partial,
                int32_t* n_chunks, int32_t* segment, uint64_t* fingerprint) {
    if (n_items) *n_items = d.n_items;
    if (n_prefix) *n_prefix = d.n_prefix;
    if (n_partial) *n_partial = d.n_partial;
    if (n_chunks) *n_chunks = d.n_chunks;
    if (segment) *segment = d.segment;
    if (fingerprint) {
        DeviceGuard g(p->device);
        std::unique_ptr<RowDesc[]> desc(new (std::nothrow) RowDesc[(size_t)d.n_items]);
        if (!desc) return cbm::fail(CBM_B200_ERR_ALLOC, "plan_schedule: out of host memory");
        if (d.n_items) CBM_CUDA(cudaMemcpy(desc.get(), d.d_desc, (size_t)d.n_items * sizeof(RowDesc), cudaMemcpyDeviceToHost));
        *fingerprint = fingerprint_of(desc.get(), (size_t)d.n_items);
    }
    return CBM_B200_OK;
}
}  // namespace

extern "C" int cbm_b200_plan_schedule(const cbm_b200_plan* p, int32_t* n_items, int32_t* n_prefix, int32_t* n_partial,
                                      int32_t* n_chunks, int32_t* segment, uint64_t* fingerprint) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, "plan_schedule: NULL plan");
    return schedule_of(p, p->tree, n_items, n_prefix, n_partial, n_chunks, segment, fingerprint);
}

extern "C" int cbm_b200_plan_product_schedule(const cbm_b200_plan* p, int32_t f, int32_t* n_items, int32_t* n_prefix,
                                              int32_t* n_partial, int32_t* n_chunks, int32_t* segment, uint64_t* fingerprint) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, "plan_product_schedule: NULL plan");
    if (f <= 0) return cbm::fail(CBM_B200_ERR_ARG, "plan_product_schedule: f must be positive");
    return schedule_of(p, p->schedule_for(MODE_FUSED, f), n_items, n_prefix, n_partial, n_chunks, segment, fingerprint);
}

extern "C" int cbm_b200_plan_tune(cbm_b200_plan* p, int32_t slab_width, int32_t n_blocks,
                                  int32_t host_chunk, int32_t form) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, "plan_tune: NULL plan");
    if (slab_width < 0 || n_blocks < 0 || host_chunk < 0 || form < 0 || form > 1)
        return cbm::fail(CBM_B200_ERR_ARG, "plan_tune: knob out of range");
    if (host_chunk % 4 != 0) return cbm::fail(CBM_B200_ERR_ARG, "plan_tune: host_chunk must be a multiple of 4");
    p->form = form;
    p->slab_width = slab_width;
    p->n_blocks = n_blocks;
    p->host_chunk = host_chunk;
    return CBM_B200_OK;
}

extern "C" int cbm_b200_plan_status(cbm_b200_plan* p, void* stream) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, "plan_status: NULL plan");
    DeviceGuard g(p->device);
    CBM_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    i32 st = 0;
    CBM_CUDA(cudaMemcpy(&st, p->d_status, sizeof(st), cudaMemcpyDeviceToHost));
    if (st != 0) {
        CBM_CUDA(cudaMemset(p->d_status, 0, sizeof(i32)));
        return cbm::fail(CBM_B200_ERR_TIMEOUT,
                         "a bounded wait for a parent row ran out; the last product is invalid");
    }
    return CBM_B200_OK;
}

namespace {

int check_dense(const char* who, const void* x, i64 ldx, const void* y, i64 ldy, i32 f) {
    if (f <= 0) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": f must be positive");
    if (!y || ldy < f) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": bad y / ldy");
    if (x && ldx < f) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": ldx < f");
    if (ldx > INT32_MAX || ldy > INT32_MAX)
        return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": leading dimension exceeds 2^31-1");
    if (x && x == y) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": x and y alias");
    return CBM_B200_OK;
}

// How one product is cut into claims and which kernel form runs it.
struct LaunchCfg {
    Shape sh{};
    int tma = 0;       // 0: register form; otherwise the bulk-copy form (variant number)
    i32 group = 1;     // prefix items per claim
    bool one_round = false;  // every warp draws once, and does everything there is for it to do
    i32 n_pclaims = 0, claims_per_slab = 0;
    i64 n_claims = 0;
    bool chunked = false;      // the clustered plan's kernel
    i64 need_flags = 0;        // int32 words
    i64 need_scratch = 0;      // floats
    i64 need_pack = 0;         // floats
    bool in_turn = false;      // see KParams
    bool pack = false;         // the operand is first copied to 16-byte aligned rows
    bool ragged = false;       // 16-byte fetches, but rows of y are not aligned or end inside a vector
    i32 left_out = 0;          // PARTIAL items, the last ones, that the finishing items do themselves
};

// Blocks of 256 threads that an SM holds of the kernel a product runs, see launch_regs and launch_narrow.
constexpr int resident_regs(int nv, bool v4, bool ragged) { return nv == 1 ? (v4 ? (ragged ? 5 : 6) : 4) : (nv == 2 ? 3 : 2); }
constexpr int NARROW_RESIDENT = 6;
int resident_blocks(const Shape& sh, i32 f, bool ragged, int mode) {
    return sh.v4 && sh.nv == 1 && f <= 64 && mode != MODE_UPDATE_ONLY ? NARROW_RESIDENT : resident_regs(sh.nv, sh.v4, ragged);
}

// A product that the resident warps can do in one round draws no second claim: every warp takes its share of the
// prefix, and as long as few items wait (a quarter of the warps) one of those or none.  1 000 rows, 16 columns 8.2 ->
// 6.2 us, 4 096 rows, 500 columns (two or three items a warp) 32.0 -> 22.0.
// Returns the items of the prefix that a warp takes, 0 where one round does not do: an operand so wide that there are more
// slabs than warps has some left over even with all of a slab's prefix to one warp.
i32 one_round_group(i32 n_prefix, i32 n_waiting, i64 n_slabs, i64 warps) {
    const i64 waiting = n_waiting * n_slabs;
    if (waiting >= warps / 4) return 0;
    const i64 per_slab = (warps - waiting) / n_slabs;  // warps for a slab's prefix
    return per_slab == 0 ? 0 : (i32)((n_prefix + per_slab - 1) / per_slab);
}

int plan_cfg(const cbm_b200_plan* p, const DeviceSchedule& d, const char* who, const float* x, i64 ldx, const float* y, i64 ldy,
             i32 f, int mode, bool may_pack, bool in_turn, LaunchCfg& c) {
    c = LaunchCfg{};  // (it may hold what was found for another schedule)
    const bool y_vec = ldy % 4 == 0 && aligned16(y);
    const bool x_vec = ldx % 4 == 0 && aligned16(x) && ldx < (i64)1 << 30;
    // An operand whose rows are not 16-byte aligned can only be fetched 4 bytes a lane, at less than half
    // the rate (4.4 TB/s).  Copying it to aligned rows first costs a launch and one pass over it, about 5 us on a small
    // operand, so it pays when every operand row is fetched several times and the 4-byte fetches would take
    // some 15 us (16 M multiply-adds).
    c.pack = may_pack && mode != MODE_UPDATE_ONLY && !x_vec && f > 4 && d.n_entries >= 4 * (i64)p->n_labels &&
             d.n_entries * f >= (i64)1 << 24;
    c.in_turn = in_turn;
    const bool can_v4 = !in_turn && (mode == MODE_UPDATE_ONLY ? y_vec : x_vec || c.pack);
    c.ragged = can_v4 && (!y_vec || f % 4 != 0);
    int tma = p->form;
    if (!can_v4 || c.ragged || c.pack || mode == MODE_UPDATE_ONLY || d.n_chunks > 0) tma = 0;
    c.tma = tma;
    // Slabs of up to 64 columns gain nothing from the clustered order on large graphs (235 868 rows of 11 entries, 64
    // columns: 106 us against 97): several entries share a fetch there, and what a row costs is its instructions.
    // On smaller graphs the saved round trips per row still win, the more rows wait: 64 columns, few waiting rows, 17 000
    // rows 22 us against 32, 45 000 34 against 34, 60 000 41 against 39; three quarters waiting, 17 000 39 against 45,
    // 50 000 60 against 68.
    c.chunked = d.n_chunks > 0 && can_v4 && mode != MODE_UPDATE_ONLY && (f > 64 || p->n_rows <= 65536) &&
                (p->slab_width == 0 || p->slab_width >= 128);
    if (c.chunked) {
        c.sh.v4 = true;
        c.sh.nv = 1;
        c.sh.slab_w = 128;
        c.sh.n_slabs = (f + c.sh.slab_w - 1) / c.sh.slab_w;
        // One chunk to a claim.  Four of them, up to the last quarter, kept waiting rows from being handed out and small
        // products from using all blocks: 17 000 rows, three quarters of them waiting, 256 columns 70 us against 47 (54
        // by the items kernel in breadth-first order), 30 000 with few waiting 54 against 41, the same from 60 000 on.
        c.claims_per_slab = d.n_chunks;
    } else if (tma) {
        const i32 slab = 256;  // 1 KB row pieces: the copy engine is bound by copies, not bytes
        c.sh.v4 = true;
        c.sh.nv = slab / 128;
        c.sh.slab_w = slab;
        c.sh.n_slabs = (f + slab - 1) / slab;
        c.group = 16;
    } else {
        c.sh = pick_shape(f, p->slab_width, can_v4);
        // never-waiting items are claimed 4 at a time: measured best on B200 (fewer trips to the
        // claim counter, which bounds short-row workloads; larger groups unbalance the long rows).
        // Rows in community order are of mixed, mostly short length: 8 at a time where they are narrow (400 000 rows of
        // 47 columns 275 -> 269 us; 50 000 rows in order of length 46 -> 65).
        // A small product keeps single claims: with fewer claims than resident warps, grouping
        // only idles warps.
        // (Long rows: four to a claim is too coarse for so few claims, and lifted rows do not bring it about sooner: 14 000 rows
        // of 177 entries, 500 columns 288 us, 246 with single claims.)
        const i32 n_apart = p->long_rows() ? std::min(d.n_prefix, p->tree.n_prefix) : d.n_prefix;
        c.group = ((i64)n_apart * c.sh.n_slabs >= (i64)p->sm_count * 256) ? (f <= 64 && d.n_chunks > 0 ? 8 : 4) : 1;
        if (c.group == 1 && p->n_blocks == 0) {
            const i64 warps = (i64)p->sm_count * resident_blocks(c.sh, f, c.ragged, mode) * 8;
            const i32 group = one_round_group(d.n_prefix, d.n_items - d.n_prefix, c.sh.n_slabs, warps);
            c.one_round = group > 0;
            if (c.one_round) c.group = group;
        }
    }
    if (!c.chunked) {
        c.n_pclaims = (d.n_prefix + c.group - 1) / c.group;
        c.claims_per_slab = c.n_pclaims + (d.n_items - d.n_prefix);
    }
    c.n_claims = (i64)c.claims_per_slab * c.sh.n_slabs;
    c.need_flags = (i64)c.sh.n_slabs * d.n_items;
    c.need_scratch = (i64)c.sh.n_slabs * d.n_partial * c.sh.slab_w;
    c.need_pack = c.pack ? (i64)p->n_labels * ((f + 3) / 4 * 4) : 0;
    if (c.need_flags >= (i64)1 << 31)
        return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": rows x column slabs exceeds 2^31 work items");
    return CBM_B200_OK;
}

template <int SLABW, int NB, int STAGES, int WARPS>
int launch_tma(KParams& kp, int sm_count, cudaStream_t s) {
    using L = TmaLayout<SLABW, NB, STAGES>;
    static bool configured[64] = {false};
    int dev = 0;
    CBM_CUDA(cudaGetDevice(&dev));
    auto kern = cbm_items_tma_kernel<SLABW, NB, STAGES, WARPS>;
    const int smem = L::smem_bytes(WARPS);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        CBM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured[dev] = true;
    }
    const int blocks = (int)std::max<i64>(1, std::min<i64>(sm_count, (kp.n_claims + WARPS - 1) / WARPS));
    kp.n_warps = (u64)blocks * WARPS;
    kern<<<blocks, WARPS * 32, smem, s>>>(kp);
    CBM_CUDA(cudaGetLastError());
    return CBM_B200_OK;
}

template <int NV, bool V4, bool RAGGED = false>
int launch_regs(KParams& kp, bool one_round, int want_blocks, int sm_count, const cbm::Stream& s) {
    // Unroll depth and resident blocks per SM were chosen by measurement on B200.  For the default
    // form (one float4 per lane, 128-column slabs) 4 gathers in flight per warp at 48 resident
    // warps per SM (40 registers) beat 8 in flight at 32 warps (64 registers) by 3 % on wide
    // operands and tie on narrow ones; forms that spill registers lose more than extra resident
    // warps gain.
    constexpr int kUnroll = NV == 1 ? (V4 ? 4 : 8) : 4;
    constexpr int kResident = resident_regs(NV, V4, RAGGED);
    int blocks = want_blocks > 0 ? want_blocks : sm_count * (NV == 1 && V4 ? kResident : 8);
    blocks = (int)std::max<i64>(1, std::min<i64>(blocks, (kp.n_claims + 7) / 8));
    kp.n_warps = (u64)blocks * 8;
    if (one_round) cbm::launch_next(cbm_items_kernel<NV, V4, kUnroll, kResident, RAGGED, false, true>, blocks, 256, 0, s, kp);
    else cbm::launch_next(cbm_items_kernel<NV, V4, kUnroll, kResident, RAGGED>, blocks, 256, 0, s, kp);
    CBM_CUDA(cudaGetLastError());
    return CBM_B200_OK;
}

// Operands of at most 64 columns: a kernel of their own, whose smaller register need keeps 48 warps resident also where
// rows of y are not aligned.  Fetches in flight x resident blocks, 235 868 rows of 11 entries, 64 columns / 400 000 of
// 22, 47 columns: 4 x 6 97 / 279 us, 6 x 5 100 / 288, 8 x 5 104 / 298, 8 x 4 110 / 310.
template <bool RAGGED>
int launch_narrow(KParams& kp, bool one_round, int want_blocks, int sm_count, const cbm::Stream& s) {
    constexpr int kResident = NARROW_RESIDENT;
    int blocks = want_blocks > 0 ? want_blocks : sm_count * kResident;
    blocks = (int)std::max<i64>(1, std::min<i64>(blocks, (kp.n_claims + 7) / 8));
    kp.n_warps = (u64)blocks * 8;
    if (one_round) cbm::launch_next(cbm_items_kernel<1, true, 4, kResident, RAGGED, true, true>, blocks, 256, 0, s, kp);
    else if (kp.group == NARROW_ROWS) cbm::launch_next(cbm_items_kernel<1, true, 4, kResident, RAGGED, true, false, true>, blocks, 256, 0, s, kp);
    else cbm::launch_next(cbm_items_kernel<1, true, 4, kResident, RAGGED, true>, blocks, 256, 0, s, kp);
    CBM_CUDA(cudaGetLastError());
    return CBM_B200_OK;
}

template <bool RAGGED>
int launch_chunks(KParams& kp, int want_blocks, int sm_count, const cbm::Stream& s) {
    constexpr int kResident = 3;  // 45 consumer warps per SM at 40 registers
    int blocks = want_blocks > 0 ? want_blocks : sm_count * kResident;
    blocks = (int)std::max<i64>(1, std::min<i64>(blocks, kp.n_claims));
    kp.n_warps = (u64)blocks;  // one claimer per block
    cbm::launch_next(cbm_chunks_kernel<RAGGED, 4, kResident>, blocks, (CONSUMERS + 1) * 32, 0, s, kp);
    CBM_CUDA(cudaGetLastError());
    return CBM_B200_OK;
}

// Rows of `f` floats copied to rows of 4 * vecs floats, zero-filled: one thread per vector of the result, the
// source read 4 bytes at a time (its rows are not aligned).  Bound by HBM.
__global__ void __launch_bounds__(256) pack_rows_kernel(const float* x, i64 ldx, float* out, i32 f, i32 vecs, i64 n_vec) {
    cbm::wait_before();
    const i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_vec) return;
    const i64 row = i / vecs;
    const i32 c = (i32)(i - row * vecs) * 4;
    const float* r = x + row * ldx + c;
    float4 v;
    v.x = r[0];
    v.y = c + 1 < f ? r[1] : 0.f;
    v.z = c + 2 < f ? r[2] : 0.f;
    v.w = c + 3 < f ? r[3] : 0.f;
    reinterpret_cast<float4*>(out)[i] = v;
}

// Fills the launch parameters that do not depend on where the scratch lives, and launches.
struct Bcast {
    int n = 0;
    int relu = 0;
    float* dst[CBM_B200_MAX_BCAST] = {nullptr};
};

template <int NV, bool V4>
int launch_frugal(KParams& kp, i32 out, i32 segment, int sm_count, cudaStream_t s) {
    const int blocks = (int)std::max<i64>(1, std::min<i64>(sm_count * (NV == 1 ? 4 : 2), (kp.n_claims + 7) / 8));
    kp.n_warps = (u64)blocks * 8;
    cbm_items_frugal_kernel<NV, V4><<<blocks, 256, 0, s>>>(kp, out, segment);
    CBM_CUDA(cudaGetLastError());
    return CBM_B200_OK;
}

int launch_plan(cbm_b200_plan* p, const DeviceSchedule& d, const LaunchCfg& c, const float* x, i64 ldx, float* y, i64 ldy, i32 f,
                int mode, bool use_scale, u64* counter, i32* flags, float* scratch, i32 epoch,
                const cbm::Stream& on, const Bcast* bc = nullptr) {
    KParams kp{};
    kp.y_vec = ldy % 4 == 0 && aligned16(y);
    kp.in_turn = c.in_turn;
    if (bc) {
        for (int k = 0; k < bc->n; ++k) kp.y_vec = kp.y_vec && aligned16(bc->dst[k]);
        kp.n_bcast = bc->n;
        kp.bcast_relu = bc->relu;
        for (int k = 0; k < bc->n; ++k) kp.bcast[k] = bc->dst[k];
    }
    kp.desc = d.d_desc;
    kp.ent = d.d_ent;
    kp.chunks = d.d_chunks;
    kp.ldx_bytes = (unsigned)(4 * ldx);
    kp.x = x;
    kp.y = y;
    kp.ldx = ldx;
    kp.ldy = ldy;
    kp.f = f;
    kp.slab_w = c.sh.slab_w;
    kp.n_items = d.n_items - c.left_out;
    kp.n_prefix = d.n_prefix - c.left_out;
    kp.group = c.group;
    kp.n_pclaims = c.n_pclaims;
    kp.claims_per_slab = c.claims_per_slab;
    kp.n_claims = c.n_claims;
    kp.scratch = scratch;
    kp.n_partial = d.n_partial - c.left_out;
    kp.counter = counter;
    kp.flags = flags;
    kp.epoch = epoch;
    kp.status = p->d_status;
    kp.mode = mode;
    kp.use_scale = use_scale ? 1 : 0;
    kp.wait_ns = 2000000000ULL;
    if (c.left_out > 0) {
        const i32 out = c.left_out, seg = d.segment;
        if (c.sh.v4) {
            if (c.sh.nv == 1) return launch_frugal<1, true>(kp, out, seg, p->sm_count, on.s);
            if (c.sh.nv == 2) return launch_frugal<2, true>(kp, out, seg, p->sm_count, on.s);
            return launch_frugal<4, true>(kp, out, seg, p->sm_count, on.s);
        }
        if (c.sh.nv == 1) return launch_frugal<1, false>(kp, out, seg, p->sm_count, on.s);
        if (c.sh.nv == 2) return launch_frugal<2, false>(kp, out, seg, p->sm_count, on.s);
        return launch_frugal<4, false>(kp, out, seg, p->sm_count, on.s);
    }
    if (c.tma) return launch_tma<256, 16, 2, 7>(kp, p->sm_count, on.s);
    if (c.chunked)
        return c.ragged ? launch_chunks<true>(kp, p->n_blocks, p->sm_count, on)
                        : launch_chunks<false>(kp, p->n_blocks, p->sm_count, on);
    if (c.sh.v4 && c.sh.nv == 1 && f <= 64 && mode != MODE_UPDATE_ONLY)
        return c.ragged ? launch_narrow<true>(kp, c.one_round, p->n_blocks, p->sm_count, on) : launch_narrow<false>(kp, c.one_round, p->n_blocks, p->sm_count, on);
    if (c.ragged) {
        if (c.sh.nv == 1) return launch_regs<1, true, true>(kp, c.one_round, p->n_blocks, p->sm_count, on);
        if (c.sh.nv == 2) return launch_regs<2, true, true>(kp, c.one_round, p->n_blocks, p->sm_count, on);
        return launch_regs<4, true, true>(kp, c.one_round, p->n_blocks, p->sm_count, on);
    }
    if (c.sh.v4) {
        if (c.sh.nv == 1) return launch_regs<1, true>(kp, c.one_round, p->n_blocks, p->sm_count, on);
        if (c.sh.nv == 2) return launch_regs<2, true>(kp, c.one_round, p->n_blocks, p->sm_count, on);
        return launch_regs<4, true>(kp, c.one_round, p->n_blocks, p->sm_count, on);
    }
    if (c.sh.nv == 1) return launch_regs<1, false>(kp, c.one_round, p->n_blocks, p->sm_count, on);
    if (c.sh.nv == 2) return launch_regs<2, false>(kp, c.one_round, p->n_blocks, p->sm_count, on);
    return launch_regs<4, false>(kp, c.one_round, p->n_blocks, p->sm_count, on);
}

bool has_room(const cbm_b200_plan* p, const LaunchCfg& c) {
    return c.need_flags <= p->flags_cap && c.need_scratch <= p->scratch_cap && c.need_pack <= p->pack_cap;
}

int make_room(cbm_b200_plan* p, const LaunchCfg& c, cudaStream_t s) {
    int rc = grow(p, p->d_flags, p->flags_cap, c.need_flags, true, s);
    if (rc == CBM_B200_OK) rc = grow(p, p->d_scratch, p->scratch_cap, c.need_scratch, false, s);
    return rc ? rc : grow(p, p->d_pack, p->pack_cap, c.need_pack, false, s);
}

int run_plan(cbm_b200_plan* p, const char* who, const float* x, i64 ldx, float* y, i64 ldy, i32 f,
             int mode, bool use_scale, cudaStream_t s, const Bcast* bc = nullptr, bool in_turn = false) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": NULL plan");
    int rc = check_dense(who, x, ldx, y, ldy, f);
    if (rc) return rc;
    if (mode != MODE_UPDATE_ONLY && !x)
        return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": x is NULL");
    if (use_scale && !p->normalized)
        return cbm::fail(CBM_B200_ERR_ARG,
                         std::string(who) + ": plan was created without a multiplier");
    if (p->n_rows == 0) return CBM_B200_OK;
    DeviceGuard g(p->device);
    const cbm::Stream on(s);
    LaunchCfg c;
    const DeviceSchedule* d = &p->schedule_for(mode, f);
    rc = plan_cfg(p, *d, who, x, ldx, y, ldy, f, mode, !in_turn, in_turn, c);
    // With rows lifted out of the tree a product may have more sums to park: where they find no room, it goes by the tree.
    if (d != &p->tree && (rc || (!has_room(p, c) && (on.captured || make_room(p, c, s))))) {
        (void)cudaGetLastError();
        d = &p->tree;
        rc = plan_cfg(p, *d, who, x, ldx, y, ldy, f, mode, !in_turn, in_turn, c);
    }
    if (rc || (rc = make_room(p, c, s))) return rc;
    if (p->epoch == INT32_MAX) {  // epochs exhausted: start over on clean flags
        CBM_CUDA(cudaMemsetAsync(p->d_flags, 0, (size_t)p->flags_cap * sizeof(i32), s));
        p->epoch = 0;
    }
    p->captured = p->captured || on.captured;
    // A graph launches this very epoch each time: its flags are cleared as part of it, lest a row takes its parent's row or
    // parked sums of the launch before for this one's.
    if (on.captured && d->n_items > d->n_prefix) CBM_CUDA(cudaMemsetAsync(p->d_flags, 0, (size_t)c.need_flags * sizeof(i32), s));
    if (c.pack) {
        const i32 vecs = (f + 3) / 4;
        const i64 n_vec = (i64)p->n_labels * vecs;
        cbm::launch_next(pack_rows_kernel, (unsigned)((n_vec + 255) / 256), 256, 0, on, x, ldx, p->d_pack, f, vecs, n_vec);
        CBM_CUDA(cudaGetLastError());
        x = p->d_pack;
        ldx = 4 * (i64)vecs;
    }
    return launch_plan(p, *d, c, x, ldx, y, ldy, f, mode, use_scale, p->d_counter, p->d_flags, p->d_scratch,
                       ++p->epoch, on, bc);
}

}  // namespace

extern "C" int32_t cbm_b200_one_round_group(int32_t n_prefix, int32_t n_waiting, int32_t n_slabs, int32_t warps) {
    return n_prefix < 0 || n_waiting < 0 || n_slabs < 1 || warps < 1 ? 0 : one_round_group(n_prefix, n_waiting, n_slabs, warps);
}

extern "C" int cbm_b200_spmm_update(cbm_b200_plan* p, const float* x, int64_t ldx, float* y,
                                    int64_t ldy, int32_t f, void* stream) {
    return run_plan(p, "spmm_update", x, ldx, y, ldy, f, MODE_FUSED, false, (cudaStream_t)stream);
}
extern "C" int cbm_b200_fused_spmm_update(cbm_b200_plan* p, const float* x, int64_t ldx, float* y,
                                          int64_t ldy, int32_t f, void* stream) {
    return run_plan(p, "fused_spmm_update", x, ldx, y, ldy, f, MODE_FUSED, true,
                    (cudaStream_t)stream);
}
extern "C" int cbm_b200_update(cbm_b200_plan* p, float* y, int64_t ldy, int32_t f, void* stream) {
    return run_plan(p, "update", nullptr, 0, y, ldy, f, MODE_UPDATE_ONLY, false,
                    (cudaStream_t)stream);
}
extern "C" int cbm_b200_fused_update(cbm_b200_plan* p, float* y, int64_t ldy, int32_t f,
                                     void* stream) {
    return run_plan(p, "fused_update", nullptr, 0, y, ldy, f, MODE_UPDATE_ONLY, true,
                    (cudaStream_t)stream);
}
extern "C" int cbm_b200_delta_spmm(cbm_b200_plan* p, const float* x, int64_t ldx, float* y,
                                   int64_t ldy, int32_t f, void* stream) {
    return run_plan(p, "delta_spmm", x, ldx, y, ldy, f, MODE_DELTA_ONLY, false,
                    (cudaStream_t)stream);
}

extern "C" int cbm_b200_spmm_update_bcast(cbm_b200_plan* p, const float* x, int64_t ldx, float* y,
                                          int64_t ldy, int32_t f, int32_t normalized, int32_t relu,
                                          int32_t n_dst, float* const* dst, void* stream) {
    if (n_dst < 0 || n_dst > CBM_B200_MAX_BCAST || (n_dst > 0 && !dst))
        return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_bcast: between 0 and " +
                                               std::to_string(CBM_B200_MAX_BCAST) + " destinations");
    Bcast bc;
    bc.n = n_dst;
    bc.relu = relu != 0;
    const bool v4 = (f % 4 == 0) && (ldy % 4 == 0);
    for (int k = 0; k < n_dst; ++k) {
        if (!dst[k]) return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_bcast: NULL destination");
        if (dst[k] == x) return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_bcast: a destination aliases x");
        if (v4 && aligned16(y) && !aligned16(dst[k]))
            return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_bcast: destinations must be 16-byte aligned like y");
        bc.dst[k] = dst[k];
    }
    return run_plan(p, "spmm_update_bcast", x, ldx, y, ldy, f, MODE_FUSED, normalized != 0,
                    (cudaStream_t)stream, &bc);
}

extern "C" int cbm_b200_csr_spmm(int32_t n_rows, const int32_t* row_b, const int32_t* row_e,
                                 const int32_t* col, const float* val, const float* x,
                                 int64_t ldx, float* y, int64_t ldy, int32_t f, void* stream) {
    if (n_rows < 0 || (n_rows > 0 && (!row_b || !row_e)))
        return cbm::fail(CBM_B200_ERR_ARG, "csr_spmm: bad row arrays");
    int rc = check_dense("csr_spmm", x, ldx, y, ldy, f);
    if (rc) return rc;
    if (!x) return cbm::fail(CBM_B200_ERR_ARG, "csr_spmm: x is NULL");
    if (n_rows == 0) return CBM_B200_OK;
    const bool can_v4 = (f % 4 == 0) && (ldy % 4 == 0) && (ldx % 4 == 0) && aligned16(y) && aligned16(x);
    const Shape sh = pick_shape(f, 256, can_v4);
    const i64 n_units = (i64)sh.n_slabs * n_rows;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int blocks = (int)std::max<i64>(1, std::min<i64>((i64)sms * 8, (n_units + 7) / 8));
    cudaStream_t s = (cudaStream_t)stream;
#define CBM_CSR_LAUNCH(NV, V4)                                                                    \
    csr_rows_kernel<NV, V4><<<blocks, 256, 0, s>>>(n_rows, row_b, row_e, col, val, x, ldx, y, ldy, \
                                                   f, sh.slab_w, n_units)
    if (sh.v4) {
        if (sh.nv == 1) CBM_CSR_LAUNCH(1, true);
        else if (sh.nv == 2) CBM_CSR_LAUNCH(2, true);
        else CBM_CSR_LAUNCH(4, true);
    } else {
        if (sh.nv == 1) CBM_CSR_LAUNCH(1, false);
        else if (sh.nv == 2) CBM_CSR_LAUNCH(2, false);
        else CBM_CSR_LAUNCH(4, false);
    }
#undef CBM_CSR_LAUNCH
    CBM_CUDA(cudaGetLastError());
    return CBM_B200_OK;
}

namespace {

// Pageable host operands.  The runtime copies them through its own staging buffer, one thread, row piece by row piece:
// 100 000 x 500 floats in and out took 58 ms.  Here several threads copy rows into page-locked slots, laid
// out as on the device, while the slots before them are on their way over PCIe as single copies.
constexpr i64 BOUNCE_SLOT = 4 << 20;
constexpr int BOUNCE_SLOTS = 6;

bool is_pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Copies `rows` rows of `f` floats between pitches (in floats), several threads.
void copy_rows(float* dst, i64 dst_ld, const float* src, i64 src_ld, i64 rows, i32 f) {
    const int threads = (int)std::max<i64>(1, std::min<i64>(omp_get_max_threads(), rows * f / 65536));
#pragma omp parallel for schedule(static) num_threads(threads)
    for (i64 r = 0; r < rows; ++r) std::memcpy(dst + r * dst_ld, src + r * src_ld, (size_t)f * sizeof(float));
}

// The whole operand between host rows of f floats and device rows of ld floats, through the plan's slots.
int copy_through_slots(cbm_b200_plan* p, float* device, i64 ld, float* host, i64 rows, i32 f, bool in, cudaStream_t s) {
    if (!p->bounce) CBM_CUDA(cudaHostAlloc((void**)&p->bounce, (size_t)(BOUNCE_SLOTS * BOUNCE_SLOT), cudaHostAllocDefault));
    const i64 per = std::max<i64>(1, BOUNCE_SLOT / (ld * (i64)sizeof(float)));
    const i64 blocks = (rows + per - 1) / per;
    auto count = [&](i64 b) { return std::min(per, rows - b * per); };
    auto slot = [&](i64 b) { return reinterpret_cast<float*>(p->bounce + b % BOUNCE_SLOTS * BOUNCE_SLOT); };
    if (in) {
        for (i64 b = 0; b < blocks; ++b) {
            if (b >= BOUNCE_SLOTS) CBM_CUDA(cudaEventSynchronize(p->events[b % BOUNCE_SLOTS]));
            copy_rows(slot(b), ld, host + b * per * f, f, count(b), f);
            CBM_CUDA(cudaMemcpyAsync(device + b * per * ld, slot(b), (size_t)(count(b) * ld) * sizeof(float),
                                     cudaMemcpyHostToDevice, s));
            CBM_CUDA(cudaEventRecord(p->events[b % BOUNCE_SLOTS], s));
        }
        return CBM_B200_OK;
    }
    auto fetch = [&](i64 b) -> int {
        CBM_CUDA(cudaMemcpyAsync(slot(b), device + b * per * ld, (size_t)(count(b) * ld) * sizeof(float), cudaMemcpyDeviceToHost, s));
        CBM_CUDA(cudaEventRecord(p->events[b % BOUNCE_SLOTS], s));
        return CBM_B200_OK;
    };
    for (i64 b = 0; b < std::min<i64>(blocks, BOUNCE_SLOTS - 1); ++b)
        if (const int rc = fetch(b)) return rc;
    for (i64 b = 0; b < blocks; ++b) {
        if (b + BOUNCE_SLOTS - 1 < blocks)
            if (const int rc = fetch(b + BOUNCE_SLOTS - 1)) return rc;
        CBM_CUDA(cudaEventSynchronize(p->events[b % BOUNCE_SLOTS]));
        copy_rows(host + b * per * f, f, slot(b), ld, count(b), f);
    }
    return CBM_B200_OK;
}

}  // namespace

extern "C" int cbm_b200_spmm_update_host(cbm_b200_plan* p, const float* x, float* y, int32_t f,
                                         int32_t normalized) {
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_host: NULL plan");
    if (!x || !y || f <= 0) return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_host: bad x / y / f");
    DeviceGuard g(p->device);
    // The staging buffers use a leading dimension rounded up to 32 floats, so that rows start on
    // 128-byte lines whatever f is; chunks whose width is a multiple of 4 then take the 128-bit
    // path; a ragged last chunk is cut into a 128-bit part and a scalar tail of 1-3 columns.
    const i64 ld = ((i64)f + 31) / 32 * 32;  // whole 128-byte lines per row: gathered pieces fill whole lines
    const i64 xb = (i64)p->n_labels * ld, yb = (i64)p->n_out * ld;
    if (xb > p->stage_x_cap) {
        cudaFree(p->stage_x);
        p->stage_x = nullptr;
        p->stage_x_cap = 0;
        CBM_CUDA(cudaMalloc((void**)&p->stage_x, (size_t)xb * sizeof(float)));
        p->stage_x_cap = xb;
    }
    if (yb > p->stage_y_cap) {
        cudaFree(p->stage_y);
        p->stage_y = nullptr;
        p->stage_y_cap = 0;
        CBM_CUDA(cudaMalloc((void**)&p->stage_y, (size_t)std::max<i64>(yb, 1) * sizeof(float)));
        // padding rows of a shard are never written by the kernel: give them a defined value
        CBM_CUDA(cudaMemset(p->stage_y, 0, (size_t)std::max<i64>(yb, 1) * sizeof(float)));
        p->stage_y_cap = yb;
    }
    // Pipeline over column chunks: while chunk k is multiplied, chunk k+1 of x is on its way in
    // and chunk k-1 of y on its way out (PCIe is full duplex), so the call costs about one
    // transfer of x plus the last chunk's product and transfer instead of x + product + y.
    const i32 chunk = p->host_chunk > 0 ? p->host_chunk : 128;
    std::vector<std::pair<i32, i32>> chunks;  // (first column, width)
    for (i32 c0 = 0; c0 < f; c0 += chunk) {
        const i32 w = std::min(chunk, f - c0);
        if (w % 4 != 0 && w > 4) {  // ragged end: a 128-bit part and a short scalar tail
            chunks.emplace_back(c0, w / 4 * 4);
            chunks.emplace_back(c0 + w / 4 * 4, w % 4);
        } else {
            chunks.emplace_back(c0, w);
        }
    }
    const i32 n_chunks = (i32)chunks.size();
    if (!p->copy_in) CBM_CUDA(cudaStreamCreateWithFlags(&p->copy_in, cudaStreamNonBlocking));
    if (!p->copy_out) CBM_CUDA(cudaStreamCreateWithFlags(&p->copy_out, cudaStreamNonBlocking));
    while ((i32)p->events.size() < std::max(2 * n_chunks, BOUNCE_SLOTS)) {
        cudaEvent_t e;
        CBM_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        p->events.push_back(e);
    }
    cudaStream_t s = p->own_stream;
    const size_t pitch = (size_t)f * sizeof(float), dpitch = (size_t)ld * sizeof(float);
    // Operands of less than a few hundred KB are not worth the slots; rows that no slot holds do not fit them.
    const bool large = (i64)std::max(p->n_labels, p->n_out) * f >= 65536 && ld * (i64)sizeof(float) <= BOUNCE_SLOT;
    const bool x_slots = large && is_pageable(x), y_slots = large && is_pageable(y);
    if (x_slots || y_slots) {
        // A pageable operand keeps the host's threads busy, so there is nothing to overlap with the other
        // direction: operand in, products, result out.
        int rc = CBM_B200_OK;
        if (x_slots) rc = copy_through_slots(p, p->stage_x, ld, const_cast<float*>(x), p->n_labels, f, true, s);
        else CBM_CUDA(cudaMemcpy2DAsync(p->stage_x, dpitch, x, pitch, pitch, (size_t)p->n_labels, cudaMemcpyHostToDevice, s));
        for (i32 k = 0; k < n_chunks && rc == CBM_B200_OK; ++k) {
            const i32 c0 = chunks[k].first, w = chunks[k].second;
            rc = run_plan(p, "spmm_update_host", p->stage_x + c0, ld, p->stage_y + c0, ld, w, MODE_FUSED, normalized != 0, s,
                          nullptr, w % 4 != 0 && c0 > 0);
        }
        if (rc == CBM_B200_OK) {
            if (y_slots) rc = copy_through_slots(p, p->stage_y, ld, y, p->n_out, f, false, s);
            else CBM_CUDA(cudaMemcpy2DAsync(y, pitch, p->stage_y, dpitch, pitch, (size_t)p->n_out, cudaMemcpyDeviceToHost, s));
        }
        const int status = cbm_b200_plan_status(p, s);  // waits for the stream, whatever came before
        return rc ? rc : status;
    }
    for (i32 k = 0; k < n_chunks; ++k) {
        const i32 c0 = chunks[k].first;
        const i32 w = chunks[k].second;
        CBM_CUDA(cudaMemcpy2DAsync(p->stage_x + c0, dpitch, x + c0, pitch, (size_t)w * sizeof(float),
                                       (size_t)p->n_labels, cudaMemcpyHostToDevice, p->copy_in));
        CBM_CUDA(cudaEventRecord(p->events[2 * k], p->copy_in));
        CBM_CUDA(cudaStreamWaitEvent(s, p->events[2 * k], 0));
        // The short tail is summed entry by entry, as a device operand of this width with unaligned rows is where it is not
        // copied to aligned ones.  Where it is, or where the last slab is at most 64 columns wide, some of its
        // columns are summed in another order there: host and device operands agree to fp32 rounding, not to the bit.
        int rc = run_plan(p, "spmm_update_host", p->stage_x + c0, ld, p->stage_y + c0, ld, w, MODE_FUSED,
                          normalized != 0, s, nullptr, w % 4 != 0 && c0 > 0);
        if (rc) return rc;
        CBM_CUDA(cudaEventRecord(p->events[2 * k + 1], s));
        CBM_CUDA(cudaStreamWaitEvent(p->copy_out, p->events[2 * k + 1], 0));
        CBM_CUDA(cudaMemcpy2DAsync(y + c0, pitch, p->stage_y + c0, dpitch, (size_t)w * sizeof(float),
                                   (size_t)p->n_out, cudaMemcpyDeviceToHost, p->copy_out));
    }
    CBM_CUDA(cudaStreamSynchronize(p->copy_out));
    return cbm_b200_plan_status(p, s);
}

// Strided copy between host and device memory on a stream: one column chunk of a row-major operand
// (what the host-operand pipelines move).  A thin wrapper so that a host language without access to
// the CUDA runtime's 2-D copy can drive its own pipeline (cbm4gnn_b200/sharding.py does).
extern "C" int cbm_b200_copy2d_async(void* dst, int64_t dst_pitch, const void* src, int64_t src_pitch,
                                     int64_t width_bytes, int64_t rows, int32_t to_device, void* stream) {
    if (!dst || !src || width_bytes < 0 || rows < 0 || dst_pitch < width_bytes || src_pitch < width_bytes)
        return cbm::fail(CBM_B200_ERR_ARG, "copy2d_async: bad arguments");
    if (width_bytes == 0 || rows == 0) return CBM_B200_OK;
    CBM_CUDA(cudaMemcpy2DAsync(dst, (size_t)dst_pitch, src, (size_t)src_pitch, (size_t)width_bytes, (size_t)rows,
                               to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    return CBM_B200_OK;
}

// ------------------------------------------------------------------------------------------
// Self-test of the bounded wait: one warp waits, with a limit of `wait_ms`, for a ready flag that
// nothing ever sets, and must come back with the timeout status instead of spinning forever.
// Exercises exactly the wait the product kernels use, without disturbing any plan.
// ------------------------------------------------------------------------------------------
namespace {
__global__ void wait_probe_kernel(i32* flag_and_status, u64 wait_ns) {
    const bool ok = wait_ready(flag_and_status, 1, flag_and_status + 1, wait_ns);
    if (threadIdx.x == 0) flag_and_status[2] = ok ? 1 : 0;
}
}  // namespace

extern "C" int cbm_b200_selftest_wait(int32_t device, int32_t wait_ms, void* stream) {
    if (wait_ms <= 0 || wait_ms > 1000)
        return cbm::fail(CBM_B200_ERR_ARG, "selftest_wait: wait_ms must be in 1..1000");
    DeviceGuard g(device);
    if (!g.ok) return cbm::fail(CBM_B200_ERR_CUDA, "selftest_wait: cudaSetDevice failed");
    i32* d = nullptr;
    CBM_CUDA(cudaMalloc((void**)&d, 3 * sizeof(i32)));
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(d, 0, 3 * sizeof(i32), s);
    i32 h[3] = {0, 0, -1};
    if (e == cudaSuccess) {
        wait_probe_kernel<<<1, 32, 0, s>>>(d, (u64)wait_ms * 1000000ULL);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d);
    if (e != cudaSuccess) return cbm::fail(CBM_B200_ERR_CUDA, std::string("selftest_wait: ") + cudaGetErrorString(e));
    if (h[1] == CBM_B200_ERR_TIMEOUT && h[2] == 0)
        return cbm::fail(CBM_B200_ERR_TIMEOUT, "selftest_wait: the wait ran out as it should");
    return cbm::fail(CBM_B200_ERR_FORMAT, "selftest_wait: the wait did not report a timeout");
}

// ------------------------------------------------------------------------------------------
// Measurement aid: the rate at which all SMs together stream a buffer that is resident in L2
// (32 MB, read 64 times with L2-only 128-bit loads, eight independent loads in flight per thread).
// The product kernels gather operand rows out of L2, so this rate — not the HBM rate — is the
// ceiling of their gather traffic; bench.py reports the gather rate against it.
// ------------------------------------------------------------------------------------------
namespace {
__global__ void __launch_bounds__(512) l2_read_probe_kernel(const float4* __restrict__ buf, u64 n_vec, int rounds,
                                                            float* sink) {
    const u64 stride = (u64)gridDim.x * blockDim.x;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < rounds; ++r) {
        for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i + 7 * stride < n_vec; i += 8 * stride) {
            float4 t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = __ldcg(buf + i + (u64)k * stride);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                a.x += t[k].x;
                a.y += t[k].y;
                a.z += t[k].z;
                a.w += t[k].w;
            }
        }
    }
    if (a.x + a.y + a.z + a.w == 12345.678f) *sink = a.x;  // keeps the loads alive
}
}  // namespace

extern "C" double cbm_b200_probe_l2_read_gbps(int32_t device) {
    DeviceGuard g(device);
    if (!g.ok) return -1.0;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int threads = 512, blocks = sms * 2;
    const u64 per_pass = (u64)blocks * threads * 8;            // vectors read per sweep of the grid
    const u64 n_vec = ((32ull << 20) / 16) / per_pass * per_pass;  // about 32 MB, a whole number of sweeps
    float4* buf = nullptr;
    float* sink = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    double out = -1.0;
    if (cudaMalloc((void**)&buf, n_vec * 16) == cudaSuccess && cudaMalloc((void**)&sink, 4) == cudaSuccess &&
        cudaMemset(buf, 0, n_vec * 16) == cudaSuccess && cudaEventCreate(&e0) == cudaSuccess &&
        cudaEventCreate(&e1) == cudaSuccess) {
        const int rounds = 64;
        l2_read_probe_kernel<<<blocks, threads>>>(buf, n_vec, 4, sink);  // warm-up: brings the buffer into L2
        cudaEventRecord(e0);
        l2_read_probe_kernel<<<blocks, threads>>>(buf, n_vec, rounds, sink);
        cudaEventRecord(e1);
        float ms = 0.f;
        if (cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess && ms > 0.f)
            out = (double)n_vec * 16.0 * rounds / (ms * 1e-3) / 1e9;
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(buf);
    cudaFree(sink);
    return out;
}

// ------------------------------------------------------------------------------------------
// Product without any allocation in the call path.
//
// The ordinary product entry points grow the plan's ready-flag and partial-sum buffers, and the room for a packed
// operand, from the device's workspace pool the first time a wider operand arrives.  Some callers must never reach an allocator
// once they are running: a serving loop that has handed all device memory to its own pool, code
// that runs while a stream is being captured, a real-time path that cannot absorb the implicit
// device synchronisation of an allocation.  For them the same kernel is offered with its
// per-call scratch (claim counters, ready flags, partial sums of long rows) carved out of one
// fixed array that lives in the library image: every GPU that loads the library holds
// CBM_B200_STATIC_SCRATCH_BYTES of it until the process exits.
//
// The array is shared by every plan and every call on a device and keeps whatever the previous
// call left in it, so each call first clears the counters and the flags it is about to use (on
// the caller's stream).  Two such calls that overlap on one GPU — different streams, or different
// host threads — race on the array; the caller has to order them.
// ------------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_scratch[CBM_B200_STATIC_SCRATCH_BYTES];

namespace {

constexpr int kMaxDevices = 64;
unsigned char* g_static_scratch_addr[kMaxDevices] = {nullptr};

// In host code the name g_static_scratch is only a handle for the runtime, not a device address.
// The address a kernel can use is asked for once per device, with that device current.
int static_scratch_address(int device, unsigned char** out) {
    if (device < 0 || device >= kMaxDevices)
        return cbm::fail(CBM_B200_ERR_ARG, "spmm_update_static: device ordinal out of range");
    if (!g_static_scratch_addr[device]) {
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || !ptr)
            return cbm::fail(CBM_B200_ERR_CUDA, std::string("cudaGetSymbolAddress(g_static_scratch): ") +
                                                    cudaGetErrorString(e));
        g_static_scratch_addr[device] = static_cast<unsigned char*>(ptr);
    }
    *out = g_static_scratch_addr[device];
    return CBM_B200_OK;
}

i64 round_up_256(i64 v) { return (v + 255) / 256 * 256; }

// layout inside the fixed array: counters | ready flags | partial sums
i64 static_need(i64 n_flags, i64 n_scratch) { return 256 + round_up_256(n_flags * (i64)sizeof(i32)) + n_scratch * (i64)sizeof(float); }

// A product that does not fit the fixed array with all partial sums parked: what it takes is decided by a schedule whose
// rows are cut only beyond 192 entries, at 128, and by operands that are fetched 16 bytes a lane only where all rows are
// aligned, so that finer cuts and wider fetches, which need more, refuse no product.  One that would fit so parks the
// sums of as many of its longest rows as there is room for.  50 000 rows of the second benchmark configuration's kind,
// 500 columns: 10.1 MiB with 5 076 sums, 4.2 MiB with the 1 719 of coarser cuts; 238 us here with the sums that there is
// room for, 215 with all of them on the ordinary path, 244 with the coarser cuts.
bool takes_static(const cbm_b200_plan* p, const float* x, i64 ldx, const float* y, i64 ldy, i32 f) {
    const bool all_vec = f % 4 == 0 && ldx % 4 == 0 && aligned16(x) && ldy % 4 == 0 && aligned16(y);
    const Shape coarse = pick_shape(f, p->form && all_vec ? 256 : p->slab_width, all_vec);
    const i64 sums = p->tree.n_partial_coarse;
    return static_need(coarse.n_slabs * (p->n_rows + sums), (i64)coarse.n_slabs * sums * coarse.slab_w) <=
           (i64)CBM_B200_STATIC_SCRATCH_BYTES;
}

bool fit_static(const cbm_b200_plan* p, const float* x, i64 ldx, const float* y, i64 ldy, i32 f, LaunchCfg& c) {
    const bool x_vec = ldx % 4 == 0 && aligned16(x), all_vec = f % 4 == 0 && x_vec && ldy % 4 == 0 && aligned16(y);
    const i64 rows = p->n_rows;
    c = LaunchCfg{};
    c.sh = pick_shape(f, p->form && all_vec ? 256 : p->slab_width, x_vec && ldx < (i64)1 << 30);
    c.ragged = c.sh.v4 && !all_vec;
    const i64 per_sum = (i64)c.sh.n_slabs * (c.sh.slab_w + 1) * (i64)sizeof(i32);
    const i64 room = (i64)CBM_B200_STATIC_SCRATCH_BYTES - static_need(c.sh.n_slabs * rows, 0) - 256;
    const DeviceSchedule& d = p->schedule_for(MODE_FUSED, f);
    const auto& ends = d.part_ends;
    const auto past = std::upper_bound(ends.begin(), ends.end(), std::max<i64>(0, room / per_sum));
    const i32 kept = past == ends.begin() ? 0 : past[-1];
    c.left_out = d.n_partial - kept;
    const i32 n_prefix = d.n_prefix - c.left_out;
    c.group = (i64)n_prefix * c.sh.n_slabs >= (i64)p->sm_count * 256 ? 4 : 1;
    c.n_pclaims = (n_prefix + c.group - 1) / c.group;
    c.claims_per_slab = c.n_pclaims + (d.n_items - d.n_prefix);
    c.n_claims = (i64)c.claims_per_slab * c.sh.n_slabs;
    c.need_flags = (i64)c.sh.n_slabs * (rows + kept);
    c.need_scratch = (i64)c.sh.n_slabs * kept * c.sh.slab_w;
    return static_need(c.need_flags, c.need_scratch) <= (i64)CBM_B200_STATIC_SCRATCH_BYTES;
}

}  // namespace

extern "C" int cbm_b200_spmm_update_static(cbm_b200_plan* p, const float* x, int64_t ldx, float* y,
                                           int64_t ldy, int32_t f, int32_t normalized,
                                           void* stream) {
    const char* who = "spmm_update_static";
    if (!p) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": NULL plan");
    int rc = check_dense(who, x, ldx, y, ldy, f);
    if (rc) return rc;
    if (!x) return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": x is NULL");
    if (normalized && !p->normalized)
        return cbm::fail(CBM_B200_ERR_ARG, std::string(who) + ": plan was created without a multiplier");
    if (p->n_rows == 0) return CBM_B200_OK;

    LaunchCfg c;
    rc = plan_cfg(p, p->tree, who, x, ldx, y, ldy, f, MODE_FUSED, false, false, c);
    if (rc) return rc;
    const i64 need = static_need(c.need_flags, c.need_scratch);
    const bool taken = need <= (i64)CBM_B200_STATIC_SCRATCH_BYTES || takes_static(p, x, ldx, y, ldy, f);
    if (taken) {  // (by its tree; with rows lifted out of it there may be more sums to park)
        rc = plan_cfg(p, p->schedule_for(MODE_FUSED, f), who, x, ldx, y, ldy, f, MODE_FUSED, false, false, c);
        if (rc) return rc;
    }
    if (!taken || (static_need(c.need_flags, c.need_scratch) > (i64)CBM_B200_STATIC_SCRATCH_BYTES && !fit_static(p, x, ldx, y, ldy, f, c)))
        return cbm::fail(CBM_B200_ERR_ARG,
                         std::string(who) + ": this product needs " + std::to_string(need) +
                             " bytes of scratch, the fixed array holds " +
                             std::to_string((i64)CBM_B200_STATIC_SCRATCH_BYTES) +
                             "; use cbm_b200_spmm_update / cbm_b200_fused_spmm_update");

    DeviceGuard g(p->device);
    if (!g.ok) return cbm::fail(CBM_B200_ERR_CUDA, std::string(who) + ": cudaSetDevice failed");
    unsigned char* base = nullptr;
    rc = static_scratch_address(p->device, &base);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const i64 off_flags = 256, off_slots = off_flags + round_up_256(c.need_flags * (i64)sizeof(i32));
    // counters and flags must start at zero; the partial sums are written before they are read
    CBM_CUDA(cudaMemsetAsync(base, 0, (size_t)(off_flags + c.need_flags * (i64)sizeof(i32)), s));
    // flags were just cleared, so any non-zero mark will do as this launch's epoch
    return launch_plan(p, p->schedule_for(MODE_FUSED, f), c, x, ldx, y, ldy, f, MODE_FUSED, normalized != 0,
                       reinterpret_cast<u64*>(base), reinterpret_cast<i32*>(base + off_flags),
                       reinterpret_cast<float*>(base + off_slots), 1, s);
}
