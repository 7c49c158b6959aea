// Shared by the dense-map kernels: tcgen05 helpers, the split of fp32 into three bf16 terms, the order of the
// products, bounded waits.
//
// An fp32 value is x = b0 + b1 + b2 to 24 bits, each b a bf16 (8 bits).  Of the nine products a_i b_j the six with
// i + j <= 2 are issued as bf16 tcgen05.mma with fp32 accumulation in tensor memory; the three others are
// below 2^-24 of |a||b|.
//
// The tensor cores cut the accumulator off at every step instead of rounding it, always towards zero, so a long
// contraction in one accumulator drifts: 1.7e-6 of the result for 256 columns, 1e-5 for the rows of a graph.  Hence
// an accumulator holds a short stretch of the contraction only: first the small products, while it is 2^-8 of what
// it will be, then the large ones; the epilogue warps add it to sums in registers, rounded.
//   * Forward and input gradient: 16 columns, one step.  With 64 columns the maps took three quarters of the time, but
//     the drift (6e-8 of the result instead of 4e-8) is the same for all rows and does not average out in the product that
//     follows: 128 -> 256 -> 64 with its products 1.36e-7 against 1.17e-7 of the result; 64 columns 7.9e-8 against 6.3e-8.
//   * Weight gradient: 64 rows, 1.7e-7 for 235 868 rows (256 to 64 columns).
// Measured against float64: 6e-8 - 1.2e-7 of the result for 64 - 512 columns (cuBLAS fp32: 1.4e-7 - 4e-7; 1.5e-6 over
// 235 868 rows).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <string>

#include "cbm_b200.h"
#include "cbm_common.h"

namespace cbm_map {

using u32 = uint32_t;
using u64 = unsigned long long;

constexpr int TMEM_COLS = 512;
constexpr int D_COLS = 128;  // two accumulators of up to 128 columns, at columns 0 and 128, ...
constexpr int A_COL = 256;   // ... then the ring of split A operands,
constexpr int A_SLOTS = 4;   // 4 slots, each 32 values deep: 3 terms x 16 columns (two bf16 per column)
constexpr int A_SLOT_COLS = 48;
constexpr int CHUNK_K = 32;
constexpr u64 WAIT_NS = 2000000000ULL;

// Word that a kernel sets when one of its waits runs out; lives in page-locked host memory, so that
// the next call can look at it without a synchronisation.  NULL on failure.
int* timeout_word();
// OK, or the error to return when an earlier map gave up waiting.
int check_timeout(const char* who);
// SMs of the current device.
int sm_count();
// Lets a kernel use that much shared memory; asked for once per device, not on every call.
template <auto Kernel>
bool allow_smem(int bytes) {
    static std::atomic<u64> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const u64 bit = dev < 64 ? 1ull << dev : 0;
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

#ifdef __CUDACC__
__device__ __forceinline__ u32 smem_u32(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ u64 now_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void bar_init(u32 bar, u32 count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(u32 bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_poll(u32 bar, u32 parity) {
    u32 done;
    asm volatile(
        "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Bounded wait of a whole warp, and the fence without which what it then does in tensor memory (loads, stores, MMAs)
// would not be ordered behind what the barrier reports.  `gave_up` (shared memory) lets every role of the block stop
// once one wait has run out.
__device__ __forceinline__ bool warp_wait(u32 bar, u32 parity, volatile int* gave_up, int* timeout) {
    u64 t0 = 0;
    bool ok = true;
    for (u32 spins = 0;; ++spins) {
        if (bar_poll(bar, parity)) break;
        if ((spins & 31u) == 31u) {
            const u64 t = now_ns();
            if (t0 == 0) t0 = t;
            if (*gave_up || t - t0 > WAIT_NS || spins > (1u << 26)) {
                *gave_up = 1;
                *(volatile int*)timeout = 1;
                ok = false;
                break;
            }
        }
    }
    ok = __all_sync(0xffffffffu, ok);
    fence_after();
    return ok;
}

// ---- tensor memory and tcgen05 ------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(u32 where) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(where), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(u32 base) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(TMEM_COLS));
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// MMAs and commits are issued by one elected thread, but the whole warp runs the loop around them: with warp-uniform
// control flow the descriptors live in uniform registers; issued from a divergent branch every one had to be
// moved there first, and the issue, not the tensor cores, took the time (forward 128 -> 256: 147 us against 122).
__device__ __forceinline__ void commit(u32 bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
        : "memory");
}
// D[128, N] (+)= A[128, 16] B[N, 16]^T: A in tensor memory, B in shared memory.
__device__ __forceinline__ void mma(u32 d, u32 a, u64 b, u32 idesc, bool add) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.u32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"((u32)add)
        : "memory");
}
// Instruction descriptor: fp32 accumulator, bf16 operands, both K-major, M = 128.
__host__ __device__ constexpr u32 idesc_of(u32 n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// Shared-memory descriptor of a K-major operand in 128-byte swizzled rows (64 bf16), groups of 8 rows 1024
// bytes apart.
__device__ __forceinline__ u64 desc_of(u32 addr) {
    return (u64)((addr & 0x3ffff) >> 4) | ((u64)1 << 16) | ((u64)(1024 >> 4) << 32) | ((u64)1 << 46) | ((u64)2 << 61);
}
// 16-byte piece `k8` (8 bf16) of row `row` in that layout, from the start of the 64-wide block of rows.
__device__ __forceinline__ u32 swizzled(u32 row, u32 k8) { return row * 128 + ((k8 ^ (row & 7)) << 4); }

// (s, t) += (x, y), both with one instruction.
__device__ __forceinline__ void add2(float& s, float& t, float x, float y) {
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tadd.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(s), "+f"(t)
        : "f"(x), "f"(y));
}

// The five small products of one 16-deep step, smallest first; `b_term` bytes lie between B's terms.
__device__ __forceinline__ void mma_small(u32 d, u32 a, u32 b, u32 b_term, u32 idesc, bool add) {
    const u64 b0 = desc_of(b), b1 = desc_of(b + b_term), b2 = desc_of(b + 2 * b_term);
    mma(d, a + 32, b0, idesc, add);
    mma(d, a + 16, b1, idesc, true);
    mma(d, a, b2, idesc, true);
    mma(d, a + 16, b0, idesc, true);
    mma(d, a, b1, idesc, true);
}

// ---- operands -----------------------------------------------------------------------------------
// Fetches, zero where `on` is false.  Written as volatile asm so that a batch of fetches stays a batch,
// ahead of the work it is meant to hide behind: the compiler may not sink one to its use.  (Not
// ld.global.nc: see cbm_launch.cuh.)
__device__ __forceinline__ float fetch1(const float* p, bool on) {
    float v;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.f32 %0, [%1];\n\t}"
        : "=f"(v)
        : "l"(p), "r"((int)on));
    return v;
}
__device__ __forceinline__ float4 fetch4(const float* p, bool on) {
    float4 v;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
        "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p), "r"((int)on));
    return v;
}

// max(x, 0) that passes NaN on, as torch.relu does (fmaxf would make it 0).
__device__ __forceinline__ float relu(float x) {
    float y;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float4 relu(float4 x) { return make_float4(relu(x.x), relu(x.y), relu(x.z), relu(x.w)); }

// Two neighbours of the contraction (x at the lower address) -> their three bf16 pairs.
__device__ __forceinline__ void split2(float x, float y, u32& b0, u32& b1, u32& b2) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b0) : "f"(y), "f"(x));
    x -= __uint_as_float(b0 << 16);
    y -= __uint_as_float(b0 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b1) : "f"(y), "f"(x));
    x -= __uint_as_float(b1 << 16);
    y -= __uint_as_float(b1 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(b2) : "f"(y), "f"(x));
}
// Eight of them -> one 16-byte piece per term, stored `term` bytes apart.
__device__ __forceinline__ void store_split8(unsigned char* at, u32 term, const float (&x)[8]) {
    uint4 t0, t1, t2;
    split2(x[0], x[1], t0.x, t1.x, t2.x);
    split2(x[2], x[3], t0.y, t1.y, t2.y);
    split2(x[4], x[5], t0.z, t1.z, t2.z);
    split2(x[6], x[7], t0.w, t1.w, t2.w);
    *reinterpret_cast<uint4*>(at) = t0;
    *reinterpret_cast<uint4*>(at + term) = t1;
    *reinterpret_cast<uint4*>(at + 2 * term) = t2;
}
#endif

}  // namespace cbm_map
