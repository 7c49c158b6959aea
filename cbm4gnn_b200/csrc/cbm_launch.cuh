// Launches whose blocks are put in place while the stream's kernel before them is ending (programmatic stream serialization).
//
// A kernel that follows another on its stream otherwise starts after the last block has left, its writes have been flushed and
// the launch itself has been fetched and set up: about 1 us, which is a sixth of the smallest products.  With the
// attribute, blocks are set up as soon as the last of the kernel before has left, and wait in wait_before() for its writes.
// Back to back: 1 000 rows, 16 columns 6.15 -> 5.55 us a product (the host issues no more), 4 096 rows, 500 columns
// 21.6 -> 20.5, 50 000 rows, 64 columns 42.7 -> 40.7; a two-layer training step over 235 868 rows 1 093 -> 1 078.
//
// What a kernel launched like this has to keep to:
//   - every thread calls wait_before() ahead of any access to memory that the caller or another kernel may write, and no
//     thread leaves before it: the kernel cannot be done before the one ahead of it is, and so on along the stream;
//   - such memory is not read through ld.global.nc / __ldg, whose data must not change while the kernel is resident (a plan's
//     own tables, written before the plan is handed out, may be);
//   - it never signals its dependents early (griddepcontrol.launch_dependents): their blocks take places only when all of
//     its own have left, so tensor memory and shared memory are free again and nobody that is waited for is kept out.
#pragma once
#include <cuda_runtime.h>

namespace cbm {

__device__ __forceinline__ void wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A stream, and whether what is issued to it is captured into a graph.
struct Stream {
    cudaStream_t s;
    bool captured;
    Stream(cudaStream_t stream) : s(stream) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        const bool asked = cudaStreamIsCapturing(s, &capture) == cudaSuccess;
        if (!asked) (void)cudaGetLastError();  // (a stream that another one's capture forbids to use: the launch says so)
        captured = !asked || capture != cudaStreamCaptureStatusNone;
    }
};

// Under stream capture the launch is a plain one: what a graph's branches and joins wait for stays whole kernels.
// Errors are left for cudaGetLastError.
template <class... P, class... A>
void launch_next(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, const Stream& on, const A&... args) {
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = on.s;
    config.attrs = &early;
    config.numAttrs = on.captured ? 0 : 1;
    (void)cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}

}  // namespace cbm
