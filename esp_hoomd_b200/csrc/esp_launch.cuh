// Launches that overlap their start with the end of the stream's previous
// kernel (programmatic dependent launch): what a chain of short kernels spends
// between them. One evaluation of 512 ions, a chain of ten kernels of 2 to 6
// us: 61.6 us launched plainly, 47.1 overlapped; 15,912 ions 86.1 and 77.9.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace espb {

// First statement of a kernel launched with launch_after: waits until the
// previous kernel of the stream has completed and its writes are visible, then
// lets the next one start its own blocks.
__device__ __forceinline__ void after_previous() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

template <typename... K, typename... A>
inline cudaError_t launch_after(bool overlap, void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

// Where the overlap pays: blocks that start early hold their place while they
// wait, and with several waves of blocks in flight the concurrent pair term
// lacks it. Launched from the host, evaluations gain up to about 200 blocks of
// 256 particles (42,000 water charges 141.6 against 136.0 us, 60,000 187.7
// against 189.1, 98,304 250.6 against 255.3); in a captured graph, whose kernels
// follow one another faster, up to about 32 (an MD step of 1,000 ions 64.0
// against 58.9 us, 8,000 73.3 against 72.1, eight systems of 1,300 77.3 against
// 78.6).
inline bool overlap_starts(int n_chunks, cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n_chunks <= (cs == cudaStreamCaptureStatusNone ? 192 : 32);
}

}  // namespace espb
