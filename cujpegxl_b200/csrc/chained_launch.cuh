// Launches of kernels that follow each other on a stream with programmatic
// stream serialisation: the next grid is launched once the last block of the
// previous one has left, while its memory is still being flushed, which saves
// about a microsecond per launch of a frame's chain of short kernels. Every
// kernel launched so waits for the previous grid (all of
// it, its writes visible) before it reads or writes anything; and nothing
// here triggers the next grid early, so no block sits on an SM, waiting, that
// another stream's blocks could use. Because such a kernel can be resident
// while the grid before it still writes, it reads what that grid writes by
// ordinary loads: read-only-cache loads (__ldg) are for data that no one
// writes while the kernel lives, and a compiler may move them ahead of the
// wait.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace jxb {

// (No effect in a kernel launched the ordinary way.)
__device__ __forceinline__ void wait_for_previous_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// False when a test asked for this launch to fail
// (cujpegxl_b200_debug_fail_launch).
bool launch_allowed();

// One launch, chained to the previous grid or an ordinary one. A failed launch
// leaves no error behind for a later check on this thread to find.
template <class... P, class... A>
bool launch_one(bool chained, void (*kernel)(P...), unsigned blocks, unsigned threads, std::size_t smem,
                cudaStream_t stream, const A&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    if (!launch_allowed()) return false;
    if (cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

template <class... P, class... A>
bool launch_chained(void (*kernel)(P...), unsigned blocks, unsigned threads, std::size_t smem, cudaStream_t stream,
                    const A&... args) {
    return launch_one(true, kernel, blocks, threads, smem, stream, args...);
}

template <class... P, class... A>
bool launch_plain(void (*kernel)(P...), unsigned blocks, unsigned threads, std::size_t smem, cudaStream_t stream,
                  const A&... args) {
    return launch_one(false, kernel, blocks, threads, smem, stream, args...);
}

}  // namespace jxb
