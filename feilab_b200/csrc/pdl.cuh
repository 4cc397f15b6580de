// pdl.cuh -- programmatic dependent launch: the launcher and the wait that belongs
// to it; the number of SMs.
#pragma once
#include <cuda_runtime.h>

namespace icon {

constexpr int kSMs = 148;   // of a B200: the launch rules count in them

// First statement of every kernel that is launched with programmatic dependent
// launch: wait until the stream's previous kernel has completed and its writes
// are visible, then let the next launch's blocks become resident.  All data is
// touched after it, so each kernel still sees everything before it in the stream.
// Without the attribute both are no-ops.
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches with programmatic dependent launch: the kernel's blocks may become
// resident while the stream's previous kernel drains, and wait (pdl_wait, first
// thing in every kernel launched here) until that kernel has completed before
// they touch data.  Taken where launches follow one another within microseconds to
// tens of microseconds of work (figures of its introduction): one 64 x 40 slice forward 25.6 -> 19.9 us, 10
// iterations with the NUFFT operator on 32 slices of 256 x 128 2.63 -> 2.47 ms,
// warm-start predict of 8 slices of 1024 x 300 1.005 -> 0.978 ms, gradients of 16
// slices of 512 x 256 3.47 -> 3.44 ms, mask of 16 slices of 1024 x 1024 202 -> 186 us.
// early false: an ordinary launch, where measurement has the early one behind.
template <class... P, class... A>
inline void pdl_if(bool early, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
inline void pdl(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args)
{
    pdl_if(true, kernel, grid, threads, smem, st, args...);
}

}  // namespace icon
