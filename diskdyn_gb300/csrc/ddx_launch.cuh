// Kernel launches that overlap the start of a kernel with the end of the one before it in the
// stream (programmatic stream serialization).  A step with few tracers is 5 to 35 short kernels
// in a row, and starting one only when the last has drained costs a microsecond or two each.
//
// Every kernel launched by launch_after calls after_previous() first, in every thread: it waits
// until the kernel before has finished and its writes are visible, then lets the next kernel's
// blocks take free slots.  So a kernel still sees everything that came before it in the stream;
// launches without the attribute, copies and event waits keep their full order.  (Steps, us:
// star and eight planets, 16,384 tracers 53 -> 46; 3,001 planetesimals with a halo, 10,003 tracers
// 550 -> 492; collision pass of a million 248 -> 224.)
//
// A long kernel whose blocks do not fill the GPU is launched in full order when the one before is
// long too: its blocks would crowd the SMs that come free first (compensated step with 4,096
// planetesimals and 45,003 tracers: 4060 us so, 5810 us with its dust kernel overlapped).
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace ddx {

// Massive bodies up to which the massive passes and the dust kernel overlap their start (us a step;
// passes, 256 planetesimals and 2,003 tracers: 92 with, 96 without, 1,500: 285 / 270; dust, no
// planetesimals: 64 / 68, 300 compensated, 45,003 tracers: 735 / 504).
constexpr int kOverlapPasses = 512, kOverlapDust = 64;

__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_with(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t st, A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}
template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    return launch_with(true, kernel, grid, block, smem, st, std::forward<A>(args)...);
}
// The first kernel of a call: what came before it may be anything.
template <class... P, class... A>
inline cudaError_t launch_first(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    return launch_with(false, kernel, grid, block, smem, st, std::forward<A>(args)...);
}

}  // namespace ddx
