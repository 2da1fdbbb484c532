// sl_pdl.cuh -- programmatic dependent launch: the kernels of a step follow
// each other on one stream, and a kernel of a few microseconds loses a
// microsecond or two to the previous one's last block, its own launch and its
// set-up.  launch_pdl lets a kernel's blocks start once every block of the
// kernel before it has called pdl_next (or ended); a kernel so launched calls
// pdl_wait before its first access to memory that an earlier kernel writes or
// reads, which returns when the kernel before has ended and its writes are
// visible.  As every kernel of a chain waits, the order of the whole chain
// holds.  Launched plainly, both calls do nothing.
//
// A kernel that waits is resident while earlier kernels still write what it
// reads.  Its loads of global memory are therefore ordinary ones: no __ldg
// and no __restrict__ parameter, which lets the compiler use the non-coherent
// path -- that path requires data that nothing writes while the kernel is
// resident, and the wait does not order it.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace sl {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// <<<grid, block, smem, st>>>, as a dependent of the stream's last kernel
// when `pdl` (only where that kernel was launched on the same stream with no
// event or copy between that the new one must wait for early).
template <typename... P, typename... A>
inline cudaError_t launch_pdl(bool pdl, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                              cudaStream_t st, A&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace sl
