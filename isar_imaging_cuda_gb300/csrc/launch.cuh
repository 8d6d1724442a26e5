// Launches that overlap the end of the kernel before them.
//
// A frame is a chain of ~20 kernels of a few microseconds each; between two of
// them the GPU drains, launches and fills its tables.  launch_after() marks a
// launch as programmatically dependent: its CTAs may be scheduled once every
// CTA of the kernel before has started and passed pdl_begin(), and wait there
// until that kernel has completed and its writes are visible.  Whatever a
// kernel does before pdl_begin() may touch shared memory and the context's
// constant tables only; the one exception is k_ra_spec0, which starts copying
// the frame's echoes.  They are the caller's or an earlier kernel's, and the
// kernel in front of it, k_zero_shift, is launched in the ordinary way: it
// began only once all of that had completed, and does not touch them.
//
// Single frames use it; the lanes of a batch do not (a waiting CTA holds
// shared memory and registers that another lane's kernel could use).  The
// first kernel of a frame is launched in the ordinary way, so everything
// before the frame has completed.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "isar_kernels.h"

namespace isar {

__device__ __forceinline__ void pdl_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
cudaError_t launch_after(bool overlap, void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
    if (!overlap) {
        k<<<grid, block, smem, st>>>(std::forward<A>(args)...);
        const cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) ISAR_COUNT(1);
        return e;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
    if (e == cudaSuccess) ISAR_COUNT(1);
    return e;
}

}  // namespace isar
