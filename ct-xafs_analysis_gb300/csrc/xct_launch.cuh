// xct_launch.cuh -- dependent launches of the OS-EM kernels.
//
// The steps of an OS-EM loop are short kernels that follow one another on one stream.  They are
// launched with programmatic stream serialization: a kernel's blocks are scheduled while its
// predecessor's last blocks still run, and xct_grid_wait() holds every block until the
// predecessor has finished and its writes are visible.  Every kernel launched through
// xct_launch calls xct_grid_wait() before its first access to data that another launch writes
// (all of them but the angle table, which a plan writes once), so the order of the launches'
// memory accesses is the plain stream order.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "xct_internal.h"

__device__ __forceinline__ void xct_grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// lets the next launch's blocks be scheduled as this grid's leave room for them
__device__ __forceinline__ void xct_grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
static inline int xct_launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    g_xct_launches.fetch_add(1, std::memory_order_relaxed);
    XCT_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
    return XCT_OK;
}
