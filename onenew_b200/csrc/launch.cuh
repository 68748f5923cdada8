// launch.cuh -- how every kernel of this library is launched: with programmatic stream serialisation (unless
// switched off), so that a launch's blocks are placed while the previous kernel on the stream drains and only
// the kernel's own wait orders them.  A kernel launched this way calls pdl_entry() before it touches memory.
//
// Why for the short glue kernels too: without the attribute a launch starts only after the previous grid has
// retired (~1 us of an idle GPU each time, and the contraction after it cannot run its set-up early either);
// a one-image network is 60 - 100 launches of a few microseconds each.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <utility>

#include "ctx.h"

namespace one {

int get_pdl();

// A call on the caller's own tensors (the drop-in operators): its first launch has no such attribute.  That launch therefore
// starts when everything before it on the stream has completed, and so does all that follows within the call: its kernels may
// read the caller's tensors (the activation table, the bias) ahead of their own wait, which only has to order them behind each
// other.  Without it a contraction could stage a table that a kernel before the call was still writing, since each of the launches
// between the two releases its successor at once.  The stream is usually idle at that point, and the launch costs nothing more;
// ordering the reads inside the contraction kernels did (int8 backbone of 64 images 1614 -> 1649 us), and so did launching the
// contraction plainly (3 - 4 us of every drop-in Conv).
struct FirstLaunchPlain {
    static inline thread_local bool pending = false;
    FirstLaunchPlain() { pending = true; }
    ~FirstLaunchPlain() { pending = false; }
    static bool take() { const bool p = pending; pending = false; return p; }
};

// Launch with the programmatic-stream-serialisation attribute when `pdl`, and as clusters of `cluster` CTAs when
// that is above 1.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_ex(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, int cluster, Args &&...args)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (!FirstLaunchPlain::take() && pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// A plain kernel that begins with pdl_entry().
template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args)
{
    return launch_ex(kernel, grid, block, smem, stream, get_pdl() != 0, 1, std::forward<Args>(args)...);
}

#ifdef __CUDACC__
template <typename P> __device__ __forceinline__ void launder(P &p) { asm volatile("" : "+l"(p)); }
// Start of a kernel launched by launch_k: the next launch may be placed, this one waits until the previous kernel
// has completed and its writes are visible.  The pointers the kernel reads through are passed here so that the
// compiler cannot turn loads through a `const __restrict__` pointer into read-only ones (ld.global.nc), or move them above the
// wait: the wait does not order read-only loads.  So no __ldg of what an earlier kernel may have written either (an activation
// table never is: a prepared operator's copy, or complete before the call, see FirstLaunchPlain).
template <typename... P> __device__ __forceinline__ void pdl_entry(P &...ptrs)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (launder(ptrs), ...);
}
#endif

}  // namespace one
