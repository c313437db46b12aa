#pragma once
// Host-side helpers shared by the launchers: a thread-local error string and CUDA call checking
// that reports instead of aborting, because these launchers are called from inside a framework.
#include "fu_kernels.h"

#include <cuda_runtime.h>
#include <cstdarg>
#include <cstdio>
#include <utility>

namespace fu {

char* error_buffer();  // thread-local, 512 bytes

inline int fail(int code, const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(error_buffer(), 512, fmt, ap);
    va_end(ap);
    return code;
}

// Raises a kernel's dynamic shared-memory limit on the current device, once per device and kernel. Launches come
// from several threads (autograd's beside the caller's): the record of what has been raised is locked.
int raise_smem_limit(const void* kernel, int bytes);

template <class Kernel>
int raise_smem_limit(Kernel kernel, int bytes)
{
    return raise_smem_limit(reinterpret_cast<const void*>(kernel), bytes);
}

// Launches a kernel whose threads all call ptx::grid_wait() before they touch global memory, so that it may be set up while
// the kernel before it in the stream is still running: its CTAs come onto SMs as they become free and initialise their
// barriers, tensor memory and descriptors there. Otherwise each launch waits for the last CTA before it to have left and
// then starts from nothing, 1 - 3 us a kernel. Only kernels that trigger (ptx::grid_trigger) are overlapped: behind any other,
// PyTorch's for instance, or behind a copy, this is an ordinary launch.
//
// Not for kernels that other ranks wait for, and not for clusters of more than two that fill the device: taken up as SMs
// become free they leave SMs over that no whole cluster fits into, or crowd on the first ones. Nor does a kernel whose grid
// the caller has limited (`ctas`) start so or let the next one: the SMs that it leaves free are meant for another stream, and
// the next kernel's CTAs would hold them until it ends. Kernels without a limit are launched so on groups of any size: an
// exchange that is queued on another stream meanwhile may find the next kernel's CTAs in the SMs that became free, and
// waits for one kernel as it does when it comes just after its launch; none of these waits for a peer.
template <class... P, class... A>
cudaError_t launch_behind(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args)
{
    cudaLaunchConfig_t  cfg  = {};
    cudaLaunchAttribute attr = {};
    attr.id                  = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim              = grid;
    cfg.blockDim             = block;
    cfg.dynamicSmemBytes     = smem;
    cfg.stream               = stream;
    cfg.attrs                = &attr;
    cfg.numAttrs             = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace fu

#define FU_CUDA_OK(expr)                                                                                      \
    do {                                                                                                      \
        cudaError_t fu_err__ = (expr);                                                                        \
        if (fu_err__ != cudaSuccess) {                                                                        \
            (void)cudaGetLastError(); /* reported here: the next launch's own check must not find it again */ \
            return ::fu::fail(FU_E_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(fu_err__),        \
                              __FILE__, __LINE__);                                                            \
        }                                                                                                     \
    } while (0)
