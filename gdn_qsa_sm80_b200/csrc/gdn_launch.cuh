// Host side of a kernel launch: the dynamic shared-memory limit (set once per kernel and context, not on every call) and
// the launch as a programmatic dependent of the kernel before it in the stream.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "gdn_common.cuh"

namespace gdn {

// Held by an entry point while it enqueues: calls that use the same scratch buffer hand data from kernel to kernel through it (a
// packed batch: tables the kernels index with), so two threads' calls must not interleave.  Calls on different buffers
// do not wait for each other; nothing is allocated and nothing kept behind the call.
class EnqueueLock {
public:
    explicit EnqueueLock(const void* scratch);
    ~EnqueueLock();
    EnqueueLock(const EnqueueLock&) = delete;
    EnqueueLock& operator=(const EnqueueLock&) = delete;

private:
    const void* scratch_;
    EnqueueLock* next_;
};

// Lets `kernel` use `bytes` of dynamic shared memory in the current context; 0 on success.
int allow_smem(const void* kernel, size_t bytes);

// Launches with the programmatic-stream-serialization attribute: the CTAs may set up while the kernel before this one in the
// stream drains.  What that kernel makes is touched behind grid_dependency_wait only.  What is older may be read in front of it (the chain:
// K, V and the initial state, Problem::behind_prepare; the normalisation: z, its z_ready), but only behind a kernel all of whose CTAs have
// themselves waited before they trigger or end: a launch by this function says nothing about the kernels before the last one.
// `pairs`: clusters of two CTAs along x.  Where the context has neither, an ordinary launch, in which that wait is a no-op.
template <typename Kernel, typename... Args>
inline cudaError_t launch_dependent(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pairs, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pairs ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        cfg.numAttrs = 0;
        e = cudaLaunchKernelEx(&cfg, kernel, args...);
    }
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace gdn
