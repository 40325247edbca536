// Kernel launches with programmatic stream serialisation: a kernel is scheduled as the CTAs of the one before it in the
// stream leave, so that its launch latency and set-up (barriers, TMEM, descriptor fetch, clearing shared memory) run
// beside the predecessor's last CTAs and its memory flush instead of after them.  Every kernel of the library executes
// pdl_wait() in every thread before the first access to global memory; after it all earlier work of the stream is
// complete and visible, as in a plain launch.  A kernel that skipped it could finish before its predecessor did and
// break that for its successors, so all of them call it.
//
// The trains of kernels of a few microseconds that the small networks and layers are gain 5-15 % (28x28 CNN step 494 ->
// 353 us on top of the native host path, 8x8 256->256 convolution 112 -> 95 us).  No kernel triggers its successor
// earlier (griddepcontrol.launch_dependents), neither at its start nor after its last load: the waiting CTAs take L1
// capacity and thread slots from the running ones (measured 353 -> 437 / 876 us on that step, 490 -> 532 / 546 us on the
// 56x56 64->128 convolution).  An early trigger before a TMEM allocation could also deadlock: a successor that allocates
// first on the SM and then waits for a kernel whose allocation waits for it.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include <utility>

namespace aether {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// `cluster` > 1: clusters of that many CTAs along x.  Errors are left for cudaGetLastError (check_launch).
template <typename... P, typename... A>
static inline void launch_cluster(void (*kernel)(P...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
static inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    launch_cluster(kernel, 1, grid, block, smem, st, std::forward<A>(args)...);
}

}  // namespace aether
