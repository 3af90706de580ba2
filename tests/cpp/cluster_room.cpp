// cluster_room.cpp -- the CUDA runtime of a device with room for clusters of
// at most MAX_CTAS blocks, for a library linked with
//   --wrap=cudaOccupancyMaxActiveClusters --wrap=cudaLaunchKernelExC
// Larger ones are refused on the host, as the runtime refuses them.
#include <cuda_runtime.h>

#ifndef MAX_CTAS
#define MAX_CTAS 8
#endif

namespace {

bool too_large(const cudaLaunchConfig_t *c)
{
    for (unsigned k = 0; k < c->numAttrs; ++k)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension &&
            c->attrs[k].val.clusterDim.x > MAX_CTAS)
            return true;
    return false;
}

} // namespace

extern "C" {

cudaError_t __real_cudaOccupancyMaxActiveClusters(
    int *n, const void *f, const cudaLaunchConfig_t *c);
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t *c,
                                       const void *f, void **args);

cudaError_t __wrap_cudaOccupancyMaxActiveClusters(int *n, const void *f,
                                                  const cudaLaunchConfig_t *c)
{
    if (too_large(c)) {
        *n = 0;
        return cudaSuccess;
    }
    return __real_cudaOccupancyMaxActiveClusters(n, f, c);
}

cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *c,
                                       const void *f, void **args)
{
    if (too_large(c))
        return cudaErrorInvalidClusterSize;
    return __real_cudaLaunchKernelExC(c, f, args);
}
}
