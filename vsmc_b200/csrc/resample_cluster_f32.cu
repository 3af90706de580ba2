// resample_cluster_f32.cu -- the one-cluster filter step over float log-weights:
// see resample_cluster.cu.
#include "resample_cluster.cuh"

namespace vsmc_b200 {

template bool launch_cluster_finish<WeightsFromLog<float>>(
    int, const FinalizeArgs &, const WeightsFromLog<float> &,
    const ResampleWorkspace &, int32_t *, cudaStream_t);

} // namespace vsmc_b200
