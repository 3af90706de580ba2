// resample_cluster_f64.cu -- the one-cluster filter step over double log-weights:
// see resample_cluster.cu.
#include "resample_cluster.cuh"

namespace vsmc_b200 {

template bool launch_cluster_finish<WeightsFromLog<double>>(
    int, const FinalizeArgs &, const WeightsFromLog<double> &,
    const ResampleWorkspace &, int32_t *, cudaStream_t);

} // namespace vsmc_b200
