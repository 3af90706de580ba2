// resample_launch.cu -- see resample_launch.cuh.
#include "resample_cluster.cuh"

namespace vsmc_b200 {

int launch_finish(int scheme, const FinalizeArgs &fa,
                  const WeightsFromLog<double> &w, ResampleWorkspace &ws,
                  int32_t *copy_from, bool resample, cudaEvent_t seq,
                  cudaStream_t s)
{
    return launch_finish_t(scheme, fa, w, ws, copy_from, resample, seq, s);
}

int launch_finish(int scheme, const FinalizeArgs &fa,
                  const WeightsFromLog<float> &w, ResampleWorkspace &ws,
                  int32_t *copy_from, bool resample, cudaEvent_t seq,
                  cudaStream_t s)
{
    return launch_finish_t(scheme, fa, w, ws, copy_from, resample, seq, s);
}

void launch_sequence(long long N, const EngineRef &eng, ResampleWorkspace &ws,
                     cudaStream_t s)
{
    launch_spec_sorted(N, eng, ws, s);
}

void launch_resample_expand(const int32_t *rep, long long M, long long N,
                            ResampleWorkspace &ws, int32_t *copy_from,
                            cudaStream_t s)
{
    launch_expand(rep, M, N, ws, copy_from, s);
}

} // namespace vsmc_b200
