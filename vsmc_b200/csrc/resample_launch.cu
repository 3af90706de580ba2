// resample_launch.cu -- the resampling launch sequence and the choice between
// it and one cluster: see resample_launch.cuh.
#include "resample_launch.cuh"

namespace vsmc_b200 {

bool launch_resample(int scheme, WeightsGiven w, long long N,
                     const EngineRef &eng, ResampleWorkspace &ws,
                     const ResampleCtl &h, ResampleCtl *slot,
                     const double *u_given, long long n_given,
                     int32_t *rep_out, int32_t *copy_from, cudaStream_t s,
                     bool cfrp)
{
    if (u_given != nullptr || !rc_fits(N, h.Nout) ||
        !launch_cluster_resample(scheme, w, N, eng, ws, h,
                                 slot != nullptr ? slot : ws.ctl, rep_out,
                                 copy_from, s, cfrp)) {
        const ResampleCtl *src = &h;
        if (slot != nullptr) { // (pinned: copied without staging)
            *slot = h;
            src = slot;
        }
        // a failed copy leaves its error for the caller's check
        if (cudaMemcpyAsync(ws.ctl, src, sizeof(h), cudaMemcpyHostToDevice,
                            s) == cudaSuccess)
            launch_resample_core(scheme, w, N, eng, ws, u_given, n_given,
                                 false, rep_out, copy_from, s, false, cfrp,
                                 h.Nout);
        return false;
    }
    return slot != nullptr;
}

namespace {

// Dynamic shared memory that k_cv_finalize may have without asking for more
// (48 KB less its static part, rounded down).
constexpr size_t kFinalPlainSmem = 32 << 10;

template <typename W>
int launch_finish_t(int scheme, const FinalizeArgs &fa, const W &w,
                    ResampleWorkspace &ws, int32_t *copy_from, bool resample,
                    cudaEvent_t seq, cudaStream_t s)
{
    const long long N = fa.N;
    if (rc_fits(N, 0) &&
        launch_cluster_finish(scheme, fa, w, ws, copy_from, s))
        return 1;
    const size_t smem = fa.ntiles <= kFinalSmemTiles
                            ? (size_t)fa.ntiles * sizeof(double)
                            : 0;
    if (smem > kFinalPlainSmem)
        cudaFuncSetAttribute(k_cv_finalize,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kFinalSmemTiles * (int)sizeof(double));
    launch_early(true, k_cv_finalize, 1, kFinalThreads, smem, s, fa);
    if (!resample)
        return 1;
    const bool ready = seq != nullptr;
    if (ready)
        cudaStreamWaitEvent(s, seq, 0);
    launch_resample_core(scheme, w, N, fa.eng, ws, nullptr, 0,
                         /*spine_done=*/true, nullptr, copy_from, s, ready);
    return 1 +
           resample_launches(scheme, false, W::kExactNorm, W::kApprox) -
           (ready ? 5 : 0);
}

} // namespace

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
