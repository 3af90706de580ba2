// resample_launch.cuh -- the resamplings and filter steps of the library as
// host calls.  Their kernels (one cluster for small filters, the launch
// sequence for the others, six schemes, three kinds of weights) are compiled
// once, in resample_launch.cu: instantiated in every caller they doubled the
// library's device code, which the first call of a process loads.
#pragma once

#include "cv_kernels.cuh"

namespace vsmc_b200 {

constexpr int kRcMaxCtas = 16; // CTAs of a cluster (above 8: non-portable)
constexpr int kRcGroups = 2;   // tiles of a CTA, at most
constexpr int kRcMaxTiles = kRcMaxCtas * kRcGroups;

// Whether a resampling of N weights to Nout children (0: N) runs in one
// cluster: its weights and its uniforms must fit in kRcMaxTiles tiles.
inline bool rc_fits(long long N, long long Nout)
{
    const long long n = Nout > N ? Nout : N;
    return resample_ntiles(n) <= kRcMaxTiles;
}

// The one-cluster forms (rc_fits): a resampling of given weights whose
// control block goes to *out; a filter step's finalisation and resampling.
// False: the device has no room for the cluster, nothing is launched.
bool launch_cluster_resample(int scheme, WeightsGiven w, long long N,
                             const EngineRef &eng, const ResampleWorkspace &ws,
                             const ResampleCtl &h, ResampleCtl *out,
                             int32_t *rep_out, int32_t *copy_from,
                             cudaStream_t s, bool cfrp);
template <typename W>
bool launch_cluster_finish(int scheme, const FinalizeArgs &fa, const W &w,
                           const ResampleWorkspace &ws, int32_t *copy_from,
                           cudaStream_t s);

// A resampling of given weights: one cluster where it fits, the launch
// sequence of resample.cuh otherwise (and for caller-supplied uniforms).
// `h` holds the call's initial control block; `slot` is a call's pinned
// memory, or nullptr.  Returns whether the result is in *slot (else in the
// workspace's control block) once the stream gets there.
bool launch_resample(int scheme, WeightsGiven w, long long N,
                     const EngineRef &eng, ResampleWorkspace &ws,
                     const ResampleCtl &h, ResampleCtl *slot,
                     const double *u_given, long long n_given,
                     int32_t *rep_out, int32_t *copy_from, cudaStream_t s,
                     bool cfrp = true);

// The M != N copy_from of a resampling's counts (launch_expand).
void launch_resample_expand(const int32_t *rep, long long M, long long N,
                            ResampleWorkspace &ws, int32_t *copy_from,
                            cudaStream_t s);

// A filter step after its tile statistics: the finalisation (fa) and the
// resampling of the weights w into copy_from (unless `resample` is false:
// a replayed step).  One cluster where it fits; else k_cv_finalize and the
// launch sequence.  seq: the event after which the sorted sequence, drawn
// elsewhere, is ready (nullptr: it is drawn here).  Returns the kernels
// launched.
int launch_finish(int scheme, const FinalizeArgs &fa,
                  const WeightsFromLog<double> &w, ResampleWorkspace &ws,
                  int32_t *copy_from, bool resample, cudaEvent_t seq,
                  cudaStream_t s);
int launch_finish(int scheme, const FinalizeArgs &fa,
                  const WeightsFromLog<float> &w, ResampleWorkspace &ws,
                  int32_t *copy_from, bool resample, cudaEvent_t seq,
                  cudaStream_t s);

// launch_spec_sorted.
void launch_sequence(long long N, const EngineRef &eng, ResampleWorkspace &ws,
                     cudaStream_t s);

} // namespace vsmc_b200
