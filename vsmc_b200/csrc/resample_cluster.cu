// resample_cluster.cu -- the one-cluster resampling of given weights
// (resample_cluster.cuh) as a host call.  The filter steps' forms are in
// resample_cluster_f64.cu and resample_cluster_f32.cu: a process loads the
// modules that it uses, and the three together took 20 ms to load.
#include "resample_cluster.cuh"

namespace vsmc_b200 {

bool launch_cluster_resample(int scheme, WeightsGiven w, long long N,
                             const EngineRef &eng, const ResampleWorkspace &ws,
                             const ResampleCtl &h, ResampleCtl *out,
                             int32_t *rep_out, int32_t *copy_from,
                             cudaStream_t s, bool cfrp)
{
    RcArgs a = rc_args(N, eng, ws, rep_out, copy_from, cfrp);
    a.offset = h.offset;
    a.Nout = h.Nout;
    a.out = out;
    bool done = false;
    const RcShape sh = rc_shape(resample_ntiles(h.Nout > N ? h.Nout : N));
    rc_scheme(scheme, [&](auto res, auto seq) {
        constexpr bool Re = decltype(res)::value;
        constexpr int U = decltype(seq)::value;
        if (sh.r == 8)
            done = rc_launch(k_resample_cluster<WeightsGiven, Re, U, 8>, sh,
                             false, s, w, a);
        else
            done = rc_launch(k_resample_cluster<WeightsGiven, Re, U, 2>, sh,
                             false, s, w, a);
    });
    return done;
}

} // namespace vsmc_b200
