"""Sharply peaked weights: one weight 2^53 times and more the sum of all before
it, zeros between, as a likelihood far narrower than the particles gives them.
The approximate prefixes that the exact scan classifies with must keep the small
sums beside the peak, at the edges of threads, warps and tiles."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.gpu_util import dev, empty

pytestmark = pytest.mark.gpu

RTOL = 1e-9  # as the FP64 filter against the oracle elsewhere


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


def peaks(N):
    at = [2, 7, 8, 63, 64, 100, 255, 256, 2047, 2048, 2049, 4096 + 31, N // 2, N - 3]
    return sorted({p for p in at if 2 <= p < N - 2})


def peaked(N, kind, seed):
    """Weight arrays of a kind."""
    rng = np.random.default_rng([N, seed])
    if kind == "narrow":  # a Gaussian likelihood of standard normal particles
        for s in (0.3, 0.01, 0.003):
            yield np.exp(-0.5 * (rng.normal(size=N) / s) ** 2)
        return
    for p in peaks(N):
        w = np.where(rng.uniform(size=N) < 0.5, 0.0, rng.uniform(size=N) * 1e-6)
        if kind == "zeros":  # two small weights, then zeros, then the peak
            w[:p] = 0.0
            w[:2] = 1e-20, 1e-25
        else:  # small sums that the peak's roundings would move to another binade
            w[:p] = np.where(rng.uniform(size=p) < 0.3, 0.0,
                             rng.uniform(size=p) * (3e-16 / p))
            w[0] = 1e-18
        w[p] = 1.0
        yield w


@pytest.mark.parametrize("kind", ["narrow", "zeros", "small"])
@pytest.mark.parametrize("sch", range(6))
@pytest.mark.parametrize("N", [1000, 2050, 5000, 40000, 70001])
def test_resample_against_oracle(capi, N, sch, kind):
    rep, cf = empty(N, torch.int32), empty(N, torch.int32)
    nb = capi.resample_workspace_size(N)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    for k, w in enumerate(peaked(N, kind, sch)):
        w /= w.sum()
        ref_rep, ref_cf, ref_words = O.resample(sch, w, 77, 2)[:3]
        wd = dev(w)
        words = capi.resample(sch, N, wd.data_ptr(), capi.threefry_state(77, offset=2),
                              rep.data_ptr(), cf.data_ptr(), ws.data_ptr(), nb)
        assert words == ref_words, k
        assert np.array_equal(rep.cpu().numpy(), ref_rep), k
        assert np.array_equal(cf.cpu().numpy(), ref_cf), k


@pytest.mark.parametrize("N", [1000, 3000, 40000, 70000])
@pytest.mark.parametrize("sch", range(6))
def test_filter_against_oracle(capi, sch, N):
    """A filter, alone and in a batch, that resamples only when nearly one
    particle is left: its log-weights spread over many hundreds, so that most
    weights are 0."""
    T, threshold = 40, 1.2 / N
    ox, oy = O.cv_simulate(T, obs_seed=4)
    r = O.cv_filter(N, T, sch, ox, oy, seed=5, threshold=threshold)
    assert r["resampled"].sum() > 0
    with capi.CVFilter(N, T, scheme=sch, threshold=threshold, seed=5) as f:
        f.set_observations_host(ox, oy)
        f.initialize()
        f.iterate(T - 1)
        got = [f.history()]
        assert f.resample_words() == r["words_used"]
    with capi.CVBatch(1, scheme=sch, threshold=threshold) as b:
        slot = b.admit(N, T, seed=5)
        b.set_observations([slot], [(ox, oy)])
        b.run([slot])
        got.append(b.history(slot))
    for h in got:
        assert np.array_equal(h["resampled"], r["resampled"])
        for q in ("ess", "logz_inc", "mean_x", "mean_y"):
            np.testing.assert_allclose(h[q], r[q], rtol=RTOL, atol=1e-12, err_msg=q)
