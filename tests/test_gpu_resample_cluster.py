"""Resampling of up to 65536 particles runs as one thread-block cluster: its
edges (tiles of 2048, one or two tiles a CTA, 1 to 16 CTAs) against the oracle,
and device-drawn sequences against the launch sequence larger sizes use."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.gpu_util import dev, empty

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 7, 2047, 2048, 2049, 6000, 16 * 2048, 16 * 2048 + 1, 20 * 2048 + 5, 65535,
         65536, 65537]


def weights(kind, N, seed):
    rng = np.random.default_rng(seed)
    if kind == "lognormal":
        lw = rng.normal(size=N) * 2.0
        w = np.exp(lw - lw.max())
        return w / w.sum()
    if kind == "sparse":  # few parents, leading zeros
        w = np.zeros(N)
        k = rng.integers(N // 2, N, size=min(N, 5))
        w[k] = rng.uniform(0.5, 1.5, size=k.size)
        w[-1] += 0.25
        return w / w.sum()
    if kind == "ties":  # every addition to the sum a rounding tie, then ordinary weights
        w = rng.uniform(0.5, 1.5, size=N) * (0.5 / N)
        w[: N // 2] = 2.0 ** -54
        w[0] = 0.5
        return w
    return np.full(N, 1.0 / N)


def run(capi, scheme, w, seed, skip, align=0):
    N = w.size
    wd = dev(w)
    rep = torch.empty(N + 8, dtype=torch.int32, device="cuda")
    cf = torch.full((N + 8,), -7, dtype=torch.int32, device="cuda")
    nb = capi.resample_workspace_size(N)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    rng = capi.threefry_state(seed, offset=skip)
    words = capi.resample(scheme, N, wd.data_ptr(), rng, rep.data_ptr() + 4 * align,
                          cf.data_ptr() + 4 * align, ws.data_ptr(), nb)
    cf = cf.cpu().numpy()
    assert (cf[:align] == -7).all() and (cf[N + align:] == -7).all()
    return rep.cpu().numpy()[align:N + align], cf[align:N + align], words


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


@pytest.mark.parametrize("kind", ["lognormal", "sparse", "ties", "equal"])
@pytest.mark.parametrize("sch", range(6))
def test_against_oracle(capi, sch, kind):
    for N in SIZES:
        w = weights(kind, N, N + sch)
        ref_rep, ref_cf, ref_words = O.resample(sch, w, 103, 3)[:3]
        rep, cf, words = run(capi, sch, w, 103, 3, align=N % 3)
        assert words == ref_words, N
        # a sorted sequence goes through the device's log and exp, which may
        # round otherwise than the host's: none differs at these sizes
        assert np.array_equal(rep, ref_rep), N
        assert np.array_equal(cf, ref_cf), N


@pytest.mark.parametrize("sch", [0, 1, 3, 4])
@pytest.mark.parametrize("M,N", [(5000, 65536), (65536, 300), (40000, 2049), (1, 4096)])
def test_other_number_of_children(capi, sch, M, N):
    w = weights("lognormal", M, M + N)
    ref_rep, ref_cf, ref_words = O.resample(sch, w, 19, 2, M=M, N=N)[:3]
    rep, cf = empty(M, torch.int32), empty(N, torch.int32)
    nb = capi.resample_mn_workspace_size(M, N)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    wd = dev(w)
    words = capi.resample_mn(sch, M, N, wd.data_ptr(), capi.threefry_state(19, offset=2),
                             rep.data_ptr(), cf.data_ptr(), ws.data_ptr(), nb)
    assert words == ref_words
    assert np.array_equal(rep.cpu().numpy()[:M], ref_rep)
    assert np.array_equal(cf.cpu().numpy()[:N], ref_cf)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("sch", range(6))
def test_filter_equals_launch_sequence(capi, sch, form):
    """A filter beside one of more than 65536 particles in a batch runs the
    launch sequence; alone it resamples in a cluster."""
    T = 6
    sizes = [1000, 2049, 30000, 40000, 65536]
    ox, oy = capi.cv_simulate(T, obs_seed=5)
    with capi.CVBatch(len(sizes) + 1, scheme=sch, form=form, threshold=0.9) as b:
        slots = [b.admit(n, T, seed=11 + k) for k, n in enumerate(sizes + [70000])]
        b.set_observations(slots, [(ox, oy)] * len(slots))
        b.run(slots)
        for k, n in enumerate(sizes):
            want = b.history(slots[k])
            with capi.CVFilter(n, T, scheme=sch, form=form, threshold=0.9, seed=11 + k) as f:
                f.set_observations_host(ox, oy)
                f.initialize()
                f.iterate(T - 1)
                got = f.history()
            assert want["resampled"].sum() > 0
            for q in want:
                assert np.array_equal(got[q], want[q]), (n, q)
