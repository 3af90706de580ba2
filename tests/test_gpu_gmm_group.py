"""The tempered sampler's choice of lanes per particle, where a poor one costs
more than a tenth of a sweep: between one and two waves of CTAs, and with data
that leave room for one CTA on an SM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


# (form, n, N, the lanes within 5% of the fastest of a sweep on a B200 of 148 SMs)
FAST = [(0, 4000, 20000, (8, 16)), (0, 16384, 4096, (8,)), (0, 12000, 20000, (8, 16)),
        (0, 1000, 65536, (1,)), (1, 8000, 20000, (8, 16)), (1, 16384, 20000, (8, 16)),
        (1, 16384, 65536, (4, 8)), (1, 1000, 65536, (1,)), (1, 250, 300, (16,))]


@pytest.mark.parametrize("form,n,N,lanes", FAST)
def test_choice(capi, form, n, N, lanes):
    data = np.random.default_rng(n).normal(size=n) * 3.0
    with capi.GmmSampler(data, N=N, iters=16, sweeps=1, form=form) as s:
        assert s.group() in lanes
