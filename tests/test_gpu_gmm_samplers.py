"""Tempered samplers with different numbers of data points side by side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("large", [1000, 2000, 16384])
def test_smaller_sampler_created_between(capi, form, large):
    data = np.random.default_rng(large).normal(size=large) * 3.0
    kw = dict(N=500, iters=16, sweeps=1, form=form)
    with capi.GmmSampler(data, **kw) as s:
        s.initialize()
        s.iterate(4)
        want = s.read_params()[0]
    with capi.GmmSampler(data, **kw) as s:
        s.initialize()
        s.iterate(2)
        with capi.GmmSampler(data[:50].copy(), **kw) as small:
            small.initialize()
            s.iterate(2)
            small.iterate(2)
            small.history()
        got = s.read_params()[0]
    assert np.array_equal(got, want)
