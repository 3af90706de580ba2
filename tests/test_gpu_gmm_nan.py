"""A data point that is NaN makes the tempered sampler's likelihood NaN and its
run degenerate, in both forms and wherever the point stands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("at", [0, 1, 77, 256, 299])
@pytest.mark.parametrize("form", [0, 1])
def test_nan_point(capi, form, at, sign):
    rng = np.random.default_rng(1)
    data = np.array([-3.0, 0.0, 3.0, 6.0])[rng.integers(0, 4, 300)] + 0.55 * rng.standard_normal(300)
    data[at] = np.copysign(np.nan, sign)
    with capi.GmmSampler(data, N=500, iters=16, sweeps=2, form=form) as s:
        s.initialize()
        for f in (capi.FP64, capi.MIXED):
            assert np.isnan(s.loglik(f)).all()
        s.iterate(3)
        with pytest.raises(capi.VsmcCudaError) as e:
            s.history()
        assert e.value.status == capi.EDEGENERATE
        assert np.isnan(s.log_evidence()[0])
