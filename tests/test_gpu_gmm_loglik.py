"""The tempered sampler's FP64 likelihood: a table-driven 2^t, products of
densities and one logarithm per particle, against numpy's extended precision,
at the edges of its loops (rounds of 16 points, exponents moved every 8 rounds)
and for every lane split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


def exact(data, p):
    x = data.astype(np.longdouble)
    out = np.zeros(len(p), np.longdouble)
    for i, r in enumerate(p):
        mu, lam, w = (r[4 * k:4 * k + 4].astype(np.longdouble)[:, None] for k in range(3))
        e = w * np.exp(0.5 * np.log(lam) - 0.5 * lam * (x - mu) ** 2)
        out[i] = np.log(e.sum(0) + np.longdouble(1e-13)).sum()
    return out


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 127, 128, 129, 1000, 1037])
def test_loglik_against_extended_precision(capi, n):
    rng = np.random.default_rng(n)
    data = np.array([-3.0, 0.0, 3.0, 6.0])[rng.integers(0, 4, n)] + 0.55 * rng.standard_normal(n)
    data[-1] += 40.0 * (n > 100)  # one far point: densities at the 1e-13 floor
    if n == 1:
        data = np.array([0.7, 0.9])
    N = 300
    want = None
    for group in (1, 2, 4, 8, 16):
        with capi.GmmSampler(data, N=N, iters=16, sweeps=2, group=group) as s:
            s.initialize()
            s.iterate(4)
            p, _, _ = s.read_params()
            ll = s.loglik(capi.FP64)
        assert np.array_equal(ll, p[:, 13])
        if want is None:
            want, first = exact(data, p), ll
            # per point at most a few ulps of its log density (|log p| <= 30), plus
            # the rounding of the whole
            tol = 2.0 ** -52 * (8.0 * len(data) + 2.0 * np.abs(want))
            assert np.all(np.abs(ll - want) <= tol)
        assert np.array_equal(ll, first), group
