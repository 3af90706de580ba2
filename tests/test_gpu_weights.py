"""The weight updates and prospective ESS / CESS at the edges of their tiles (2048) and of
the one-cluster form (65536), against extended precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 2047, 2048, 2049, 16 * 2048, 16 * 2048 + 1, 65535, 65536, 65537, 33 * 2048 + 9]

# exp of arguments down to -60 (rounded to 60 * 2^-53 = 7e-15) and sums whose chains are shorter
# than 100 roundings (1.1e-14), squared and divided: below 5e-14
RTOL = 1e-13


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


def log_weights(kind, N, rng):
    lw = np.maximum(rng.normal(size=N) * 3.0, -30.0)
    if kind == "gaps":  # zero weights, the first tile all of them where another follows
        lw[rng.uniform(size=N) < 0.4] = -np.inf
        lw[: min(2048, N - 1)] = -np.inf
        lw[N - 1] = -1.0
    return lw


def put(a, align):
    t = torch.full((a.size + 8,), 7.0, dtype=torch.float64, device="cuda")
    t[align:align + a.size] = torch.from_numpy(a)
    return t, t.data_ptr() + 8 * align


@pytest.mark.parametrize("align", [0, 1])
@pytest.mark.parametrize("kind", ["normal", "gaps"])
@pytest.mark.parametrize("N", SIZES)
def test_weights(capi, N, kind, align):
    rng = np.random.default_rng([N, align, kind == "gaps"])
    lw, inc = log_weights(kind, N, rng), rng.normal(size=N)
    L = np.longdouble
    lt, lp = put(lw, align)
    wt, wp = put(np.zeros(N), align)
    it, ip = put(inc, align)

    def taken(t):
        a = t.cpu().numpy()
        assert (a[:align] == 7.0).all() and (a[align + N:] == 7.0).all()
        return a[align:align + N]

    ess = capi.weight_add_log(N, lp, wp, None)
    lw = lw - lw.max()
    e = np.exp(lw.astype(L))
    assert np.array_equal(taken(lt), lw)
    np.testing.assert_allclose(taken(wt), (e / e.sum()).astype(float), rtol=RTOL, atol=0)
    np.testing.assert_allclose(ess, float(e.sum() ** 2 / (e * e).sum()), rtol=RTOL)
    w = taken(wt).astype(L)
    f = np.exp((lw + inc).astype(L))
    for use_log in (True, False):
        b = np.exp(inc.astype(L)) if use_log else np.abs(inc).astype(L)
        if not use_log:
            it, ip = put(np.abs(inc), align)
        v = f if use_log else w * b
        want = float(v.sum() ** 2 / (v * v).sum())
        np.testing.assert_allclose(capi.weight_ess(N, lp, wp, ip, use_log), want, rtol=RTOL)
        want = float((w * b).sum() ** 2 / (w * b * b).sum())
        np.testing.assert_allclose(capi.weight_cess(N, wp, ip, use_log), want, rtol=RTOL)
    it, ip = put(inc, align)
    ess = capi.weight_add_log(N, lp, wp, ip)
    lw = lw + inc
    lw = lw - lw.max()
    e = np.exp(lw.astype(L))
    assert np.array_equal(taken(lt), lw)
    np.testing.assert_allclose(taken(wt), (e / e.sum()).astype(float), rtol=RTOL, atol=0)
    np.testing.assert_allclose(ess, float(e.sum() ** 2 / (e * e).sum()), rtol=RTOL)
