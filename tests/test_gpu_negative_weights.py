"""Residual schemes over weights whose integer parts are negative in sum: as many
residual children as would not fit the sequence's arrays.  Such a call is
degenerate."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


@pytest.mark.parametrize("sch", [1, 4, 5])
@pytest.mark.parametrize("N", [100, 2048, 6000, 40000, 65536, 70000])
def test_refused(capi, N, sch):
    rep = torch.empty(2 * N, dtype=torch.int32, device="cuda")
    cf = torch.empty(2 * N, dtype=torch.int32, device="cuda")
    nb = max(capi.resample_workspace_size(N), capi.resample_mn_workspace_size(N, 2 * N))
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    w = torch.full((N,), 0.25 / N, dtype=torch.float64, device="cuda")
    rng = capi.threefry_state(1)
    for big in (-1.5 / N, -4.0, -1e6):
        w[N // 3] = big
        for call in (lambda: capi.resample(sch, N, w.data_ptr(), rng, rep.data_ptr(),
                                           cf.data_ptr(), ws.data_ptr(), nb),
                     lambda: capi.resample_mn(sch, N, 2 * N, w.data_ptr(), rng, rep.data_ptr(),
                                              cf.data_ptr(), ws.data_ptr(), nb)):
            with pytest.raises(capi.VsmcCudaError) as e:
                call()
            assert e.value.status == capi.EDEGENERATE
    w.fill_(1.0 / N)  # the next call is itself again
    capi.resample(sch, N, w.data_ptr(), rng, rep.data_ptr(), cf.data_ptr(), ws.data_ptr(), nb)
    assert bool((rep[:N] == 1).all())
