"""A generic call that fails after its launches has waited for them: their result
goes to a pinned slot that the next call, of any thread, may be given."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from vsmc_b200 import capi as C

    C.lib()
    return C


class Call:
    """The generic calls over N weights on a stream."""

    def __init__(self, capi, N, stream):
        self.capi, self.N, self.stream = capi, N, stream.cuda_stream
        self.w = torch.full((N,), 1.0 / N, dtype=torch.float64, device="cuda")
        self.lw = torch.zeros(N, dtype=torch.float64, device="cuda")
        self.inc = torch.from_numpy(np.random.default_rng(N).normal(size=N)).cuda()
        self.rep = torch.empty(2 * N, dtype=torch.int32, device="cuda")
        self.cf = torch.empty(2 * N, dtype=torch.int32, device="cuda")
        self.bytes = max(capi.resample_workspace_size(N),
                         capi.resample_mn_workspace_size(N, 2 * N))
        self.ws = torch.empty(self.bytes, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def resample(self):
        return self.capi.resample(3, self.N, self.w.data_ptr(), self.capi.threefry_state(5),
                                  self.rep.data_ptr(), self.cf.data_ptr(), self.ws.data_ptr(),
                                  self.bytes, stream=self.stream)

    def resample_mn(self):
        return self.capi.resample_mn(0, self.N, 2 * self.N, self.w.data_ptr(),
                                     self.capi.threefry_state(5), self.rep.data_ptr(),
                                     self.cf.data_ptr(), self.ws.data_ptr(), self.bytes,
                                     stream=self.stream)

    def weight_add_log(self):
        return self.capi.weight_add_log(self.N, self.lw.data_ptr(), self.w.data_ptr(), None,
                                        stream=self.stream)

    def weight_ess(self):
        return self.capi.weight_ess(self.N, self.lw.data_ptr(), self.w.data_ptr(),
                                    self.inc.data_ptr(), True, stream=self.stream)


def leave_error(call, stream):
    """A call on a stream that is being captured is refused (it waits for its
    result); the refusal stays behind as the library's last CUDA error."""
    rt = ctypes.CDLL("libcudart.so.12")
    s = ctypes.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(s, 2) == 0  # relaxed
    with pytest.raises(call.capi.VsmcCudaError):
        call.weight_ess()
    graph = ctypes.c_void_p()
    rt.cudaStreamEndCapture(s, ctypes.byref(graph))
    rt.cudaGetLastError()


@pytest.mark.parametrize("N", [1000, 100000])
@pytest.mark.parametrize("name", ["resample", "resample_mn", "weight_add_log", "weight_ess"])
def test_failed_call_waits(capi, name, N):
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    call = Call(capi, N, stream)
    want = getattr(call, name)()
    leave_error(Call(capi, 2000, other), other)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)  # about 0.1 s
    try:  # refused for that error unless a CUDA call on the way has cleared it
        getattr(call, name)()
    except capi.VsmcCudaError:
        pass
    assert stream.query()
    again = getattr(call, name)()  # and the next call is itself again
    assert again == want or name == "weight_add_log"
