"""Where the device has no room for a cluster (a partition of a GPU), the calls
that use one take their other way, with the same results: the library's objects
linked against a runtime that has room for 8 or for no CTAs a cluster
(tests/cpp/cluster_room.cpp)."""
import os
import subprocess
import sys

import pytest

from vsmc_b200 import build

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys
import numpy as np, torch
from oracle import oracle as O
from vsmc_b200 import capi

def run():
    out = {}
    for N in (1000, 20000, 60000):
        rng = np.random.default_rng(N)
        lw = torch.from_numpy(rng.normal(size=N) * 2.0).cuda()
        inc = torch.from_numpy(rng.normal(size=N)).cuda()
        w = torch.empty_like(lw)
        out["ess", N] = capi.weight_add_log(N, lw.data_ptr(), w.data_ptr(), inc.data_ptr())
        for use_log in (True, False):
            out["ahead", N, use_log] = capi.weight_ess(N, lw.data_ptr(), w.data_ptr(),
                                                       inc.data_ptr(), use_log)
            out["cess", N, use_log] = capi.weight_cess(N, w.data_ptr(), inc.data_ptr(), use_log)
        out["w", N], out["lw", N] = w.cpu().numpy(), lw.cpu().numpy()
        for sch in range(6):
            rep = torch.empty(N, dtype=torch.int32, device="cuda")
            cf = torch.empty(N, dtype=torch.int32, device="cuda")
            nb = capi.resample_workspace_size(N)
            ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
            words = capi.resample(sch, N, w.data_ptr(), capi.threefry_state(3, offset=1),
                                  rep.data_ptr(), cf.data_ptr(), ws.data_ptr(), nb)
            out["rep", N, sch], out["cf", N, sch] = rep.cpu().numpy(), cf.cpu().numpy()
            out["words", N, sch] = words
            for form in (0, 1):
                T = 8
                ox, oy = O.cv_simulate(T, obs_seed=2)
                with capi.CVFilter(N, T, scheme=sch, form=form, threshold=0.9, seed=7) as f:
                    f.set_observations_host(ox, oy)
                    f.initialize()
                    f.iterate(T - 1)
                    for k, v in f.history().items():
                        out["cv", N, sch, form, k] = v
    with capi.GmmSampler(O.gmm_simulate(200), N=5000, iters=16, sweeps=1) as g:
        g.initialize()
        g.iterate(16)
        out["gmm"] = g.read_params()[0]
    return out

path = sys.argv[1]
want = run()
capi._lib, capi.LIB_PATH = None, path
got = run()
for k in want:
    assert np.array_equal(want[k], got[k]), k
print("ok", len(want))
"""


@pytest.mark.parametrize("ctas", [8, 0])
def test_results_without_room(tmp_path, ctas):
    objs = [os.path.join(build.OBJ, os.path.basename(s)[:-3] + ".o") for s in build.sources()]
    if not all(map(os.path.exists, objs)):
        pytest.skip("the build's objects are not here")
    lib = str(tmp_path / "libvsmc_cuda.so")
    subprocess.run([build.NVCC, *build.ARCH, "-shared", "-Xcompiler", "-fPIC", f"-DMAX_CTAS={ctas}",
                    "-o", lib, *objs, os.path.join(build.ROOT, "tests", "cpp", "cluster_room.cpp"),
                    "-Xlinker", "--wrap=cudaOccupancyMaxActiveClusters",
                    "-Xlinker", "--wrap=cudaLaunchKernelExC"],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, lib], cwd=build.ROOT, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
