"""The generic calls' pinned slots and memory pool belong to one context: after
cudaDeviceReset the next context, whose handle may be the same, gets its own
(tests/cpp/scratch_main.cu)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def test_device_reset(tmp_path):
    exe = str(tmp_path / "scratch_main")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-O2",
                    os.path.join(ROOT, "tests", "cpp", "scratch_main.cu"),
                    os.path.join(ROOT, "vsmc_b200", "csrc", "call_scratch.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
