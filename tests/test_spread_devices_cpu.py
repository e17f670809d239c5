"""Long fcollects, collects and broadcasts after the engine moved to another
device: the launch's shared-memory claim is asked for on that device too
(tests/c/spread_devices_model.cu, the launch code built for the host with the
runtime's call recorded).  Needs nvcc (no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_the_claim_is_made_on_every_device(tmp_path):
    if not (os.path.exists(NVCC) or shutil.which("nvcc")):
        pytest.skip("nvcc is not available")
    exe = str(tmp_path / "spread_devices_model")
    subprocess.run([NVCC if os.path.exists(NVCC) else "nvcc", "-O1", "-std=c++17",
                    "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "osss-ucx_b200", "csrc"),
                    os.path.join(ROOT, "tests", "c", "spread_devices_model.cu"), "-o", exe],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert r.returncode == 0, r.stdout + r.stderr
