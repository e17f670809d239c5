"""How the lanes of a column share the members of a reduction, built for the
host from the source the kernels run (tests/c/lane_model.cu): shares lie end
to end over all members, up to the largest member count an int holds.  Needs
nvcc (no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_lane_shares_cover_every_member(tmp_path):
    if not (os.path.exists(NVCC) or shutil.which("nvcc")):
        pytest.skip("nvcc is not available")
    exe = str(tmp_path / "lane_model")
    subprocess.run([NVCC if os.path.exists(NVCC) else "nvcc", "-O2", "-std=c++17",
                    "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "osss-ucx_b200", "csrc"),
                    os.path.join(ROOT, "tests", "c", "lane_model.cu"), "-o", exe],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
