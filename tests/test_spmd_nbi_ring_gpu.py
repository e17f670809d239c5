"""Fetching atomics left outstanding over more requests than the serving ring
has slots (tests/c/spmd_nbi_ring.c): each gets its own old value."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "osss-ucx_b200", "lib")


@pytest.mark.gpu
def test_fetches_outlive_their_ring_slots(tmp_path):
    import __graft_entry__
    __graft_entry__.build_library()
    exe = str(tmp_path / "spmd_nbi_ring")
    subprocess.run(["gcc", "-std=gnu11", "-O2", "-Wall", "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "c", "spmd_nbi_ring.c"), "-L" + LIB,
                    "-lshmem_b200", "-Wl,-rpath," + LIB, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
