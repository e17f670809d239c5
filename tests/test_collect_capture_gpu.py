"""A captured collect of uneven contributions gives the same at every replay,
also where the team is too large for the table of sizes to be a kernel
parameter and the graph uploads it: the caller's sizes are gone by then."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = textwrap.dedent("""
    import sys
    import numpy as np
    import torch
    sys.path[:0] = [{pkg!r}]
    import b200shm as B
    B.init(1100, 1 << 20)
    rng = np.random.default_rng(4)
    most, graphs = 40, []
    s = torch.cuda.Stream()
    for P in (135, 1031, 1032, 1100):
        team, counts = (0, 1, P), rng.integers(0, most + 1, P).astype(np.uint64)
        x = rng.integers(0, 256, (P, most), dtype=np.uint8)
        want = np.concatenate([x[k, :int(c)] for k, c in enumerate(counts)])
        src, dst = B.malloc(most), B.malloc(len(want) + 16)
        B.put_rows(src, x, team=team)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            B.collect(dst, src, counts, team=team, stream=s.cuda_stream)
        counts[:] = 1 << 60
        graphs.append((g, team, dst, want))
    junk = [np.full(n, 0xFFFFFFFFFFFFFFF, np.uint64) for n in (1101, 1033, 1032) for _ in range(50)]
    for _ in range(3):
        for g, team, dst, want in graphs:
            B.memset(dst, 0xA5, len(want) + 16, team=team)
            g.replay()
            torch.cuda.synchronize()
            got = B.get_rows(dst, len(want) + 16, np.uint8, team=team)
            assert (got[:, :len(want)] == want).all() and (got[:, len(want):] == 0xA5).all(), team
    del g, graphs
    torch.cuda.synchronize()
    B.finalize()
    print("ok")
""")


def test_replays_of_a_captured_collect():
    code = CODE.format(pkg=os.path.join(ROOT, "osss-ucx_b200"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
