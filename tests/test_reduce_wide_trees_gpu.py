"""Float trees over more than 256 members, where two or four lanes hold 64 or
128 leaves each, with extra members (257, 300, 511, 513) and without, few and
many columns, rows on and off the grid; real and complex, SUM and PROD, bit
for bit against the oracle.  In a process of its own: the teams are wider
than the test session's world."""
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
    sys.path[:0] = [{pkg!r}, {oracle!r}]
    import b200shm as B
    import oracle
    rs = oracle.Restatement()
    B.init(520, 2 << 20)
    P, dt = {P}, np.dtype({dt!r})
    V, es, team = max(1, 16 // dt.itemsize), dt.itemsize, (0, 1, P)
    real = np.empty(0, dt).real.dtype
    src, dst = B.malloc(1 << 19), B.malloc(1 << 19)
    # 37888 threads fill the chip: on both sides of that at 2, 4 and 8 lanes
    for cols in (19500, 10500, 5200) if P < 512 else (10500, 5200, 700):
        n = cols * V + V // 2
        rng = np.random.default_rng(P + cols)
        for op in ("sum", "prod"):
            x = rng.standard_normal((P, n)).astype(dt)
            if dt.kind == "c":
                x = (x + 1j * rng.standard_normal((P, n))).astype(dt)
            if op == "prod":
                x = (1 + real.type(0.01) * x).astype(dt)
            for algo in ("rec_dbl", "binomial") if P in (300, 512) else ("rec_dbl",):
                want = rs.reduce(algo, op, x).tobytes()
                for shift in (0, es):
                    B.put_rows(src + shift, x, team=team)
                    B.reduce(op, dt.name, algo, dst + shift, src + shift, n, team=team)
                    got = B.get_rows(dst + shift, n * es, dt, team=team)
                    assert got.tobytes() == want, (op, algo, cols, shift)
    B.finalize()
    print("ok")
""")


@pytest.mark.parametrize("P", [257, 300, 511, 512, 513])
@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
def test_trees_over_wide_teams(P, dt):
    code = CODE.format(pkg=os.path.join(ROOT, "osss-ucx_b200"),
                       oracle=os.path.join(ROOT, "oracle"), P=P, dt=dt)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
