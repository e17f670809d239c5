"""Float trees whose lanes hold up to 128 leaves: team sizes around 128, 256
and 512, with and without extra members and edges, columns few and many, both
tree orders; bit for bit against the oracle."""
import numpy as np
import pytest

import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [127, 128, 129, 255, 256])
@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("n", [1, 65, 4096, 40001, 90000])
def test_wide_trees(B, heap, rs, P, dt, n):
    x = gen.normal(np.dtype(dt), P, n, P + n)
    team, es = (0, 1, P), np.dtype(dt).itemsize
    for algo in ("rec_dbl", "binomial"):
        want = rs.reduce(algo, "sum", x).tobytes()
        for shift in (0, es):
            src, dst = heap(x[0].nbytes + 16) + shift, heap(x[0].nbytes + 16) + shift
            B.put_rows(src, x, team=team)
            B.reduce("sum", dt, algo, dst, src, n, team=team)
            assert B.get_rows(dst, x[0].nbytes, x.dtype, team=team).tobytes() == want, (algo, shift)
