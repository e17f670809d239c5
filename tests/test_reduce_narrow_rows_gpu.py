"""Reductions of 1- and 2-byte elements off the 16-byte grid, on both sides of
the count (2^18 over all members) from which they go in packs, and chains that
one lane folds alone next to chains several lanes share; bit for bit against
the oracle, nothing beside the dest."""
import numpy as np
import pytest

import gen
from test_reduce_edges_gpu import shifted_reduce

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["int8", "uint8", "int16", "uint16"])
@pytest.mark.parametrize("P", [1, 2, 7, 15, 16, 33])
@pytest.mark.parametrize("past", [-1, 0, 1, 500])
def test_around_the_line(B, heap, rs, dt, P, past):
    es, n = np.dtype(dt).itemsize, (1 << 18) // P + past
    x = gen.random_values(np.dtype(dt), P, n, P + n)
    for op in ("sum", "max", "xor"):
        want = rs.reduce("rec_dbl", op, x).tobytes()
        for shift in (0, es, 16 - es, 96):
            assert shifted_reduce(B, heap, "rec_dbl", op, x, shift, shift).tobytes() == want, (op, shift)


@pytest.mark.parametrize("dt", ["int32", "int64", "float32", "float64", "complex64", "complex128"])
@pytest.mark.parametrize("P", [2, 9, 15, 16, 17, 31])
def test_one_lane_and_several(B, heap, rs, dt, P):
    es = np.dtype(dt).itemsize
    for n in (3, 1000, 40003):
        x = gen.random_values(np.dtype(dt), P, n, 7 * P + n)
        for algo in ("linear", "binomial"):
            for op in ("sum", "prod"):
                y = x if op == "sum" or "int" in dt else (1 + x.real.dtype.type(0.01) * x).astype(dt)
                want = rs.reduce(algo, op, y).tobytes()
                for shift in (0, es):
                    got = shifted_reduce(B, heap, algo, op, y, shift, shift)
                    assert got.tobytes() == want, (algo, op, n, shift)
