"""The reduce kernel's ways to reach its columns: rows off the 16-byte grid,
dest and source shifted against each other, elements at odd byte offsets,
counts below a pack and around the lane and line boundaries, team sizes on
both sides of every split rule; and the exact replay of order-dependent
MIN/MAX columns inside the streaming kernel and, for larger teams, after it.
Bit for bit against the oracle; bytes beside the dest stay untouched."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import gen
from test_reduce_gpu import NAME, nan_equal_bytes, special

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

GUARD = 256


def shifted_reduce(B, heap, algo, op, x, src_shift, dst_shift, in_place=False):
    """The reduction with source and dest that many bytes past a 256-byte
    boundary; checks the guard bytes on both sides of the dest."""
    P, nb = x.shape[0], x[0].nbytes
    team = (0, 1, P)
    src = heap(2 * GUARD + nb) + GUARD + src_shift
    dst = src if in_place else heap(2 * GUARD + nb) + GUARD + dst_shift
    if not in_place:
        B.memset(dst - GUARD, 0xA5, 2 * GUARD + nb - dst_shift, team=team)
    B.put_rows(src, x, team=team)
    B.reduce(op, NAME[x.dtype], algo, dst, src, x.shape[1], team=team)
    if not in_place:
        got = B.get_rows(dst - GUARD, 2 * GUARD + nb - dst_shift, np.uint8, team=team)
        assert (got[:, :GUARD] == 0xA5).all() and (got[:, GUARD + nb:] == 0xA5).all()
    return B.get_rows(dst, nb, x.dtype, team=team)


@pytest.mark.parametrize("dt", ["int8", "int16", "int32", "int64", "float32", "float64",
                                "complex64", "complex128"])
@pytest.mark.parametrize("P", [1, 2, 3, 7, 8, 9, 16, 24, 64, 127, 130])
def test_shifted_rows(B, heap, rs, dt, P):
    es = np.dtype(dt).itemsize
    for k, n in enumerate((1, 5, 33, 257, 4096 // es + 37)):
        x = gen.random_values(np.dtype(dt), P, n, 31 * P + n)
        algo = ["rec_dbl", "rabenseifner", "linear", "rec_dbl", "binomial"][k]
        for op in ("sum", "max") if dt[0] in "if" else ("sum",):
            want = rs.reduce(algo, op, x)
            for a, b in ((0, 0), (es, es), (3 * es, 3 * es), (es, 0), (1, 1), (2, 7)):
                got = shifted_reduce(B, heap, algo, op, x, a, b)
                assert nan_equal_bytes(got, want), (algo, op, n, a, b)


@pytest.mark.parametrize("algo", ["linear", "binomial", "rec_dbl", "rabenseifner", "rabenseifner2"])
@pytest.mark.parametrize("dt", ["float32", "float64"])
def test_order_dependent_columns(B, heap, rs, algo, dt):
    """NaNs with payloads and zeros of both signs among the operands, in every
    column: the warp's own replay up to 127 members, the deferred list above."""
    es = np.dtype(dt).itemsize
    for P in (1, 2, 3, 5, 16, 24, 33, 64, 100, 127, 128, 255):
        for n in (1, 40, 1501):
            x = special(dt, P, n, 1000 * P + n)
            for op in ("min", "max"):
                want = rs.reduce(algo, op, x)
                for a, b, in_place in ((0, 0, False), (es, es, True), (es, 0, False)):
                    got = shifted_reduce(B, heap, algo, op, x, a, b, in_place)
                    assert got.tobytes() == want.tobytes(), (P, n, op, a, b, in_place)


def test_zeros_of_one_sign_and_of_both(B, heap, rs):
    """Columns whose result is a zero: all +0, all -0, both (order dependent),
    and both beside a larger operand (not order dependent)."""
    P, n = 24, 4 * 257
    for dt in (np.float32, np.float64):
        x = np.zeros((P, n), dt)
        x[:, 1::4] = -0.0
        x[::3, 2::4] = -0.0
        x[::3, 3::4] = -0.0
        x[5, 3::4] = 1.0
        for op, y in (("max", x), ("min", -x)):
            for algo in ("rec_dbl", "linear", "rabenseifner"):
                got = shifted_reduce(B, heap, algo, op, y, 0, 0)
                assert got.tobytes() == rs.reduce(algo, op, y).tobytes(), (dt, op, algo)


def test_more_turns_than_bits(tmp_path):
    """A grid of one CTA per SM, so that a warp takes more than 32 turns and
    the last bit of its record stands for several: in place, 2 members."""
    code = textwrap.dedent("""
        import sys
        sys.path[:0] = [%r, %r, %r]
        import numpy as np, oracle, b200shm as B
        from test_reduce_gpu import special
        B.init(2, 24 << 20)
        n = 2500001
        x = special("float64", 2, n, 3)
        x[:, : n // 2] = np.abs(np.nan_to_num(x[:, : n // 2])) + 1.0  # sparse turns too
        src = B.malloc(x[0].nbytes)
        B.put_rows(src, x)
        B.reduce("max", "float64", "rec_dbl", src, src, n)
        got = B.get_rows(src, x[0].nbytes, np.float64)
        assert got.tobytes() == oracle.Restatement().reduce("rec_dbl", "max", x).tobytes()
        print("same")
    """) % tuple(os.path.join(ROOT, d) for d in ("osss-ucx_b200", "oracle", "tests"))
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, B200SHM_REDUCE_CTAS_PER_SM="1"))
    assert p.returncode == 0 and "same" in p.stdout, p.stderr[-2000:]
