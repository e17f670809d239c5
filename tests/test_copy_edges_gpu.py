"""The copy kernels off the 16-byte grid: source and dest at every shift
against each other, blocks below, at and around a vector and a CTA's tile,
empty contributions, blocks whose ends meet inside one vector; per call and
through the serving loop.  Byte for byte against the oracle (or the rows'
concatenation); bytes beside the dest stay untouched."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import gen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu
GUARD = 64
SHIFTS = [(0, 0), (1, 0), (0, 5), (4, 12), (8, 0), (15, 15), (3, 14)]


def guarded(B, heap, x, nb, a, b, team, call):
    """Rows x at a source shifted by a; call(dst, src) writes nb bytes to a
    dest shifted by b; returns them, the guard bytes checked."""
    src, box = heap(x.shape[1] + 32) + a, heap(nb + 2 * GUARD + 32)
    B.put_rows(src, x, team=team)
    B.memset(box, 0xA5, nb + 2 * GUARD + b, team=team)
    call(box + GUARD + b, src)
    got = B.get_rows(box, nb + 2 * GUARD + b, np.uint8, team=team)
    lo = GUARD + b
    assert (got[:, :lo] == 0xA5).all() and (got[:, lo + nb:] == 0xA5).all()
    return got[:, lo:lo + nb]


@pytest.mark.parametrize("P", [1, 2, 3, 8, 33])
@pytest.mark.parametrize("nb", [1, 3, 8, 15, 16, 17, 40, 251, 4096, 4100, 8193])
def test_fcollect_alltoall_shifted(B, heap, rs, P, nb):
    team = (0, 1, P)
    x = gen.uniform_int(np.uint8, P, nb, P * 31 + nb)
    y = gen.uniform_int(np.uint8, P, P * nb, P * 37 + nb)
    for a, b in SHIFTS:
        got = guarded(B, heap, x, P * nb, a, b, team, lambda d, s: B.fcollect(d, s, nb, team=team))
        assert got.tobytes() == rs.fcollect(x).tobytes(), (a, b)
        got = guarded(B, heap, y, P * nb, a, b, team, lambda d, s: B.alltoall(d, s, nb, team=team))
        assert got.tobytes() == rs.alltoall(y).tobytes(), (a, b)


@pytest.mark.parametrize("P,nb", [(64, 4096), (64, 16383), (130, 1004), (256, 1040), (256, 200)])
def test_alltoall_of_many_vectors(B, heap, rs, P, nb):
    """Grids of more than one vector a thread."""
    y = gen.uniform_int(np.uint8, P, P * nb, P + nb)
    for a, b in ((0, 0), (0, 4), (7, 2)):
        got = guarded(B, heap, y, P * nb, a, b, (0, 1, P),
                      lambda d, s: B.alltoall(d, s, nb, team=(0, 1, P)))
        assert got.tobytes() == rs.alltoall(y).tobytes(), (a, b)


@pytest.mark.parametrize("P,most", [(1, 1), (3, 5), (8, 40), (64, 3), (127, 700), (128, 700),
                                    (200, 9)])
def test_collect_shifted(B, heap, P, most):
    rng = np.random.default_rng(P + most)
    x = gen.uniform_int(np.uint8, P, most, P)
    for a, b in SHIFTS:
        counts = rng.integers(0, most + 1, P)
        counts[rng.integers(P)] = most
        want = np.concatenate([x[k, :c] for k, c in enumerate(counts)])
        got = guarded(B, heap, x, len(want), a, b, (0, 1, P),
                      lambda d, s: B.collect(d, s, counts.astype(np.uint64), team=(0, 1, P)))
        assert (got == want).all(), (a, b)


@pytest.mark.parametrize("nb", [1, 15, 16, 31, 4099])
def test_broadcast_shifted(B, heap, nb):
    P, root = 5, 3
    x = gen.uniform_int(np.uint8, P, nb, nb)
    for a, b in SHIFTS:
        got = guarded(B, heap, x, nb, a, b, (0, 1, P),
                      lambda d, s: B.broadcast(root, d, s, nb, team=(0, 1, P)))
        for j in range(P):
            assert (got[j] == (0xA5 if j == root else x[root])).all(), (a, b, j)


@pytest.mark.parametrize("nb", [1, 15, 16, 200, 4097, 32767, 32768, 40001, 70013])
def test_served_copies_shifted(B, heap, rs, nb):
    team, P = (0, 1, 4), 4
    y = gen.uniform_int(np.uint8, P, P * nb, nb)
    srv = B.Server(queue_slots=8)
    try:
        for a, b in SHIFTS:
            for kind, rows, want in (("fcollect", y[:, :nb].copy(), None), ("alltoall", y, None),
                                     ("put", y, 1), ("get", y, 0)):
                def call(d, s):
                    r = dict(kind=kind, team=team if want is None else (0, 1, 1), pe=1, dest=d,
                             src=s, n=nb)
                    srv.wait(srv.enqueue(B.make_requests([r])[0]))
                got = guarded(B, heap, rows, nb if want is not None else P * nb, a, b, team, call)
                if kind == "fcollect":
                    assert got.tobytes() == rs.fcollect(rows).tobytes(), (kind, a, b)
                elif kind == "alltoall":
                    assert got.tobytes() == rs.alltoall(rows).tobytes(), (kind, a, b)
                else:
                    for j in range(P):
                        exp = y[1 - want, :nb] if j == want else np.full(nb, 0xA5, np.uint8)
                        assert (got[j] == exp).all(), (kind, a, b, j)
    finally:
        srv.stop()


WIDE_COLLECT = textwrap.dedent("""
    import sys
    import numpy as np
    sys.path[:0] = [{pkg!r}]
    import b200shm as B
    B.init(1100, 1 << 20)
    rng = np.random.default_rng(3)
    for P, most in ((135, 50), (136, 50), (1031, 40), (1032, 40), (1100, 3)):
        team, counts = (0, 1, P), rng.integers(0, most + 1, P)
        x = rng.integers(0, 256, (P, most), dtype=np.uint8)
        want = np.concatenate([x[k, :c] for k, c in enumerate(counts)])
        for a, b in ((0, 0), (3, 5)):
            src, dst = B.malloc(most + 16), B.malloc(len(want) + 32)
            B.put_rows(src + a, x, team=team)
            B.memset(dst, 0xA5, len(want) + 32, team=team)
            B.collect(dst + b, src + a, counts.astype(np.uint64), team=team)
            got = B.get_rows(dst, len(want) + 32, np.uint8, team=team)
            assert (got[:, b:b + len(want)] == want).all(), (P, a, b)
            assert (got[:, :b] == 0xA5).all() and (got[:, b + len(want):] == 0xA5).all()
            B.free(src); B.free(dst)
    B.finalize()
    print("ok")
""")


def test_collect_of_wide_teams():
    """Size tables of each kind: the small and the large kernel parameter, and
    the one in device memory, on both sides of their limits."""
    code = WIDE_COLLECT.format(pkg=os.path.join(ROOT, "osss-ucx_b200"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
