"""Served reductions read what an earlier request of the same resident loop
wrote: reduce X, put new values into X, reduce X again, for every element
type, packs and single elements, in loops so small that a CTA meets its own
sources again."""
import numpy as np
import pytest

import gen

pytestmark = pytest.mark.gpu

NP_T = {"int32": np.int32, "uint32": np.uint32, "int64": np.int64, "uint64": np.uint64,
        "float32": np.float32, "float64": np.float64}


@pytest.mark.parametrize("ctas", [1, 2, 0])
@pytest.mark.parametrize("dt", sorted(NP_T))
def test_reduce_sees_the_last_put(B, heap, rs, dt, ctas):
    P, rounds = 5, 6
    team, es = (3, 1, P), np.dtype(NP_T[dt]).itemsize
    for n, shift, op, algo in ((1024, 0, "sum", "rec_dbl"), (1000, 0, "max", "linear"),
                               (333, es, "sum", "binomial")):
        xs = [gen.random_values(NP_T[dt], P, n, 50 + k) for k in range(rounds)]
        nb = xs[0][0].nbytes
        src, dst = heap(nb + 16) + shift, heap(nb + 16) + shift
        fresh = [heap(nb + 16) + shift for _ in xs]
        for off, x in zip(fresh, xs):
            B.put_rows(off, x, team=team)
        srv = B.Server(queue_slots=16, ctas=ctas, idle_seconds=5.0)
        try:
            for off, x in zip(fresh, xs):
                for t in [srv.enqueue(B.make_requests([dict(
                        kind="put", team=(3 + m, 1, 1), pe=3 + m, dest=src, src=off, n=nb)])[0])
                        for m in range(P)]:
                    srv.wait(t)
                srv.wait(srv.enqueue(B.make_requests([dict(
                    kind="reduce", op=op, dtype=dt, algo=algo, team=team, src=src, dest=dst, n=n)])[0]))
                got = B.get_rows(dst, nb, x.dtype, team=team)
                assert got.tobytes() == rs.reduce(algo, op, x).tobytes(), (op, algo, n)
        finally:
            srv.stop()
