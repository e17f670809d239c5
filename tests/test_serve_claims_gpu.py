"""Which CTA serves which request of the loop: rings of fewer and of more
slots than the claim words a CTA looks at in one go, requests of one share
and of many next to each other; every request is served exactly once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [1, 2, 31, 32, 33, 300])
@pytest.mark.parametrize("ctas", [1, 5, 0])
def test_every_request_is_served_once(B, heap, slots, ctas):
    """Fetch-adds of 1 on one counter, a put of several tiles after every
    seventh: the old values are a permutation, the copies arrive."""
    n, nb = 700, 200000
    rng = np.random.default_rng(slots)
    x = rng.integers(0, 256, (1, nb), dtype=np.uint8)
    src, dst, ctr = heap(nb), heap(nb), heap(64)
    B.put_rows(src, x, team=(1, 1, 1))
    B.memset(dst, 0, nb, team=(0, 1, 8))
    B.memset(ctr, 0, 64, team=(2, 1, 1))
    reqs = [dict(kind="put", team=(1, 1, 1), pe=k % 6 + 2, dest=dst, src=src, n=nb) if k % 7 == 6 else
            dict(kind="amo", op="fetch_add", dtype="int64", pe=2, dest=ctr, value=1) for k in range(n)]
    amos = np.array([r["kind"] == "amo" for r in reqs])
    srv = B.Server(queue_slots=slots, ctas=ctas, idle_seconds=0.01)
    try:
        _, old = B.replay(B.make_requests(reqs), np.zeros(n), srv)
    finally:
        srv.stop()
    assert (np.sort(old[amos]) == np.arange(amos.sum())).all()
    assert B.get_rows(ctr, 8, np.int64, team=(2, 1, 1))[0, 0] == amos.sum()
    got = B.get_rows(dst, nb, np.uint8, team=(2, 1, 6))
    assert (got == x).all()
