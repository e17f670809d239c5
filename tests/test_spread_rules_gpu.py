"""fcollect, collect and broadcast on both sides of the lines between bytes,
vectors and the broadcast to few members: row lengths around 1024 and 8192
bytes, on and off the 16-byte grid, and broadcasts around 128 KiB and 32 MiB in
all; byte for byte, nothing beside the dest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 64


def check(B, x, run, src, dst, a, b, want, skip=None):
    P, nb = len(x), want.shape[0]
    team = (0, 1, P)
    B.put_rows(src + a, x, team=team)
    B.memset(dst, 0xA5, nb + 2 * GUARD, team=team)
    run(dst + GUARD + b, src + a, team)
    got = B.get_rows(dst, nb + 2 * GUARD, np.uint8, team=team)
    at = GUARD + b
    for j in range(P):
        if j != skip:
            assert (got[j, at:at + nb] == want).all(), (P, nb, a, b, j)
    assert (got[:, :at] == 0xA5).all() and (got[:, at + nb:] == 0xA5).all(), (P, nb, a, b)


@pytest.mark.parametrize("P", [1, 2, 3, 8, 17, 100])
@pytest.mark.parametrize("row", [1, 15, 1008, 1024, 1040, 8176, 8192, 8193, 8208])
def test_fcollect_and_collect_rows(B, heap, P, row):
    rng = np.random.default_rng(P + row)
    src, dst = heap(row + 64), heap(row + P * 16 + 4 * GUARD)
    for nb in {max(1, row // P), max(16, row // P // 16 * 16)}:
        x = rng.integers(0, 256, (P, nb), dtype=np.uint8)
        for a, b in ((0, 0), (16, 16), (3, 5)):
            check(B, x, lambda d, s, t: B.fcollect(d, s, nb, team=t), src, dst, a, b, x.reshape(-1))
    sizes = rng.integers(0, 2 * (row // P) + 2, P)
    sizes[0] += max(0, row - sizes.sum())
    sizes = np.minimum(sizes, row)
    while sizes.sum() > row:
        sizes[np.argmax(sizes)] -= min(sizes.max(), sizes.sum() - row)
    x = rng.integers(0, 256, (P, row), dtype=np.uint8)
    want = np.concatenate([x[k, :c] for k, c in enumerate(sizes)])
    for a, b in ((0, 0), (1, 2)):
        check(B, x, lambda d, s, t: B.collect(d, s, sizes.astype(np.uint64), team=t), src, dst, a, b, want)


@pytest.mark.parametrize("P,nb", [(2, 16), (2, 1023), (2, 5 << 20), (3, 131056), (3, 131072),
                                  (8, 1024), (8, 1040), (8, 4 << 20), (8, (4 << 20) + 16),
                                  (16, 2 << 20), (16, (2 << 20) + 16), (17, 131072), (40, 700000)])
def test_broadcast_rows(B, heap, P, nb):
    x = np.random.default_rng(P + nb).integers(0, 256, (P, nb), dtype=np.uint8)
    src, dst = heap(nb + 64), heap(nb + 4 * GUARD)
    for root, a, b in ((0, 0, 0), (P - 1, 16, 16), (P // 2, 3, 5)):
        team = (0, 1, P)
        B.memset(dst, 0xA5, nb + 4 * GUARD, team=team)
        B.put_rows(src + a, x, team=team)
        B.broadcast(root, dst + GUARD + b, src + a, nb, team=team)
        got = B.get_rows(dst, nb + 4 * GUARD, np.uint8, team=team)
        at = GUARD + b
        for j in range(P):
            want = np.full(nb, 0xA5, np.uint8) if j == root else x[root]
            assert (got[j, at:at + nb] == want).all(), (root, a, b, j)
        assert (got[:, :at] == 0xA5).all() and (got[:, at + nb:] == 0xA5).all()
