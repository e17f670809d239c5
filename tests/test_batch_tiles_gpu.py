"""The batch kernels at the edges of their tiles: counts around one pass of a
CTA, around a tile, below one 16-byte pack and with trailing elements, for
team sizes on both sides of every plan rule.  Each result equals the per-call
reduction of the same arguments bit for bit (which other tests hold against
the oracle)."""
import numpy as np
import pytest

import gen

pytestmark = pytest.mark.gpu

NP_T = {"int32": np.int32, "uint64": np.uint64, "float32": np.float32, "float64": np.float64}


@pytest.mark.parametrize("dtype", sorted(NP_T))
@pytest.mark.parametrize("op", ["sum", "max"])
@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 33, 100, 256])
def test_tile_edges(B, heap, dtype, op, P):
    V = 16 // np.dtype(NP_T[dtype]).itemsize
    packs = (1, 127, 128, 129, 255, 257, 1023, 1025) if P <= 33 else (1, 127, 129)
    counts = sorted({1, V - 1 or 1, V, V + 1} | {V * p + t for p in packs for t in (0, 1, V - 1)})
    items, inputs = [], []
    for k, n in enumerate(counts):
        x = gen.random_values(NP_T[dtype], P, n, 7000 + k)
        if op == "max" and dtype.startswith("float"):
            x.reshape(-1)[::11] = np.nan   # deferred elements, whole tiles of them
            x.reshape(-1)[3::5] = -0.0
            x.reshape(-1)[4::5] = 0.0
        src, dst = heap(x[0].nbytes), heap(x[0].nbytes + 64)
        B.put_rows(src, x, team=(0, 1, P))
        algo = ["rec_dbl", "binomial", "linear", "rabenseifner"][k % 4]
        items.append(dict(op=op, dtype=dtype, algo=algo, team=(0, 1, P), dest=dst, src=src, nelems=n))
        inputs.append(x)

    def read():
        return [B.get_rows(it["dest"], x[0].nbytes + 64, np.uint8, team=it["team"])
                for it, x in zip(items, inputs)]

    def clear():
        for it, x in zip(items, inputs):
            B.memset(it["dest"], 0x5A, x[0].nbytes + 64, team=it["team"])

    clear()
    for it in items:
        B.reduce(it["op"], it["dtype"], it["algo"], it["dest"], it["src"], it["nelems"], team=it["team"])
    want = read()
    clear()
    b = B.Batch(B.make_descs(items), B.BATCH_NO_TUNE)
    b.run()
    b.close()
    for it, g, w in zip(items, read(), want):  # the 64 bytes past the dest are untouched
        assert (g == w).all(), it
