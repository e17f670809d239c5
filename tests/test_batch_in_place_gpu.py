"""A batch with an in-place reduction runs it once, in batch_run: creating
the batch (default flags, so plans may be tuned by running them) leaves the
vectors as they are, whether the batch kernels cover the reduction's type or
it runs as a launch of its own."""
import numpy as np
import pytest

import gen

pytestmark = pytest.mark.gpu

NP_T = {"float32": np.float32, "int16": np.int16, "uint8": np.uint8, "complex64": np.complex64,
        "complex128": np.complex128}


@pytest.mark.parametrize("in_place", [["int16"], ["uint8", "complex64"], ["complex128"], ["float32"]])
def test_in_place_reductions_run_once(B, heap, in_place):
    P, n = 8, 4099
    team, items, inputs, want = (0, 1, P), [], [], []
    for k, dt in enumerate(["float32"] + in_place):
        x = gen.random_values(NP_T[dt], P, n, 300 + k)
        src, ref = heap(x[0].nbytes), heap(x[0].nbytes)
        dst = heap(x[0].nbytes) if k == 0 else src
        B.put_rows(src, x, team=team)
        B.reduce("sum", dt, "rec_dbl", ref, src, n, team=team)
        want.append(B.get_rows(ref, x[0].nbytes, x.dtype, team=team))
        items.append(dict(op="sum", dtype=dt, algo="rec_dbl", team=team, dest=dst, src=src, nelems=n))
        inputs.append(x)
    b = B.Batch(B.make_descs(items))
    try:
        for it, x in zip(items, inputs):
            assert (B.get_rows(it["src"], x[0].nbytes, np.uint8, team=team) ==
                    x.view(np.uint8).reshape(P, -1)).all(), it["dtype"]
        b.run()
    finally:
        b.close()
    for it, x, w in zip(items, inputs, want):
        got = B.get_rows(it["dest"], x[0].nbytes, x.dtype, team=team)
        assert got.tobytes() == w.tobytes(), it["dtype"]
