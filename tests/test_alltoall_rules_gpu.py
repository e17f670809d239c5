"""All-to-alls on both sides of the lines between words one a thread and
aligned vectors, for blocks and offsets of every common width, with rows that
begin and end inside a vector; byte for byte, nothing beside the dest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 64
# common width -> block sizes around the lines (blocks of 4, 9 and 128 words;
# steps of 70000, 120000, 130000 and 200000 words at these team sizes)
SIZES = {16: (16, 48, 64, 272, 496, 528, 2048), 8: (24, 456, 1016, 1032, 1400, 2056),
         4: (20, 36, 52, 116, 140, 1004), 2: (18, 30, 46, 94), 1: (17, 25, 45, 101)}


@pytest.mark.parametrize("width", sorted(SIZES))
@pytest.mark.parametrize("P", [5, 33, 64, 100])
def test_both_sides_of_the_lines(B, heap, P, width):
    team, most = (0, 1, P), P * max(SIZES[width])
    x = np.random.default_rng(P + width).integers(0, 256, (P, most), dtype=np.uint8)
    src, dst = heap(most + 2 * GUARD), heap(most + 2 * GUARD)
    for nb in SIZES[width]:
        want = x[:, :P * nb].reshape(P, P, nb).transpose(1, 0, 2).reshape(P, P * nb)
        for a, b in ((0, 0), (width, width), (0, width), (width, 16 - width)):
            if width == 16 and (a, b) != (0, 0):
                continue
            B.put_rows(src + GUARD + a, np.ascontiguousarray(x[:, :P * nb]), team=team)
            B.memset(dst, 0xA5, P * nb + 2 * GUARD, team=team)
            B.alltoall(dst + GUARD + b, src + GUARD + a, nb, team=team)
            got = B.get_rows(dst, P * nb + 2 * GUARD, np.uint8, team=team)
            at = GUARD + b
            assert (got[:, at:at + P * nb] == want).all(), (nb, a, b)
            assert (got[:, :at] == 0xA5).all() and (got[:, at + P * nb:] == 0xA5).all(), (nb, a, b)
