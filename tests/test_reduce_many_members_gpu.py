"""Reductions over the caller's own buffer with very many members of one
element each: every member counts towards the result and gets it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [(1 << 27) - 1, 1 << 27, (1 << 27) + 5])
def test_one_byte_of_each_member_in_place(B, members):
    import torch
    pad = 256
    x = torch.zeros(members + 2 * pad, dtype=torch.uint8, device="cuda")
    # one bit each from the first and last member, the middle, and where the
    # last of 16 lanes begins
    for bit, m in enumerate([0, members // 2, members * 15 // 16, members - 1]):
        x[pad + m] |= 1 << bit
    torch.cuda.synchronize()
    at = x.data_ptr() + pad
    B.reduce_noalloc("xor", "uint8", "rec_dbl", members, at, 1, at, 1, 1)
    row = x[pad:pad + members]
    assert bool((row == 15).all())
    assert not bool(x[:pad].any()) and not bool(x[pad + members:].any())
