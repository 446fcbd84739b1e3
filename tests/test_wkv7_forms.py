"""CPU tests of which form the bf16 RWKV-7 forward takes (rings of CTAs, blocks side by side, the walk), by sizes and device."""
import pytest

from jaxrwkv_b200 import _lib

WALK, BLOCKS = 0, 1


def form(B, T, H, residual=False, sms=148, largest=16):
    return _lib.load().b200wkv_debug_wkv7_fwd_form(sms, largest, B, T, H, int(residual))


@pytest.mark.parametrize("residual", [False, True])
def test_a_ring_is_no_larger_than_the_device_takes(residual):
    assert form(1, 1536, 4, residual) == 16 and form(1, 1999, 32, residual) == 8
    for largest in range(3, 17):
        assert form(1, 1536, 4, residual, largest=largest) == largest
        assert form(1, 1024, 32, residual, largest=largest) in (min(8, largest), BLOCKS)
    for largest in (0, 1, 2):                                  # a context without clusters: the other forms, which need none
        assert form(1, 1536, 4, residual, largest=largest) == BLOCKS
        assert form(1, 192, 4, residual, largest=largest) == WALK
    for sms in range(1, 148):                                  # a share of the SMs: what is launched at once fits
        for heads in (1, 2, 5, 16, 40):
            n = form(1, 1024, heads, residual, sms=sms)
            assert n <= 1 or n * heads <= 2 * sms


# (one count of sequences, its neighbour with the same rings), every length: no count falls out of its group
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("one,other", [(65, 66), (66, 74), (75, 86), (52, 64), (44, 51), (38, 43), (10, 21)])
def test_neighbours_take_the_same_form(one, other, residual):
    for T in range(64, 5000, 64):
        a, b = form(1, T, one, residual), form(1, T, other, residual)
        assert a == b or (a in (WALK, BLOCKS) and b in (WALK, BLOCKS)), T      # (the form behind a ring has limits of its own)


# the longest sequences, in blocks of 64 tokens, that rings take by the count of sequences
@pytest.mark.parametrize("heads,ring,longest,with_residual", [(1, 16, 24, 24), (9, 16, 24, 24), (10, 9, 24, 24), (21, 9, 24, 24), (22, 9, None, None),
                                                              (37, 7, None, None), (38, 6, 48, 48), (48, 5, 40, 48), (64, 4, 32, 48), (65, 3, 7, 7),
                                                              (74, 3, 7, 7), (75, 3, 16, 23), (86, 3, 16, 23)])
def test_where_rings_end(heads, ring, longest, with_residual):
    for residual, most in ((False, longest), (True, with_residual)):
        assert form(1, 64 * (4 if most == 7 else 16), heads, residual) == min(ring, 16)
        if most is None:
            assert form(1, 64 * 200, heads, residual) == ring
        else:
            assert form(1, 64 * most, heads, residual) in (ring, most) and form(1, 64 * most + 1, heads, residual) in (WALK, BLOCKS)
    assert form(1, 128, heads) == WALK and form(1, 129, heads) == 3 and form(1, 192, heads, True) == WALK
    assert form(1, 1024, 87) == WALK and form(1, 1024, 87, True) == WALK
