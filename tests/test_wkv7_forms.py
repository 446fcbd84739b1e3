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
