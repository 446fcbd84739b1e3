"""Decoding: the step kernel deals the (sequence, head) pairs out in equal shares over a grid of a fixed number of thread blocks
per SM, so no more of them may fit an SM, or a launch behind another one is spread unevenly over the SMs."""
import ctypes

import pytest

from jaxrwkv_b200 import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [_lib.F32, _lib.BF16])
def test_an_sm_takes_exactly_the_grids_share_of_thread_blocks(dtype):
    lib = _lib.load()
    grid, fit = ctypes.c_int(), ctypes.c_int()
    assert lib.b200wkv_debug_step_residency(dtype, ctypes.byref(grid), ctypes.byref(fit)) == 0
    assert fit.value == grid.value > 0
