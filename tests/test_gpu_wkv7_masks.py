"""GPU tests of the chunked RWKV-7 kernels where start flags and `length` fall inside 64-token blocks: the flags are
masks of the block's products, and a `length` inside a block cuts it in two, the second part in the sequence's last
slot of the residual."""
import pytest
import torch

from test_gpu_wkv7 import check_bwd, check_fwd
from gpu_util import wkv7_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [64, 67, 200])
@pytest.mark.parametrize("cut", [1, 15, 16, 17, 32, 63])
def test_flags_and_length_inside_blocks(T, cut):
    starts = [[cut], [0, cut - 1, cut], range(0, T, cut), [cut, T - 1], [T - cut], []]
    lengths = [T, cut, T - cut, T - 1, min(64 + cut, T), min(cut, T)]
    d = wkv7_case(len(starts), T, 2, seed=T + cut, s0_scale=0.5, starts=starts, lengths=lengths)
    check_fwd(d, torch.bfloat16)
    check_bwd(d, torch.bfloat16)
