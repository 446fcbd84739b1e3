"""GPU test of a forward over few sequences on a device that has no room for the block-parallel form's workspace."""
import pytest
import torch

from jaxrwkv_b200 import rwkv7
from gpu_util import NAMES7, flags, to_dev, wkv7_case

pytestmark = pytest.mark.gpu


def test_without_room_for_the_workspace_the_walk_is_taken():
    T, H = 4096, 4
    d = wkv7_case(1, T, H, seed=3, s0_scale=0.3)
    t = to_dev(d, torch.bfloat16)
    length, ns = (x.cuda() for x in flags(d))
    walk = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, 1, need_residual=False)[0]
    roomy = rwkv7.CudaRWKV.inner_loop(*[t[n] for n in NAMES7], length, ns)
    assert not torch.equal(roomy[1], walk[1])                   # (the two forms round differently)
    room = torch.empty(6 << 20, dtype=torch.uint8, device="cuda")   # (so that two pieces are there to give back)
    del roomy, room
    torch.cuda.synchronize()
    fill = []
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / torch.cuda.get_device_properties(0).total_memory)
        with pytest.raises(torch.OutOfMemoryError):             # what the allocator still has, in pieces of 3 MB
            while True:
                fill.append(torch.empty(3 << 20, dtype=torch.uint8, device="cuda"))
        del fill[-2:]                                           # the workspace takes some 13 MB, the results 2.2
        tight = rwkv7.CudaRWKV.inner_loop(*[t[n] for n in NAMES7], length, ns)
        assert all(torch.equal(a, b) for a, b in zip(tight, walk))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
