"""GPU test of the number of kernel launches that bench.py states for a step."""
import pytest
import torch

import bench

pytestmark = pytest.mark.gpu


def test_launches_per_step():
    hd = bench.Headline(torch, 2, torch.device("cuda", 0), 1, Tn=256, Hn=2)
    hd.step()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        hd.step()
        torch.cuda.synchronize()
    on_device = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    assert sum("b200wkv" in n for n in on_device) == bench.LAUNCHES_PER_STEP, on_device
    assert not [n for n in on_device if "memset" in n.lower() or "memcpy" in n.lower()], on_device
