"""GPU tests of RWKV-5 / 5.2 calls without gradients: the bits of a training call, without its checkpoints."""
import numpy as np
import pytest
import torch

from jaxrwkv_b200 import _lib, rwkv5, rwkv5_2
from gpu_util import flags
from test_gpu_wkv6 import NAMES, case, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,mod", [("5_2", rwkv5_2), ("5", rwkv5)])
@pytest.mark.parametrize("T", [1, 16, 17, 64, 65, 260])
def test_results_are_those_of_a_training_call(version, mod, T):
    d = case(version, 3, T, 3, seed=T, p_start=0.02, random_length=True)
    d["length"][0] = T
    d["w"] = np.array(d["w"])
    d["w"][1] = 1.0078125                     # a head outside the run-parallel kernels' domain
    t = [x.requires_grad_(True) for x in dev(d, torch.bfloat16).values()]
    length, ns = (x.cuda() for x in flags(d))
    s, y = mod.CudaRWKV.inner_loop(*t, length, ns)
    assert y.requires_grad
    with torch.no_grad():
        s0, y0 = mod.CudaRWKV.inner_loop(*t, length, ns)
    assert torch.equal(y, y0) and torch.equal(s, s0)


def test_no_checkpoints_without_gradients():
    B, T, H = 2, 2048, 4
    t = [x for x in dev(case("5_2", B, T, H, seed=1), torch.bfloat16).values()]
    assert len(t) == len(NAMES)
    length, ns = torch.full((B,), T, dtype=torch.int32, device="cuda"), torch.zeros(B, T, dtype=torch.uint8, device="cuda")
    rwkv5_2.CudaRWKV.inner_loop(*t, length, ns)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    with torch.no_grad():
        out = rwkv5_2.CudaRWKV.inner_loop(*t, length, ns)
    stream = B * T * H * 64 * 2
    assert torch.cuda.max_memory_allocated() - before < 4 * stream + (1 << 20), out[1].shape   # the output, and a state per 64 tokens
    assert _lib.load().b200wkv6_residual_bytes(_lib.BF16, B, T, H, 64) > 8 * stream
