"""GPU tests of operands that lie where the widest vector accesses do not fit: they take the kernels with narrower ones."""
import pytest
import torch

import oracle
from jaxrwkv_b200 import _lib, rwkv5_2
from conftest import rel_err
from gpu_util import TOL, flags, npf
from test_gpu_wkv6 import NAMES, case, dev

pytestmark = pytest.mark.gpu


def moved(x, elements):
    """The same values in a contiguous tensor that starts `elements` behind a 512-byte boundary."""
    room = torch.empty(x.numel() + elements, dtype=x.dtype, device=x.device)
    room[elements:].copy_(x.flatten())
    return room[elements:].view(x.shape)


@pytest.mark.parametrize("which", ["r", "v", "s0", "gy", "all"])
def test_rwkv5_2_training_on_8_byte_boundaries(which):
    d = case("5_2", 2, 100, 2, seed=11, p_start=0.02, random_length=True)
    t = dev(d, torch.bfloat16)
    t = {n: moved(x, 4) if which in (n, "all") else x for n, x in t.items()}
    leaves = [t[n].requires_grad_(True) for n in NAMES]
    length, ns = (x.cuda() for x in flags(d))
    s, y = rwkv5_2.CudaRWKV.inner_loop(*leaves, length, ns)
    gy, gs = torch.randn_like(y), torch.randn_like(s)
    if which in ("gy", "all"):
        gy = moved(gy, 4)
    grads = torch.autograd.grad((y, s), leaves, (gy, gs))
    ins = [npf(x) for x in leaves]
    so, yo = oracle.wkv6_base_batched(*ins, d["length"], d["new_starts"], "5_2")
    ref = oracle.wkv6_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy), npf(gs), "5_2")
    for a, b in zip((y, s) + grads, (yo, so) + tuple(ref)):
        assert rel_err(npf(a).reshape(b.shape), b) < TOL[torch.bfloat16]


def test_addresses_that_suit_no_access_are_an_error():
    d = case("5_2", 1, 20, 1, seed=1)
    t = dev(d, torch.bfloat16)
    length, ns = (x.cuda() for x in flags(d))
    t["k"] = moved(t["k"], 1)
    with pytest.raises(_lib.B200WKVError, match="address"):
        rwkv5_2.CudaRWKV.inner_loop(*[t[n].requires_grad_(True) for n in NAMES], length, ns)
