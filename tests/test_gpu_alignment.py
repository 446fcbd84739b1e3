"""GPU tests of operands that lie where the widest vector accesses do not fit: they take the kernels with narrower ones."""
import numpy as np
import pytest
import torch

import oracle
from jaxrwkv_b200 import _lib, rwkv5_2, rwkv7
from jaxrwkv_b200.time_mixing import time_mixing_seq
from conftest import rel_err
from gpu_util import NAMES7, TOL, flags, npf, to_dev, wkv7_case
from test_gpu_wkv6 import NAMES, case, dev
from test_oracle import unflatten_params

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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cotangents_that_are_slices(dtype):
    """Autograd hands in slices of a concatenation's gradient, which begin anywhere."""
    d = wkv7_case(2, 70, 2, seed=5, p_start=0.05, random_length=True, s0_scale=0.3)
    leaves = [to_dev(d, dtype)[n].requires_grad_(True) for n in NAMES7]
    length, ns = (x.cuda() for x in flags(d))
    s, y = rwkv7.CudaRWKV.inner_loop(*leaves, length, ns)
    gy, gs = torch.randn_like(y), torch.randn_like(s)
    want = torch.autograd.grad((y, s), leaves, (gy, gs), retain_graph=True)
    one = torch.zeros(1, dtype=dtype, device="cuda")
    got = torch.autograd.grad(torch.cat([one, y.flatten(), s.flatten()]), leaves, torch.cat([one, gy.flatten(), gs.flatten()]))
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("layer_id", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_time_mixing_layer_with_slices(golden, dtype, layer_id):
    g = golden("v7_time_mixing")
    leaf = lambda a: torch.as_tensor(np.asarray(a), dtype=dtype, device="cuda").requires_grad_(True)
    att = {k: ({kk: leaf(vv) for kk, vv in v.items()} if isinstance(v, dict) else leaf(v)) for k, v in unflatten_params(g).items()}
    length, ns = torch.as_tensor(g["in_length"].astype(np.int32)).cuda(), torch.as_tensor(g["in_new_starts"]).cuda()

    def run(off, B):
        x, v_first = leaf(g["in_x"][:B]), leaf(g["in_v_first"][:B])
        state = moved(leaf(g["in_state"][:B]).detach(), off).requires_grad_(True)
        out, new_state, v = time_mixing_seq(x, state, v_first, att, length[:B], ns[:B], int(g["H"]), int(g["S"]), layer_id)
        outs = [out, new_state] + ([v] if layer_id == 0 else [])
        gen = torch.Generator(device="cuda").manual_seed(4)
        cots = [moved(torch.randn(o.shape, generator=gen, device="cuda").to(dtype), off) for o in outs]
        return outs + list(torch.autograd.grad(outs, [x, state, att["key"]["weight"], att["x_r"]], cots))

    for B in (1, len(g["in_x"])):
        for off in (1, 4):
            assert all(torch.equal(a, b) for a, b in zip(run(off, B), run(0, B)))
    x = moved(leaf(g["in_x"]).detach(), 1)
    with pytest.raises(_lib.B200WKVError, match="address"):
        time_mixing_seq(x, leaf(g["in_state"]), leaf(g["in_v_first"]), att, length, ns, int(g["H"]), int(g["S"]), layer_id)
