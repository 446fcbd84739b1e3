"""GPU tests of the RWKV-4 time scan with values that are not finite: a decay out of range (exp(w) infinite) forgets at once, and
what is not a number stays between two start flags, forward and backward."""
import numpy as np
import pytest
import torch

import oracle
from jaxrwkv_b200 import rwkv4
from conftest import rel_err
from gpu_util import TOL, flags, npf
from test_gpu_wkv4 import NAMES, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [5, 16, 40, 300])
def test_infinite_decay(T, dtype):
    d = oracle.make_wkv4_inputs(2, T, 33, seed=T, default_state=False)
    d["w"] = np.array(d["w"])
    d["w"][::2] = 100.0                                # exp(100) is no fp32 number
    d["length"][:] = (T, max(1, T // 2))
    t = dev(d, dtype)
    length, ns = flags(d)
    s, y = rwkv4.CudaRWKV.inner_loop(*[t[n] for n in NAMES], length.cuda(), ns.cuda())
    # the oracle in 64 bits, where exp(100) only makes e^(pp + w') vanish as well
    so, yo = oracle.wkv4_base_batched(*[t[n].double().cpu().numpy() for n in NAMES], d["length"], d["new_starts"])
    assert rel_err(npf(y), yo) < TOL[dtype] and rel_err(npf(s), so) < TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bad", ["k", "v", "gy"])
@pytest.mark.parametrize("lo,at,hi", [(40, 100, 128), (35, 41, 46), (130, 140, 700)])   # over segments and CTAs, inside one segment, cluster steps
def test_not_a_number_stays_between_two_flags(lo, at, hi, bad, dtype):
    T, C = 800, 40
    d = oracle.make_wkv4_inputs(1, T, C, seed=3, default_state=False)
    ns = np.zeros((1, T), dtype=bool)
    ns[0, [lo, hi]] = True
    d["new_starts"] = ns
    d["length"][:] = T
    t = dev(d, dtype)
    g = torch.Generator(device="cuda").manual_seed(2)
    gy, gs = (torch.randn(s, generator=g, device="cuda").to(dtype) for s in ((1, T, C), (1, 3, C)))
    length, starts = (x.cuda() for x in flags(d))

    def run(value):
        x = {n: v.clone() for n, v in t.items()}
        cot = gy.clone()
        (cot if bad == "gy" else x[bad])[0, at, 3] += value
        leaves = [x[n].requires_grad_(True) for n in NAMES]
        s, y = rwkv4.CudaRWKV.inner_loop(*leaves, length, starts)
        grads = torch.autograd.grad((y, s), leaves, (cot, gs))
        return [y, grads[0], grads[1], grads[2]], [s, grads[5]]

    clean, nan = run(0.0), run(float("nan"))
    for a, b in zip(clean[0], nan[0]):
        assert torch.equal(a[:, :lo], b[:, :lo]) and torch.equal(a[:, hi:], b[:, hi:])
    for a, b in zip(clean[1], nan[1]):
        assert torch.equal(a, b)
    assert torch.isnan(nan[0][2 if bad == "gy" else 0][:, lo:hi]).any()
