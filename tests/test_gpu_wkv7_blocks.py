"""GPU tests of the block-parallel RWKV-7 forward (few sequences, longer than rings take): the blocks of all sequences over the
CTAs, the chain over the blocks and its cuts behind flagged blocks, `length` inside and between blocks, ragged last blocks; and the
same inputs at the shorter sizes that rings take."""
import numpy as np
import pytest
import torch

import oracle
from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import BLOCKS, NAMES7, TOL, flags, forward_form, npf, rounded, to_dev, wkv7_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("T,H,p_start", [(193, 1, 0.0), (256, 2, 0.0), (700, 1, 0.01), (1100, 5, 1 / 128)])
def test_forward_and_backward(T, H, p_start, train):
    assert forward_form(4, T, H, train) > BLOCKS                    # a ring
    check(T, H, p_start, train)


# a chain in one piece and in eight; several heads; more sequences than rings of four take
@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("T,H,p_start", [(1601, 1, 0.0), (1664, 2, 0.02), (2111, 1, 1 / 128), (1700, 2, 1 / 256), (520, 17, 1 / 128)])
def test_forward_and_backward_side_by_side(T, H, p_start, train):
    assert forward_form(4, T, H, train) == BLOCKS
    check(T, H, p_start, train)


def check(T, H, p_start, train):
    B = 4
    d = wkv7_case(B, T, H, seed=T, p_start=p_start, s0_scale=0.5)
    d["length"][:] = [T, 0, 128, T - 37]
    d["new_starts"][0, 0] = False              # a sequence that continues from its state, and one with flags on block edges
    d["new_starts"][3, [64, 127, 128]] = True
    t = to_dev(d, torch.bfloat16)
    length, ns = flags(d)
    leaves = [t[n].detach().requires_grad_(train) for n in NAMES7]
    s, y = rwkv7.CudaRWKV.inner_loop(*leaves, length.cuda(), ns.cuda())
    ins, tol = rounded(t), TOL[torch.bfloat16]
    so, yo = oracle.wkv7_base_batched(*ins, d["length"], d["new_starts"])
    assert rel_err(npf(y), yo) < tol
    for i in range(B):
        assert rel_err(npf(s[i]), so[i]) < tol, i
    if not train:
        return
    g = torch.Generator().manual_seed(T)
    gy, gs = torch.randn(y.shape, generator=g).bfloat16().cuda(), torch.randn(s.shape, generator=g).bfloat16().cuda()
    got = dict(zip(NAMES7, torch.autograd.grad([s, y], leaves, [gs, gy])))
    ref = oracle.wkv7_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy), npf(gs))
    for n, b in zip(("r", "w", "k", "v", "a", "b", "s0"), ref):
        assert rel_err(npf(got[n]), b) < tol, n


@pytest.mark.parametrize("T,blocks", [(320, False), (1700, True)])
def test_decay_outside_the_range_is_redone(T, blocks):
    assert (forward_form(2, T, 1, False) == BLOCKS) == blocks
    d = wkv7_case(2, T, 1, seed=3)
    d["w"][1, 70:90] = 3.0                     # exp(-20) per token
    t = to_dev(d, torch.bfloat16)
    length, ns = flags(d)
    s, y = rwkv7.CudaRWKV.inner_loop(*[t[n] for n in NAMES7], length.cuda(), ns.cuda())
    so, yo = oracle.wkv7_base_batched(*rounded(t), d["length"], d["new_starts"])
    assert np.isfinite(npf(y)).all() and rel_err(npf(y), yo) < TOL[torch.bfloat16] and rel_err(npf(s), so) < TOL[torch.bfloat16]
