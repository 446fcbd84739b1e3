"""GPU tests of the RWKV-7 forward by rings of CTAs (few sequences): rings of three to sixteen, fewer blocks than CTAs, several turns
around the ring, `length` and start flags inside and on the edges of blocks; and long sequences of few heads, which keep the
block-parallel form."""
import pytest
import torch

import oracle
from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import NAMES7, TOL, flags, npf, rounded, to_dev, wkv7_case

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, scope="module")
def no_memory_left_behind():
    """What these sizes leave in the allocator's cache is given back: other tests fill the device's memory up to a byte count."""
    yield
    torch.cuda.empty_cache()


# ring of 3 (as many as blocks, then of more sequences), 16, 9, 8, 6, 4; the last two: the longest rings of few heads, blocks side by side
@pytest.mark.parametrize("B,T,H", [(4, 129, 1), (7, 450, 12), (6, 400, 11), (4, 1100, 1), (6, 650, 2), (8, 577, 4), (5, 449, 8), (8, 330, 8), (4, 1536, 1), (4, 1600, 1)])
@pytest.mark.parametrize("train", [False, True])
def test_forward_and_backward(B, T, H, train):
    d = wkv7_case(B, T, H, seed=T, p_start=0.0, s0_scale=0.5)
    d["length"][:] = ([T, 0, 128, T - 37] * 2)[:B]
    d["new_starts"][:] = False
    d["new_starts"][3, [63, 64, 127, 128]] = True
    d["new_starts"][0, [0, T - 1]] = [False, True]
    t = to_dev(d, torch.bfloat16)
    length, ns = flags(d)
    leaves = [t[n].detach().requires_grad_(train) for n in NAMES7]
    s, y = rwkv7.CudaRWKV.inner_loop(*leaves, length.cuda(), ns.cuda())
    ins, tol = rounded(t), TOL[torch.bfloat16]
    so, yo = oracle.wkv7_base_batched(*ins, d["length"], d["new_starts"])
    for i in range(B):
        assert rel_err(npf(y[i]), yo[i]) < tol, i
        assert rel_err(npf(s[i]), so[i]) < tol, i
    if not train:
        return
    g = torch.Generator().manual_seed(T)
    gy, gs = torch.randn(y.shape, generator=g).bfloat16().cuda(), torch.randn(s.shape, generator=g).bfloat16().cuda()
    got = dict(zip(NAMES7, torch.autograd.grad([s, y], leaves, [gs, gy])))
    ref = oracle.wkv7_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy), npf(gs))
    for n, b in zip(("r", "w", "k", "v", "a", "b", "s0"), ref):
        assert rel_err(npf(got[n]), b) < tol, n
