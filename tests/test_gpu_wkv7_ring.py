"""GPU tests of the RWKV-7 forward by rings of CTAs (few sequences): rings of three to sixteen, fewer blocks than CTAs, several turns
around the ring, `length` and start flags inside and on the edges of blocks; and long sequences of few heads, which keep the
block-parallel form."""
import pytest
import torch

import oracle
from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import BLOCKS, NAMES7, TOL, flags, forward_form, npf, rounded, to_dev, wkv7_case

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
    assert forward_form(B, T, H, train) > BLOCKS or T > 1536 or T == 129 and train
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


# rings in the place of the walk: of more than half a sequence per SM, of three blocks, of many
@pytest.mark.parametrize("B,T,H,train", [(5, 1000, 16, False), (5, 1000, 16, True), (10, 192, 4, False), (1, 5400, 32, False)])
def test_outputs_are_as_close_as_the_walks(B, T, H, train):
    """Both forms round operands to bf16 where they enter a product.  Rounding R~ + P_rb W~ as a sum too, where the walk has R~ alone,
    made the outputs' errors 0.15 % larger; sums in another order change them by 0.02 %."""
    assert forward_form(B, T, H, train) > BLOCKS
    d = wkv7_case(B, T, H, seed=T, s0_scale=0.3)
    t = to_dev(d, torch.bfloat16)
    length, ns = (x.cuda() for x in flags(d))
    exact = rwkv7.CudaRWKV.inner_loop(*[t[n].float() for n in NAMES7], length, ns)[1].double()    # (in fp32: 1e-7)
    walk = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, B, need_residual=train)[0][1]
    ring = rwkv7.CudaRWKV.inner_loop(*[t[n].requires_grad_(train) for n in NAMES7], length, ns)[1]
    errors = [((y.double() - exact).norm() / exact.norm()).item() for y in (walk, ring)]
    print(f"B={B} T={T} H={H} train={train}: walk {errors[0]:.5e}, ring {errors[1]:.5e}, ratio {errors[1] / errors[0]:.5f}")
    assert errors[1] <= 1.0005 * errors[0]
