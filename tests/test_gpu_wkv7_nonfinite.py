"""GPU tests of the bf16 RWKV-7 kernels with values that are no numbers: a start flag holds them back as it does in the
token-by-token recurrence, whichever form the forward takes, and in the gradients of what lies outside."""
import pytest
import torch

from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import BLOCKS, NAMES7, TOL, flags, forward_form, npf, to_dev, wkv7_case

pytestmark = pytest.mark.gpu
BAD = ("w", "k", "v", "a", "b", "s0")
FORMS = ["walk", "ring", "side by side"]
LONG = 1700                                       # blocks side by side are taken where a ring is not, above 24 blocks


def takes(form, T, H, train):
    return forward_form(1, T, H, train) == BLOCKS if form == "side by side" else forward_form(1, T, H, train) > BLOCKS


def operands(T, H, starts, bad, at, value):
    d = wkv7_case(1, T, H, seed=T + H, s0_scale=0.3, starts=[starts])
    clean = to_dev(d, torch.bfloat16)
    odd = {n: x.clone() for n, x in clean.items()}
    if bad == "s0":
        odd["s0"][0, -1, 3, 5] = value
    else:
        odd[bad][0, at, -1, 5] = value
    return clean, odd, [x.cuda() for x in flags(d)]


def outside_equals(clean, odd, lo, hi):
    """Everything outside the tokens [lo, hi) of the last head, where the value lies."""
    for a, b in zip(clean, odd):
        if a.dim() == 4 and a.shape[1] > hi and a.shape[1] != a.shape[2]:     # a stream
            a, b = (torch.cat([x[:, :lo], x[:, hi:]], 1) for x in (a, b))
        assert torch.isfinite(b.float()).all() and rel_err(npf(b), npf(a)) < TOL[torch.bfloat16]


# the value lies in front of a flag of its own 64-token block; a block and more in front of one; behind another one
@pytest.mark.parametrize("lo,at,hi", [(0, 66, 70), (0, 10, 140), (70, 100, 200), (128, 128, 192)])
@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("form", FORMS)
def test_forward(form, bad, lo, at, hi):
    T, H, value = LONG if form == "side by side" else 600, 3, float("inf") if bad in ("k", "v") else float("nan")
    assert takes(form, T, H, False)
    if bad == "s0":
        lo = 0
    clean, odd, (length, ns) = operands(T, H, sorted({lo, hi} - {0}), bad, at, value)

    def run(t):
        if form == "walk":                        # the C ABI brings no workspace
            (s, y), _ = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, 1, need_residual=False)
        else:
            s, y = rwkv7.CudaRWKV.inner_loop(*[t[n] for n in NAMES7], length, ns)
        return y, s
    outside_equals(run(clean), run(odd), lo, hi)


@pytest.mark.parametrize("lo,at,hi", [(70, 100, 200), (128, 150, 192), (64, 190, 256)])
@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("form", FORMS)
def test_gradients_of_what_lies_outside(form, bad, lo, at, hi):
    T, H = LONG if form == "side by side" else 400, 2
    assert takes(form, T, H, True)
    if bad == "s0":
        lo = 0
    clean, odd, (length, ns) = operands(T, H, sorted({lo, hi} - {0}), bad, at, float("nan"))
    g = torch.Generator(device="cuda").manual_seed(1)
    gy, gs = (torch.randn(clean[n].shape, generator=g, device="cuda").to(torch.bfloat16) for n in ("k", "s0"))
    gy[:, lo:hi] = 0                              # what lies inside has no part in the loss

    def run(t):
        if form == "walk":
            _, res = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, 1)
            grads = rwkv7.batched_wkv7_bwd(res, (gs, gy), 1)
        else:
            leaves = [t[n].clone().requires_grad_(True) for n in NAMES7]
            s, y = rwkv7.CudaRWKV.inner_loop(*leaves, length, ns)
            grads = torch.autograd.grad((y, s), leaves, (gy, gs))
        return grads[:6] + ((grads[6],) if lo > 0 else ())
    outside_equals(run(clean), run(odd), lo, hi)
