"""GPU tests of the run-parallel RWKV-5 / 5.2 kernels with values that are no numbers: a start flag holds them back as it does in
the token-by-token recurrence, forward and in the gradients of what lies outside."""
import pytest
import torch

from jaxrwkv_b200 import rwkv5_2
from conftest import rel_err
from gpu_util import flags, npf
from test_gpu_wkv6 import NAMES, case, dev

pytestmark = pytest.mark.gpu


# inside one 16-token chunk; over chunks and runs; from flag to flag at chunk edges; at run edges
@pytest.mark.parametrize("lo,at,hi", [(18, 20, 27), (40, 41, 150), (32, 40, 48), (64, 127, 128)])
@pytest.mark.parametrize("bad", ["r", "k", "v", "s0", "gy"])
def test_a_flag_ends_it(bad, lo, at, hi):
    T, H = 300, 2
    if bad == "s0":
        lo = 0
    d = case("5_2", 1, T, H, seed=7, starts=[sorted({lo, hi} - {0})])
    t = dev(d, torch.bfloat16)
    length, ns = (x.cuda() for x in flags(d))
    g = torch.Generator(device="cuda").manual_seed(1)
    gy, gs = (torch.randn(t[n].shape, generator=g, device="cuda").to(torch.bfloat16) for n in ("k", "s0"))
    gy[:, lo:hi] = 0                              # what lies inside has no part in the loss

    def run(value):
        x, cot = {n: v.clone() for n, v in t.items()}, gy.clone()
        if bad == "s0":
            x["s0"][0, -1, 3, 5] += value
        else:
            (cot if bad == "gy" else x[bad])[0, at, -1, 5] += value
        with torch.no_grad():
            s1, y1 = rwkv5_2.CudaRWKV.inner_loop(*[x[n] for n in NAMES], length, ns)
        leaves = [x[n].requires_grad_(True) for n in NAMES]
        s, y = rwkv5_2.CudaRWKV.inner_loop(*leaves, length, ns)
        assert bad == "gy" or (torch.equal(s, s1) and torch.equal(y.nan_to_num(), y1.nan_to_num()))
        grads = torch.autograd.grad((y, s), leaves, (cot, gs))
        return [y, grads[0], grads[1], grads[2]], [s] + ([grads[5]] if lo > 0 else [])

    clean, odd = run(0.0), run(float("nan"))
    outside = lambda a: torch.cat([a[:, :lo], a[:, hi:]], 1)
    for a, b in [(outside(a), outside(b)) for a, b in zip(clean[0], odd[0])] + list(zip(clean[1], odd[1])):
        # both are fp32-accurate and rounded to bf16: the last bit may differ
        assert torch.isfinite(b.float()).all() and rel_err(npf(b), npf(a)) < 2.0 ** -9
