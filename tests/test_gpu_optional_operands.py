"""GPU tests of training calls in which an optional operand is absent: the first layer (no value mix) and RWKV-4 without the
receptance.  The native node against the Python composition behind it."""
import numpy as np
import pytest
import torch

from jaxrwkv_b200 import _lib, rwkv4, time_mixing as tm
from conftest import rel_err
from test_oracle import unflatten_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 2e-2)])
def test_first_layer_gradients(golden, monkeypatch, dtype, tol):
    g = golden("v7_time_mixing")
    leaf = lambda a: torch.as_tensor(np.asarray(a), dtype=dtype, device="cuda").requires_grad_(True)
    att = {k: ({kk: leaf(vv) for kk, vv in v.items()} if isinstance(v, dict) else leaf(v)) for k, v in unflatten_params(g).items()}
    x, state, v_first = (leaf(g["in_" + n]) for n in ("x", "state", "v_first"))
    length, ns = torch.as_tensor(g["in_length"].astype(np.int32)).cuda(), torch.as_tensor(g["in_new_starts"]).cuda()
    flat = [t for k in sorted(att) for t in (att[k].values() if isinstance(att[k], dict) else [att[k]])]

    def run():
        outs = tm.time_mixing_seq(x, state, v_first, att, length, ns, int(g["H"]), int(g["S"]), 0)
        gen = torch.Generator(device="cuda").manual_seed(4)
        cots = [torch.randn(o.shape, generator=gen, device="cuda").to(dtype) for o in outs]
        return list(outs), torch.autograd.grad(outs, [x, state, v_first] + flat, cots, allow_unused=True)

    native = run()

    class Host:                                   # the native path declines: the composition of the single operators
        def time_mixing(self, *args):
            return None

        def __getattr__(self, name):
            return getattr(_lib._host, name)

    monkeypatch.setattr(_lib, "host", lambda: Host())
    plain = run()
    for a, b in zip(native[0], plain[0]):
        assert rel_err(a.detach().float().cpu().numpy(), b.detach().float().cpu().numpy()) < tol
    for i, (a, b) in enumerate(zip(native[1], plain[1])):
        assert (a is None) == (b is None), i
        if a is not None:
            assert a.shape == b.shape and rel_err(a.float().cpu().numpy(), b.float().cpu().numpy()) < tol, i


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rwkv4_without_receptance(dtype):
    B, T, C = 2, 50, 40
    gen = torch.Generator(device="cuda").manual_seed(1)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    leaves = [t.to(dtype).requires_grad_(True) for t in (rn(B, T, C), rn(B, T, C), 0.3 * rn(C), rn(C), rn(B, 3, C).abs())]
    length, ns = torch.tensor([T, 20], device="cuda"), rn(B, T) > 2
    native = rwkv4.wkv4_cuda(*leaves, length, ns)
    plain = rwkv4._WKV4.apply(*leaves, length, ns)[:2]
    cots = [torch.randn_like(o) for o in native]
    for a, b in zip(list(native) + list(torch.autograd.grad(native, leaves, cots)),
                    list(plain) + list(torch.autograd.grad(plain, leaves, cots))):
        assert a.shape == b.shape and rel_err(a.detach().float().cpu().numpy(), b.detach().float().cpu().numpy()) < (1e-6 if dtype == torch.float32 else 4e-3)
