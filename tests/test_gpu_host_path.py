"""GPU tests of the native host path (csrc/host_ext.cpp): it gives what the Python autograd functions behind it
give, for every way flags and leading axes may be passed, and refuses a second differentiation the same way."""
import pytest
import torch

from jaxrwkv_b200 import _lib, rwkv5, rwkv5_2, rwkv6, rwkv7, _wkv6_family as fam
from gpu_util import flags, to_dev, wkv7_case
from test_gpu_wkv6 import NAMES as NAMES6, case as wkv6_case, dev as dev6

pytestmark = pytest.mark.gpu
NAMES = ("r", "w", "k", "v", "a", "b", "s0")


def _grads(outs, leaves):
    g = torch.Generator(device="cuda").manual_seed(1)
    cot = [torch.randn(o.shape, generator=g, device="cuda").to(o.dtype) for o in outs]
    return torch.autograd.grad(outs, leaves, cot)


@pytest.mark.parametrize("lead", [(), (3,), (2, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_wkv7_native_path_matches_python_path(lead, dtype):
    B = max(1, int(torch.tensor(lead).prod()))
    d = wkv7_case(B, 70, 2, seed=5, p_start=0.05, random_length=True, s0_scale=0.3)
    t = to_dev(d, dtype)
    leaves = [t[n].reshape(lead + t[n].shape[1:]).requires_grad_(True) for n in NAMES]
    length, ns = (x.cuda() for x in flags(d))
    for len_, ns_ in ((length.reshape(lead), ns.reshape(lead + (70,))),          # int64, bool
                      (length.int().reshape(lead), ns.byte().reshape(lead + (70,))),
                      (length.flatten()[0], ns[0].float()),                       # shared by all rows
                      (length.cpu().reshape(lead), ns.cpu().reshape(lead + (70,)))):
        native = _lib.host().wkv7(*leaves, len_, ns_)
        assert native is not None
        plain = rwkv7._WKV7.apply(*leaves, len_, ns_)[:2]
        assert all(torch.equal(x, y) for x, y in zip(native, plain))
        assert all(torch.equal(x, y) for x, y in zip(_grads(native, leaves), _grads(plain, leaves)))
    with torch.no_grad():
        s, y = rwkv7.CudaRWKV.inner_loop(*leaves, length.reshape(lead), ns.reshape(lead + (70,)))
    assert not y.requires_grad
    tol = 1e-5 if dtype == torch.float32 else 1e-2
    assert (y.float() - _lib.host().wkv7(*leaves, length.reshape(lead), ns.reshape(lead + (70,)))[1].float()).norm() <= tol * y.float().norm()


@pytest.mark.parametrize("version,mod", [("6", rwkv6), ("5_2", rwkv5_2), ("5", rwkv5)])
def test_wkv6_family_native_path_matches_python_path(version, mod):
    d = wkv6_case(version, 2, 40, 2, seed=3, p_start=0.05, random_length=True)
    leaves = [x.requires_grad_(True) for x in dev6(d, torch.bfloat16).values()]
    assert len(leaves) == len(NAMES6)
    length, ns = (x.cuda() for x in flags(d))
    native = mod.CudaRWKV.inner_loop(*leaves, length, ns)
    plain = fam._FUNCS[version][0].apply(*leaves, length, ns)[:2]
    assert all(torch.equal(x, y) for x, y in zip(native, plain))
    for x, y in zip(_grads(native, leaves), _grads(plain, leaves)):
        assert x.shape == y.shape and x.dtype == y.dtype and torch.equal(x, y)


def test_second_differentiation_is_refused():
    d = wkv7_case(1, 16, 1, seed=2)
    t = to_dev(d, torch.float32)
    leaves = [t[n].requires_grad_(True) for n in NAMES]
    length, ns = (x.cuda() for x in flags(d))
    s, y = rwkv7.wkv7_cuda(*leaves, length, ns)
    (g,) = torch.autograd.grad(y.sum(), leaves[:1], create_graph=True)
    with pytest.raises(_lib.B200WKVError, match="second-order"):
        torch.autograd.grad(g.sum(), leaves[1:2])


def test_only_one_result_used_and_arguments_that_do_not_fit():
    d = wkv7_case(2, 16, 1, seed=2)
    t = to_dev(d, torch.float32)
    leaves = [t[n].requires_grad_(True) for n in NAMES]
    length, ns = (x.cuda() for x in flags(d))
    for which in (0, 1):
        native = torch.autograd.grad(_lib.host().wkv7(*leaves, length, ns)[which].sum(), leaves)
        plain = torch.autograd.grad(rwkv7._WKV7.apply(*leaves, length, ns)[which].sum(), leaves)
        assert all(torch.equal(x, y) for x, y in zip(native, plain))
    assert _lib.host().wkv7(*leaves, 16, ns) is None
    s, y = rwkv7.wkv7_cuda(*leaves, 16, ns)          # a plain number is still taken
    assert torch.equal(y, _lib.host().wkv7(*leaves, length, ns)[1])
    with pytest.raises(_lib.B200WKVError, match="share one element type"):
        rwkv7.wkv7_cuda(leaves[0].bfloat16(), *leaves[1:], length, ns)
