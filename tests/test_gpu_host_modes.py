"""GPU tests of what the native host path leaves to the Python functions behind it: forward-mode differentiation, which they
refuse, and tracing, which records them."""
import pytest
import torch
import torch.autograd.forward_ad as fw

from jaxrwkv_b200 import rwkv4, rwkv5_2, rwkv6, rwkv7
from gpu_util import NAMES7, flags, to_dev, wkv7_case
from test_gpu_wkv6 import NAMES as NAMES6, case as wkv6_case, dev as dev6

pytestmark = pytest.mark.gpu


def calls():
    d = wkv7_case(2, 40, 1, seed=5, p_start=0.05, s0_scale=0.3)
    length, ns = (x.cuda() for x in flags(d))
    t = to_dev(d, torch.float32)
    yield rwkv7.CudaRWKV.inner_loop, [t[n] for n in NAMES7], length, ns
    for version, mod in (("6", rwkv6), ("5_2", rwkv5_2)):
        t = dev6(wkv6_case(version, 2, 40, 1, seed=3), torch.float32)
        yield mod.CudaRWKV.inner_loop, [t[n] for n in NAMES6], length, ns
    rn = lambda *s: torch.randn(*s, device="cuda")
    yield rwkv4.CudaRWKV.inner_loop, [rn(2, 40, 32), rn(2, 40, 32), rn(2, 40, 32), rn(32), rn(32), rn(2, 3, 32).abs()], length, ns


@pytest.mark.parametrize("which", range(4))
def test_forward_mode_is_refused(which):
    fn, args, length, ns = list(calls())[which]
    fn(*args, length, ns)
    for i in range(1, len(args)):                   # (the first is RWKV-4's receptance, an ordinary product)
        with fw.dual_level(), pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
            fn(*[fw.make_dual(x, torch.ones_like(x)) if i == j else x for j, x in enumerate(args)], length, ns)


def test_a_trace_takes_its_results_from_its_arguments():
    fn, args, length, ns = next(calls())
    traced = torch.jit.trace(lambda *a: fn(*a, length, ns), tuple(args), check_trace=False)
    other = [0.5 * x for x in args]
    for a, b in zip(traced(*other), fn(*other, length, ns)):
        assert torch.equal(a, b)
