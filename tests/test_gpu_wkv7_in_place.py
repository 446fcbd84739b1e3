"""GPU test of the RWKV-7 backward in fp32 with gradients written over operands and cotangents (each address one buffer)."""
import pytest
import torch

from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import NAMES7, flags, npf, to_dev, wkv7_case

pytestmark = pytest.mark.gpu
RESULTS = ("gr", "gw", "gk", "gv", "ga", "gb", "gs")


# gradients over their own operands, over each other's and over the cotangents; few heads in 16-token chunks, and short sequences
@pytest.mark.parametrize("over", [{"gr": "r", "gw": "w", "gk": "k", "gv": "v", "ga": "a", "gb": "b"}, {"gv": "dy"}, {"gw": "r", "gr": "w"}, {"gs": "ds"},
                                  {"gs": "ds", "gk": "dy", "ga": "k"}])
@pytest.mark.parametrize("B,T,H", [(2, 300, 12), (2, 40, 3)])
def test_gradients_over_operands(B, T, H, over):
    d = wkv7_case(B, T, H, seed=T, p_start=0.01, random_length=True, s0_scale=0.3)
    t = to_dev(d, torch.float32)
    length, ns = (x.cuda() for x in flags(d))
    g = torch.Generator(device="cuda").manual_seed(1)
    dy, ds = (torch.randn(t[n].shape, generator=g, device="cuda") for n in ("k", "s0"))
    _, res = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, B)
    keep = [x.clone() for x in res]
    want = rwkv7.batched_wkv7_bwd(tuple(keep), (ds.clone(), dy.clone()), B)
    at = dict(zip(NAMES7, res[:7]), dy=dy, ds=ds)
    got = rwkv7.batched_wkv7_bwd(res, (ds, dy), B, buffers={n: at[x] for n, x in over.items()})
    for n, a, b in zip(RESULTS, got, want):
        assert rel_err(npf(a), npf(b)) < 1e-5, n          # two orders of summation, as in test_gpu_wkv7_fp32.py
