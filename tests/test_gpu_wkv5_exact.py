"""GPU tests of the run-parallel fp32-accurate RWKV-5 / 5.2 training kernels: run and chunk edges, and heads whose decay is
outside their domain beside heads that are inside."""
import numpy as np
import pytest
import torch

import oracle
from test_gpu_wkv6 import case, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [63, 64, 65, 129, 260])
def test_run_edges(T):
    starts = [[0, T - 1], [min(64, T - 1)], [16 % T, 15, 48, min(63, T - 1)], []]
    lengths = [T, min(64, T), min(65, T), T // 2]
    check("5_2", case("5_2", 4, T, 2, seed=T, starts=starts, lengths=lengths, s0_scale=0.5), torch.bfloat16)


def test_accuracy_is_that_of_fp32():
    """Against the fp64 oracle on the rounded inputs: what is left is the rounding of the bf16 results (2^-9 at most)."""
    d = case("5_2", 2, 200, 2, seed=4, p_start=0.01, s0_scale=0.5)
    from gpu_util import flags, npf
    from conftest import rel_err
    from jaxrwkv_b200 import rwkv5_2
    from test_gpu_wkv6 import NAMES, dev
    leaves = [x.requires_grad_(True) for x in dev(d, torch.bfloat16).values()]
    length, ns = (x.cuda() for x in flags(d))
    s, y = rwkv5_2.CudaRWKV.inner_loop(*leaves, length, ns)
    gy, gs = torch.randn_like(y), torch.randn_like(s)
    grads = torch.autograd.grad((y, s), leaves, (gy, gs))
    ins = [npf(x) for x in leaves]
    so, yo = oracle.wkv6_base_batched(*ins, d["length"], d["new_starts"], "5_2")
    ref = oracle.wkv6_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy), npf(gs), "5_2")
    for a, b in zip((y, s) + grads, (yo, so) + tuple(ref)):
        assert rel_err(npf(a).reshape(b.shape), b) < 2.5e-3, NAMES


@pytest.mark.parametrize("decay", [2.0 ** -14, 0.0, 1.0078125])
def test_heads_outside_the_domain(decay):
    d = case("5_2", 2, 100, 3, seed=9, p_start=0.02, random_length=True)
    d["w"] = np.array(d["w"])
    d["w"][1, 5] = decay
    check("5_2", d, torch.bfloat16)
