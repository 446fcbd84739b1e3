"""GPU tests of the fp32-arithmetic RWKV-7 kernels where their split changes: rows per lane by the number of heads, and
the runs the backward cuts a sequence into by the room its residual has."""
import numpy as np
import pytest
import torch

import oracle
from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import NAMES7, TOL, flags, npf, rounded, to_dev, wkv7_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H", [(1, 3), (4, 10), (4, 25)])         # one, two and four rows per lane
def test_rows_per_lane(B, H, dtype):
    T = 37                                                           # three chunks, the last one ragged
    d = wkv7_case(B, T, H, seed=B * H, p_start=0.05, random_length=True, s0_scale=0.3)
    d["length"][0] = T
    t = to_dev(d, dtype)
    length, ns = flags(d)
    g = torch.Generator().manual_seed(3)
    gy = torch.randn(t["k"].shape, generator=g).to(dtype).cuda()
    gs = torch.randn(t["s0"].shape, generator=g).to(dtype).cuda()
    (s, y), res = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, B, flags=1)
    got = rwkv7.batched_wkv7_bwd(res, (gs, gy), B, flags=1)
    ins = rounded(t)
    so, yo = oracle.wkv7_base_batched(*ins, d["length"], d["new_starts"])
    ref = oracle.wkv7_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy), npf(gs))
    tol = TOL[dtype]
    assert rel_err(npf(y), yo) < tol and rel_err(npf(s), so) < tol
    for n, a, b in zip(("dr", "dw", "dk", "dv", "da", "db", "ds0"), got, ref):
        assert rel_err(npf(a), b) < tol, n


@pytest.mark.parametrize("chunks_of_room", [0, 1, 2, 9])
def test_backward_runs_by_room(chunks_of_room):
    """The backward of a ten-chunk sequence with room for 0 (one run), 1, 2 and 9 state gradients behind the checkpoints."""
    from jaxrwkv_b200 import _lib
    B, T, H = 2, 150, 2
    d = wkv7_case(B, T, H, seed=6, p_start=0.02, random_length=True, s0_scale=0.3)
    t = to_dev(d, torch.float32)
    length, ns = flags(d)
    gy, gs = torch.randn_like(t["k"]), torch.randn_like(t["s0"])
    full = _lib.load().b200wkv7_residual_bytes(_lib.F32, B, T, H, 64)
    nbytes = full // 2 + chunks_of_room * B * H * 64 * 64 * 4
    (_, _), res = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, B)
    want = rwkv7.batched_wkv7_bwd(res, (gs, gy), B)
    got = rwkv7.batched_wkv7_bwd((*res[:-1], res[-1][:nbytes].clone()), (gs, gy), B)
    for a, b in zip(got, want):
        assert rel_err(npf(a), npf(b)) < 1e-5
