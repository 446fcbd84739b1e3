"""GPU tests of the chunked RWKV-6 kernels at the edges of their 16-token tiles: sequences shorter than a tile or ending
inside one (the tile's other rows belong to no sequence), one part of a tile behind `length`, and a missing cotangent."""
import numpy as np
import pytest
import torch

import oracle
from jaxrwkv_b200 import _wkv6_family as fam
from conftest import rel_err
from gpu_util import TOL, flags, npf
from test_gpu_wkv6 import NAMES, case, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 15, 17, 31, 527])
@pytest.mark.parametrize("with_gy,with_gs", [(True, True), (False, True), (True, False)])
def test_tile_edges(T, with_gy, with_gs):
    B, H = 3, 2
    d = case("6", B, T, H, seed=T, starts=[[T // 2], [], [T - 1]], lengths=[T, max(T - 2, 0), (T + 1) // 2], s0_scale=0.5)
    t = dev(d, torch.bfloat16)
    length, ns = flags(d)
    w, u = t["w"].reshape(t["r"].shape), fam._expand_hn(t["u"], H, 64, torch.bfloat16)
    (s, y), res = fam.batched_wkv6_fwd("6", t["r"], t["k"], t["v"], w, u, t["s0"], length.cuda(), ns.cuda(), B)
    g = torch.Generator().manual_seed(T)
    gy = torch.randn(y.shape, generator=g).bfloat16().cuda() if with_gy else None
    gs = torch.randn(s.shape, generator=g).bfloat16().cuda() if with_gs else None
    got = fam.batched_wkv6_bwd("6", res, (gs, gy), B)
    ins = [t[n].double().cpu().numpy() for n in NAMES]
    so, yo = oracle.wkv6_base_batched(*ins, d["length"], d["new_starts"], "6")
    ref = oracle.wkv6_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy) if with_gy else np.zeros(y.shape),
                                  npf(gs) if with_gs else np.zeros(s.shape), "6")
    assert rel_err(npf(y), yo) < TOL[torch.bfloat16] and rel_err(npf(s), so) < TOL[torch.bfloat16]
    for n, a, b in zip(("dr", "dk", "dv", "dw", "du", "ds0"), got, ref):
        a = npf(a)
        a = a.sum(0) if a.size == B * b.size else a
        if np.abs(b).max() < 1e-30:            # (a state that has decayed to nothing)
            assert np.abs(a).max() < 1e-30, n
        else:
            assert rel_err(a.reshape(b.shape), b) < TOL[torch.bfloat16], n
