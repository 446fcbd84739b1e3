"""GPU test of the fp32 RWKV-7 residual: room for state gradients between chunks only where the backward has use for it."""
import pytest
import torch

import oracle
from jaxrwkv_b200 import _lib, rwkv7
from conftest import rel_err
from gpu_util import NAMES7, TOL, flags, npf, rounded, to_dev, wkv7_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [16, 40])
def test_sequences_that_fill_their_waves_get_no_room_between_chunks(T):
    lib = _lib.load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chunks, state = (T + 15) // 16, 64 * 64 * 4
    B = 12 * sms                              # whole waves for 1, 2, 3, 4, 6 or 12 thread blocks per SM
    assert lib.b200wkv7_residual_bytes(_lib.F32, B, T, 1, 64) == B * chunks * state
    assert lib.b200wkv7_residual_bytes(_lib.F32, 2, T, 1, 64) == 2 * 2 * chunks * state
    d = wkv7_case(B, T, 1, seed=T, p_start=0.05, random_length=True, s0_scale=0.3)
    t = to_dev(d, torch.float32)
    length, ns = flags(d)
    gy, gs = torch.randn_like(t["k"]), torch.randn_like(t["s0"])
    (_, _), res = rwkv7.batched_wkv7_fwd(*[t[n] for n in NAMES7], length, ns, B)
    got = rwkv7.batched_wkv7_bwd(res, (gs, gy), B)
    some = slice(B - 3, B)                    # the oracle on the last three
    ref = oracle.wkv7_bwd_batched(*[x[some] for x in rounded(t)], d["length"][some], d["new_starts"][some], npf(gy)[some], npf(gs)[some])
    for n, a, b in zip(("dr", "dw", "dk", "dv", "da", "db", "ds0"), got, ref):
        assert rel_err(npf(a)[some], b) < TOL[torch.float32], n
