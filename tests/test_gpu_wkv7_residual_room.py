"""GPU tests of what fp32 RWKV-7 training keeps in memory where sequences fill the device, and of calls without room for it."""
import pytest
import torch

from jaxrwkv_b200 import _lib, rwkv7
from conftest import rel_err
from gpu_util import NAMES7, flags, npf, to_dev, wkv7_case

pytestmark = pytest.mark.gpu
B, T = 1, 512
MB = 1 << 20


@pytest.fixture(scope="module")
def case():
    H = 128 * torch.cuda.get_device_properties(0).multi_processor_count // 148      # a wave of CTAs, one head per SM, nearly full
    d = wkv7_case(B, T, H, seed=2, p_start=0.004, random_length=True, s0_scale=0.3)
    t = to_dev(d, torch.float32)
    length, ns = (x.cuda() for x in flags(d))
    g = torch.Generator(device="cuda").manual_seed(3)
    yield H, t, length, ns, *(torch.randn(t[n].shape, generator=g, device="cuda") for n in ("k", "s0"))
    torch.cuda.empty_cache()


def forward(case):
    H, t, length, ns, _, _ = case
    leaves = [t[n].detach().requires_grad_(True) for n in NAMES7]
    return leaves, rwkv7.CudaRWKV.inner_loop(*leaves, length, ns)


def backward(case, leaves, out):
    return torch.autograd.grad([out[1], out[0]], leaves, [case[4], case[5]])


class Room:
    """The device as full as it is, but for pieces of `n` bytes; free parts of the allocator's segments are filled as well."""
    def __init__(self, n, pieces=1):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.limit()
        self.fill = []
        for size in (64 * MB, 16 * MB, 4 * MB, MB + 512):
            try:
                while True:
                    self.fill.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        torch.cuda.set_per_process_memory_fraction(1.0)
        self.blocks = [torch.empty(n, dtype=torch.uint8, device="cuda") for _ in range(pieces)]

    @staticmethod
    def limit():
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / torch.cuda.get_device_properties(0).total_memory)

    def __enter__(self):
        self.limit()
        del self.blocks

    def __exit__(self, *_):
        torch.cuda.set_per_process_memory_fraction(1.0)
        del self.fill


def test_what_is_kept_and_what_does_without(case):
    H, t, length, ns, dy, ds = case
    chunks, state = H * T // 16, 64 * 64 * 4
    before = torch.cuda.memory_allocated()
    leaves, out = forward(case)
    kept = torch.cuda.memory_allocated() - before - sum(x.numel() * 4 for x in out)
    assert kept <= chunks * (state + 16 * 64 * 4) + MB               # checkpoints and a row per token
    assert _lib.load().b200wkv7_residual_bytes(_lib.F32, B, T, H, 64) == chunks * state        # without a workspace: checkpoints alone
    want = backward(case, leaves, out)

    small = sum(x.numel() * 4 for x in out)
    with Room(small + chunks * state + 8 * MB):                      # a workspace or the checkpoints, but not both
        leaves, tight = forward(case)
    got = backward(case, leaves, tight)
    assert not torch.equal(tight[1], out[1])                         # (the kernels that need less round differently)
    for a, b in zip((*tight, *got), (*out, *want)):
        assert rel_err(npf(a), npf(b)) < 1e-5                        # two orders of summation, as in test_gpu_wkv7_fp32.py
    del tight, got

    leaves, out = forward(case)
    with Room(chunks * state // 2, 4):                               # the gradients (a quarter each), but no workspace
        got = backward(case, leaves, out)
    assert not torch.equal(got[0], want[0])
    for a, b in zip(got, want):
        assert rel_err(npf(a), npf(b)) < 1e-5


def test_a_roomier_residual_of_the_callers(case):
    """A buffer larger than asked for: the forward and the backward take it for the same."""
    H, t, length, ns, dy, ds = case
    ops = [t[n] for n in NAMES7]
    want = rwkv7.batched_wkv7_bwd(rwkv7.batched_wkv7_fwd(*ops, length, ns, B)[1], (ds, dy), B)
    for size in (24, 48):                                            # KB per 16 tokens and head
        room = torch.empty(size * 1024 * H * T // 16, dtype=torch.uint8, device="cuda")
        got = rwkv7.batched_wkv7_bwd(rwkv7.batched_wkv7_fwd(*ops, length, ns, B, buffers={"residual": room})[1], (ds, dy), B)
        for a, b in zip(got, want):
            assert rel_err(npf(a), npf(b)) < 1e-5


def test_the_batched_calls_without_room():
    H, T = 24, 1024
    d = wkv7_case(B, T, H, seed=4, s0_scale=0.3)
    t = to_dev(d, torch.float32)
    length, ns = (x.cuda().to(y) for x, y in zip(flags(d), (torch.int32, torch.uint8)))
    ops, dy, ds = [t[n] for n in NAMES7], torch.randn_like(t["k"]), torch.randn_like(t["s0"])
    full = rwkv7.batched_wkv7_fwd(*ops, length, ns, B)
    want = rwkv7.batched_wkv7_bwd(full[1], (ds, dy), B)
    least = _lib.load().b200wkv7_residual_min_bytes(_lib.F32, B, T, H, 64)
    assert full[1][-1].numel() > 2 * least
    out, s = torch.empty_like(ops[2]), torch.empty_like(ops[6])
    with Room(least + MB):
        tight = rwkv7.batched_wkv7_fwd(*ops, length, ns, B, buffers={"out": out, "new_s": s})
    assert tight[1][-1].numel() == least
    for a, b in zip((out, s, *rwkv7.batched_wkv7_bwd(tight[1], (ds, dy), B)), (full[0][1], full[0][0], *want)):
        assert rel_err(npf(a), npf(b)) < 1e-5
