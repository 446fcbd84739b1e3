"""GPU tests of the fp32 RWKV-7 kernels that take 16 tokens at a time (csrc/wkv7_fp32.cu), against the oracle in 64 bits: the edges
of their chunks, each split of the rows over thread blocks, chunks walked token by token, decays that vanish, missing cotangents."""
import numpy as np
import pytest
import torch

import oracle
from jaxrwkv_b200 import rwkv7
from conftest import rel_err
from gpu_util import NAMES7, flags, npf, rounded, to_dev, wkv7_case

pytestmark = pytest.mark.gpu
GRADS = ("dr", "dw", "dk", "dv", "da", "db", "ds0")
# a result is a few hundred products and sums of 24-bit numbers behind one another; the tests' common tolerance is 1e-4
TOL = 1e-5


def check(d, H, gy=True, gs=True, tol=TOL):
    B, T = d["k"].shape[:2]
    t = to_dev(d, torch.float32)
    length, ns = (x.cuda() for x in flags(d))
    g = torch.Generator().manual_seed(3)
    gy = torch.randn(t["k"].shape, generator=g).cuda() if gy else None
    gs = torch.randn(t["s0"].shape, generator=g).cuda() if gs else None
    ins = rounded(t)
    so, yo = oracle.wkv7_base_batched(*ins, d["length"], d["new_starts"])
    with torch.no_grad():                                    # with a workspace
        s, y = rwkv7.CudaRWKV.inner_loop(*[t[n] for n in NAMES7], length, ns)
    leaves = [t[n].requires_grad_(True) for n in NAMES7]
    s1, y1 = rwkv7.CudaRWKV.inner_loop(*leaves, length, ns)  # with a residual
    for got in ((s, y), (s1, y1)):
        assert rel_err(npf(got[0]), so) < tol and rel_err(npf(got[1]), yo) < tol
    outs = [(y1, gy), (s1, gs)]
    grads = torch.autograd.grad([o for o, c in outs if c is not None], leaves, [c for _, c in outs if c is not None])
    ref = oracle.wkv7_bwd_batched(*ins, d["length"], d["new_starts"], npf(gy) if gy is not None else np.zeros_like(yo),
                                  npf(gs) if gs is not None else np.zeros_like(so))
    for n, a, b in zip(GRADS, grads, ref):
        assert rel_err(npf(a), b) < tol, n


# each split of a head's rows on 148 SMs; token by token, whole chunks, ragged ones; without gradients from 13 chunks on
@pytest.mark.parametrize("B,H,T", [(1, 2, 384), (1, 2, 385), (1, 2, 400), (3, 5, 224), (3, 5, 225), (3, 5, 256), (3, 5, 271), (4, 8, 161), (4, 8, 512),
                                   (4, 8, 527), (4, 10, 112), (4, 10, 113), (4, 10, 143), (16, 10, 63), (16, 10, 64), (16, 10, 65),
                                   (1, 4, 192), (1, 4, 193), (4, 9, 195)])
def test_sizes(B, H, T):
    check(wkv7_case(B, T, H, seed=T + B, s0_scale=0.3), H)


@pytest.mark.parametrize("B,H", [(4, 1), (4, 4)])
def test_flags_and_lengths_at_chunk_edges(B, H):
    T = 352
    starts = [[0, 16, 32], [15, 31, 351], [1, 48, 49, 96], []]
    lengths = [0, 48, 47, 97]                                # none; the end of a chunk; inside one; its first token
    check(wkv7_case(B, T, H, seed=H, s0_scale=0.3, starts=starts, lengths=lengths), H)


# each split: chunks walked token by token many times around the stages, among whole ones, and in a row
@pytest.mark.parametrize("B,H", [(1, 4), (3, 5), (4, 8), (4, 10)])
@pytest.mark.parametrize("p_start", [0.03, 0.3])
def test_flags_in_many_chunks(B, H, p_start):
    check(wkv7_case(B, 16 * 24 + 5, H, seed=B + H, s0_scale=0.3, p_start=p_start, random_length=True), H)


@pytest.mark.parametrize("gy,gs", [(True, False), (False, True)])
def test_one_cotangent(gy, gs):
    check(wkv7_case(2, 340, 2, seed=4, p_start=0.02, random_length=True, s0_scale=0.3), 2, gy, gs)


def test_decays_that_vanish():
    d = wkv7_case(2, 352, 2, seed=9, s0_scale=0.3)
    d["w"][:, ::3] = 6.0                                     # exp(-exp(6)) is 0 in 32 bits
    d["w"][:, 1::3] = 4.0                                    # 2e-24 a token
    check(d, 2)


@pytest.mark.parametrize("at", [16, 21])                     # the first token of a chunk; inside one
def test_a_flag_holds_back_what_is_not_a_number(at):
    B, T, H = 1, 400, 2
    d = wkv7_case(B, T, H, seed=5, starts=[[at]], s0_scale=0.3)
    length, ns = (x.cuda() for x in flags(d))
    for name in ("k", "v", "a", "b", "w", "s0"):
        clean, bad = to_dev(d, torch.float32), to_dev(d, torch.float32)
        bad[name].reshape(-1, 64)[0, 3] = float("nan")       # token 0, head 0 (s0: row 0)
        s, y = rwkv7.CudaRWKV.inner_loop(*[clean[n].requires_grad_(True) for n in NAMES7], length, ns)
        s1, y1 = rwkv7.CudaRWKV.inner_loop(*[bad[n].requires_grad_(True) for n in NAMES7], length, ns)
        assert torch.equal(y[:, at:], y1[:, at:]) and torch.equal(s, s1)
        dy = torch.randn_like(y)
        one = torch.autograd.grad(y, [clean[n] for n in NAMES7[:-1]], dy)
        two = torch.autograd.grad(y1, [bad[n] for n in NAMES7[:-1]], dy)
        for a, b in zip(one, two):
            assert torch.equal(a[:, at:], b[:, at:]), name


# each split of the rows: the stages of a walked chunk's rows are handed back behind their last use, so that repeated calls are equal
@pytest.mark.parametrize("B,H", [(1, 4), (3, 5), (4, 8), (4, 10)])
def test_walked_chunks_are_the_same_every_time(B, H):
    T = 512
    d = wkv7_case(B, T, H, seed=8, s0_scale=0.3, starts=[range(3, T, 7)] * B)
    t = to_dev(d, torch.float32)
    length, ns = (x.cuda() for x in flags(d))
    leaves = [t[n].requires_grad_(True) for n in NAMES7]
    gy, gs = torch.randn_like(t["k"]), torch.randn_like(t["s0"])

    def once():
        s, y = rwkv7.CudaRWKV.inner_loop(*leaves, length, ns)
        return s, y, *torch.autograd.grad((y, s), leaves, (gy, gs))
    first = once()
    for _ in range(60):
        assert all(torch.equal(a, b) for a, b in zip(once(), first))


# The common bound leaves room for what decays that vanish and lone cotangents lose; of the model's own distributions the worst gradient
# is 1.41e-7 off, as token by token (1.39e-7), the outputs 0.98e-7 (1.02e-7): within four roundings to 24 bits
@pytest.mark.parametrize("T,p_start", [(512, 0.0), (512, 1 / 128), (333, 1 / 16)])
def test_errors_are_those_of_a_few_roundings(T, p_start):
    check(wkv7_case(2, T, 12, seed=T, p_start=p_start, random_length=p_start > 0, s0_scale=0.3), 12, tol=2.0 ** -22)
