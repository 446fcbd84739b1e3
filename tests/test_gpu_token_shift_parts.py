"""GPU test of the token shift's backward where a tile's four parts of 16 tokens begin and end, with a start flag and the last
row on either side of a part's edge, and where channels end inside a block."""
import pytest
import torch

from jaxrwkv_b200.token_shift import token_shift

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [15, 16, 17, 49, 64, 65, 129])
@pytest.mark.parametrize("D", [64, 264])
def test_backward_at_part_edges(T, D):
    B, M = 2, 3
    g = torch.Generator().manual_seed(T + D)
    x, prev, mix = (torch.randn(*s, generator=g) for s in ((B, T, D), (B, D), (M, D)))
    ns = torch.zeros(B, T, dtype=torch.bool)
    ns[0, [t for t in (15, 16, 48) if t < T]] = True
    length = torch.tensor([T, min(16, T)])
    gout, gs = torch.randn(M, B, T, D, generator=g), torch.randn(B, D, generator=g)

    def plain(x, prev, mix):
        shifted = torch.cat([prev[:, None], x[:, :-1]], 1) * ~ns[..., None]
        return x + (shifted - x) * mix[:, None, None], x[torch.arange(B), length - 1]

    leaves = [t.clone().requires_grad_(True) for t in (x, prev, mix)]
    want = torch.autograd.grad(plain(*leaves), leaves, (gout, gs))
    cuda = [t.cuda().requires_grad_(True) for t in (x, prev, mix)]
    got = torch.autograd.grad(token_shift(*cuda, length.cuda(), ns.cuda()), cuda, (gout.cuda(), gs.cuda()))
    for a, b in zip(got, want):
        assert (a.cpu() - b).abs().max() <= 1e-5 * b.abs().max()
