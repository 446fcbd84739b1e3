"""GPU test of the token shift's bf16 backward in each split of its work: four and two parts per tile, whole tiles, groups of
tokens that do not divide them, with start flags and last rows about the parts' and tiles' edges and a ragged last tile."""
import pytest
import torch

from jaxrwkv_b200.token_shift import token_shift

pytestmark = pytest.mark.gpu


# on 148 SMs, with five rows and more: 4 parts; 2 parts by groups of 8; of 4; whole tiles by groups of 8; of 5; of 3; with fewer the
# splits change at other counts: 2 parts in front of whole tiles, up to 12 blocks per SM and above, each with channels that 8 do not divide
@pytest.mark.parametrize("B,T,D", [(2, 129, 264), (130, 65, 256), (111, 150, 256), (250, 70, 256), (100, 129, 512), (500, 70, 252),
                                   (190, 70, 512), (700, 70, 256), (700, 70, 252), (900, 70, 256)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 6, 8])
def test_backward(B, T, D, M):
    g = torch.Generator().manual_seed(T + D)
    x, prev, mix = (torch.randn(*s, generator=g).bfloat16() for s in ((B, T, D), (B, D), (M, D)))
    ns = torch.zeros(B, T, dtype=torch.bool)
    ns[0, [15, 16, 32, 63, 64]] = True
    ns[1:, 33] = True
    length = torch.full((B,), T)
    length[1] = 32
    gout, gs = torch.randn(M, B, T, D, generator=g).bfloat16(), torch.randn(B, D, generator=g).bfloat16()

    def plain(x, prev, mix):
        shifted = torch.cat([prev[:, None], x[:, :-1]], 1) * ~ns[..., None]
        return x + (shifted - x) * mix[:, None, None], x[torch.arange(B), length - 1]

    leaves = [t.float().requires_grad_(True) for t in (x, prev, mix)]
    want = torch.autograd.grad(plain(*leaves), leaves, (gout.float(), gs.float()))
    cuda = [t.cuda().requires_grad_(True) for t in (x, prev, mix)]
    got = torch.autograd.grad(token_shift(*cuda, length.cuda(), ns.cuda()), cuda, (gout.cuda(), gs.cuda()))
    for a, b in zip(got, want):
        # a result's rounding is 2^-9 of itself; the sums before it, in 32 bits, take far less
        assert (a.cpu().float() - b).abs().max() <= 2 ** -8 * b.abs().max()
