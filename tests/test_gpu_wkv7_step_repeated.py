"""GPU test of the decoding step over more pairs than the device holds at once: the same step from the same states, in place and layer
behind layer, gives the same bits each time (a stage of the ring must not be refilled while its pair is being read)."""
import pytest
import torch

from jaxrwkv_b200 import rwkv7

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,B", [(torch.float32, 128), (torch.bfloat16, 256)])
def test_the_same_bits_every_time(dtype, B):
    H, N, L = 40, 64, 8
    g = torch.Generator(device="cuda").manual_seed(7)

    def rn(*s):
        return torch.randn(*s, generator=g, device="cuda")

    start = (0.5 * rn(B, L, 2 + N, H * N)).to(dtype)
    r, k, v = (rn(B, 1, H, N).to(dtype) for _ in range(3))
    w = (-1.0 + 0.5 * rn(B, 1, H, N)).to(dtype)
    a = torch.nn.functional.normalize(rn(B, 1, H, N), dim=-1)
    b = (-a * torch.rand(B, 1, H, N, generator=g, device="cuda")).to(dtype)
    a = a.to(dtype)
    first = None
    for _ in range(12):
        state = start.clone()
        ys = [rwkv7.wkv7_step_packed(r, w, k, v, a, b, state, layer) for layer in range(L)]
        if first is None:
            first = ys, state
            continue
        assert all(torch.equal(x, y) for x, y in zip(ys, first[0])) and torch.equal(state, first[1])
    S = start[0, :, 2:].float().reshape(L, H, N, N)          # one sequence of each layer in fp32
    x = [t[0, 0].float() for t in (r, w, k, v, a, b)]
    S = S * torch.exp(-torch.exp(x[1]))[:, None] + (S @ x[4][..., None]) * x[5][:, None] + x[3][..., None] * x[2][:, None]
    got = first[1][0, :, 2:].float().reshape(L, H, N, N)
    tol = 1e-5 if dtype == torch.float32 else 2 ** -8        # one rounding of the state to bf16 is 2^-9 of itself
    assert (got - S).abs().max() <= tol * S.abs().max()
