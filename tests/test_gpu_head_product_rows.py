"""Products per head of few tokens with their weights in registers: 64 bits, and the bits of the kernel that takes all sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one token and the edges of 4, 8 and 16; rows that end inside a warp's; every count of lanes and chunks a row has, with lanes that
# hold nothing; k that the kernel does not take, and rows that do not start on 16 bytes
@pytest.mark.parametrize("tokens", [1, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("heads,n,k,gap", [(16, 512, 128, 8), (2, 40, 32, 0), (3, 129, 200, 16), (5, 128, 512, 8), (1, 17, 1024, 8),
                                           (2, 19, 776, 8), (2, 24, 44, 4), (2, 32, 64, 4), (1, 8, 1032, 8),
                                           (130, 33, 40, 8), (64, 65, 128, 8), (32, 40, 256, 8)])
def test_head_product(tokens, heads, n, k, gap):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(n + k)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda").to(torch.bfloat16)
    x_head, out_head = k + gap, n + 3
    x, w = rand(tokens, heads * x_head + gap), rand(heads, n, k) * k ** -0.5
    out = torch.full((tokens, heads * out_head), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.head_product(x, x.stride(0), x_head, w, out, out.stride(0), out_head, tokens)
    shifted = torch.empty(x.numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view_as(x).copy_(x)      # off the 16 bytes
    general = ops.head_product(shifted, x.stride(0), x_head, w, torch.full_like(out, float("nan")), out.stride(0), out_head, tokens)
    assert torch.equal(out.nan_to_num(7e4), general.nan_to_num(7e4))
    rows = torch.stack([x[:, h * x_head:h * x_head + k] for h in range(heads)]).double()           # [heads, tokens, k]
    want = rows @ w.double().transpose(1, 2)
    got = torch.stack([out[:, h * out_head:h * out_head + n] for h in range(heads)]).double()
    size = rows.abs() @ w.double().abs().transpose(1, 2)
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + size * k * 2.0 ** -24).all()
    assert torch.isnan(torch.stack([out[:, h * out_head + n:(h + 1) * out_head] for h in range(heads)])).all()
