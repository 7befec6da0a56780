"""The weighted sum of experts' rows: eight columns a thread, several choices' rows together or one after the other, against the
scalar kernel, whose sums run in the same order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# the edges of the tokens that take choices one after the other; every number of choices that travel together and remainders;
# places looked up; identity experts; a shared expert
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens", [1, 256, 257, 1025])
@pytest.mark.parametrize("top", [1, 2, 3, 4, 5, 8, 9])
def test_choices_together(tokens, top, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(tokens + top)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    width, experts = 264, 4
    rows, weights, shared, y = rand(tokens * top, width).to(dtype), rand(tokens, top), rand(tokens, width).to(dtype), rand(tokens, width).to(dtype)
    place = torch.randperm(tokens * top, generator=generator, device="cuda").int()
    ids = torch.randint(0, 6, (tokens, top), generator=generator, device="cuda").int()       # 4 and 5: the token's own row
    for where in (None, place):
        for identity in ({}, dict(ids=ids, experts=experts, y=y)):
            outs = []
            for shift in (0, 1):                                         # off the 16 bytes: the scalar kernel
                out = torch.full((tokens * width + 1,), float("nan"), device="cuda", dtype=dtype)[shift:shift + tokens * width]
                outs.append(ops.moe_combine(rows, weights, shared, out.view(tokens, width), top, place=where, **identity).clone())
            assert torch.equal(*outs)
            at = (torch.arange(tokens * top, device="cuda") if where is None else where.long()).view(tokens, top)
            chosen = rows[at].double()
            if identity:
                chosen = torch.where((ids >= experts)[..., None], y[:, None].double(), chosen)
            want = (weights[..., None].double() * chosen).sum(1) + shared.double()
            size = (weights[..., None].double() * chosen).abs().sum(1) + shared.double().abs()
            bound = size * (top + 1) * 2.0 ** -24 + (want.abs() * 2.0 ** -8 if dtype is torch.bfloat16 else 0)
            assert ((outs[0].double() - want).abs() <= bound).all()
