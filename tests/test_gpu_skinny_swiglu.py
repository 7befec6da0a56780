"""The few-token product with SwiGLU in its epilogue: the bits of the product and the SwiGLU kernel in turn."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 8, 9, 16])
@pytest.mark.parametrize("inner,k", [(8, 32), (12, 96), (130, 1536), (2816, 2048), (8960, 1536)])
def test_skinny_swiglu(tokens, inner, k):
    from from_scratch_inference_engine_b200.kernels import ops
    torch.manual_seed(tokens + inner)
    x = torch.randn(tokens, k + 8, device="cuda").bfloat16()[:, :k]
    w = (torch.randn(2 * inner, k, device="cuda") * 3 * k ** -0.5).bfloat16()
    both = torch.empty(tokens, 2 * inner, device="cuda", dtype=torch.bfloat16)
    want = torch.empty(tokens, inner, device="cuda", dtype=torch.bfloat16)
    ops.swiglu(ops.gemm_skinny(w, x, both, None), want)
    room = torch.full((tokens, inner + 3), 7.0, device="cuda", dtype=torch.bfloat16)
    got = ops.gemm_skinny_swiglu(w, x, room[:, :inner])
    assert torch.equal(got, want)
    assert torch.equal(room[:, inner:], torch.full((tokens, 3), 7.0, device="cuda", dtype=torch.bfloat16))
    if inner * k < 10 ** 6:
        gate, up = (x.double() @ w.double().T).bfloat16().double().chunk(2, dim=1)
        exact = torch.nn.functional.silu(gate) * up
        # a sum next to a rounding edge may round the other way: a unit of bfloat16 in either factor, and one of
        # the result
        assert ((got.double() - exact).abs() <= 2.0 ** -6 * exact.abs() + 1e-4).all()
