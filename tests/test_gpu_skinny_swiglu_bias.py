"""The few-token product with a bias and SwiGLU in its epilogue: the bits of the product and the SwiGLU kernel in turn."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# the edges of 8 and 16 tokens; outputs that end inside a block's 8 rows
@pytest.mark.parametrize("tokens", [1, 8, 9, 16])
@pytest.mark.parametrize("inner,k", [(8, 32), (13, 96), (130, 1536), (5632, 2048)])
def test_bias_of_a_gated_pair(tokens, inner, k):
    from from_scratch_inference_engine_b200.engine.runtime import Runtime
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(tokens + inner)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    x, w, bias = rand(tokens, k).bfloat16(), (rand(2 * inner, k) * 3 * k ** -0.5).bfloat16(), rand(2 * inner).bfloat16()
    both, want, got = (torch.empty(tokens, n, device="cuda", dtype=torch.bfloat16) for n in (2 * inner, inner, inner))
    ops.swiglu(ops.gemm_skinny(w, x, both, bias), want)
    assert torch.equal(ops.gemm_skinny_swiglu(w, x, got, bias), want)
    assert torch.equal(Runtime().linear_swiglu(x, w, None, bias), want)


# the same through the product on prepared (large) matrices: blocks that share k, tiles that end inside, 1 to 64 tokens
@pytest.mark.parametrize("tokens", [1, 16, 17, 32, 64])
@pytest.mark.parametrize("inner,k", [(64, 64), (100, 512), (5632, 2048)])
def test_bias_of_a_prepared_gated_pair(tokens, inner, k):
    from from_scratch_inference_engine_b200.engine.runtime import Runtime
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(tokens + inner)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    x, w, bias = rand(tokens, k).bfloat16(), (rand(2 * inner, k) * 3 * k ** -0.5).bfloat16(), rand(2 * inner).bfloat16()
    both, want = (torch.empty(tokens, n, device="cuda", dtype=torch.bfloat16) for n in (2 * inner, inner))
    runtime = Runtime(few_token_min_elements=1, few_token_limit=64)
    splits = ops.gemm_decode_splits(-(-inner // 64), k, runtime.sm_count)
    ops.swiglu(ops.gemm_decode(ops.DecodeWeight(w), x, both, bias, runtime.error, splits), want)
    runtime.prepare_weight(w, swiglu=True, biased=True)
    assert torch.equal(runtime.linear_swiglu(x, w, None, bias), want) and int(runtime.error.item()) == 0
