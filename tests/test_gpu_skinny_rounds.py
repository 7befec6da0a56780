"""The few-token product where blocks stay over several tiles and where each tile has a block of its own: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# a tile for each of two blocks per SM and one more; the edges of the sizes that keep a block per tile from 12 tokens on; fewer
# chunks of k than warps, chunks that end inside a warp's turn, x that stays for all tiles and x that does not
@pytest.mark.parametrize("tokens", [1, 8, 9, 11, 12, 16])
@pytest.mark.parametrize("n,k", [(4736, 96), (4737, 96), (4752, 1536), (4752, 2048), (6624, 3072), (6640, 3072), (5000, 3104), (9480, 1056)])
def test_rounds(tokens, n, k):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(n + k)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda").bfloat16()
    x, w, bias = rand(tokens, k), rand(n, k), rand(n)
    product = lambda w, b: ops.gemm_skinny(w, x, torch.full((tokens, w.shape[0]), float("nan"), device="cuda"), b)
    # up to 2,048 rows at a time are fewer tiles than SMs
    pieces = torch.cat([product(w[a:a + 2048].contiguous(), bias[a:a + 2048].contiguous()) for a in range(0, n, 2048)], 1)
    whole = product(w, bias)
    assert torch.equal(whole, pieces)
    want = x.double() @ w.double().T + bias.double()
    size = x.double().abs() @ w.double().abs().T
    # k / 16 sums of the tensor cores, which cut off below their largest term, and one of 16 warps and the bias
    assert ((whole.double() - want).abs() <= size * (k / 16 + 17) * 2.0 ** -22).all()


@pytest.mark.parametrize("tokens", [1, 9, 16])
@pytest.mark.parametrize("inner,k", [(2368, 96), (2369, 96), (2376, 2048), (3320, 2048), (4741, 1536)])
def test_gated_rounds(tokens, inner, k):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(inner + k)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda").bfloat16()
    x, gate, up, bias = rand(tokens, k), rand(inner, k), rand(inner, k), rand(2, inner)
    for biased in (False, True):
        def product(a, b):
            out = torch.full((tokens, b - a), float("nan"), device="cuda", dtype=torch.bfloat16)
            return ops.gemm_skinny_swiglu(torch.cat([gate[a:b], up[a:b]]), x, out, bias[:, a:b].flatten().contiguous() if biased else None)
        pieces = torch.cat([product(a, min(a + 1024, inner)) for a in range(0, inner, 1024)], 1)
        assert torch.equal(product(0, inner), pieces) and not torch.isnan(pieces).any()
