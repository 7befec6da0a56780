"""Norms of steps of few tokens without launches of their own: the products that add to the residual stream and the products
that finish the norm, against 64 bits and against the norm kernel between plain products; gated products with a bias."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def bf16(x):
    return x.to(torch.bfloat16)


# one token, the edges of tiles of 8 and 16 tokens; widths that end inside a block of 16 columns, inside a tile of 128, and
# with the k range cut over a cluster; a gain in either type; `few`: the tcgen05 product on both sides
@pytest.mark.parametrize("few", [False, True])
@pytest.mark.parametrize("gain_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,width,inner", [(1, 32, 32), (7, 96, 416), (8, 1536, 64), (9, 160, 2048), (16, 2048, 96), (3, 40, 64)])
def test_residual_and_norm_around_products(tokens, width, inner, gain_type, few):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(tokens * 1000 + width)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    a, w1 = bf16(rand(tokens, inner)), bf16(rand(width, inner) * inner ** -0.5)
    bias = bf16(rand(width))
    gain = (rand(width) * 0.2 + 1).to(gain_type)
    x, eps = rand(tokens, width) * 3, 1e-6
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    late = ops.LateRows(torch.empty(tokens, width, dtype=torch.bfloat16, device="cuda"),
                        torch.full((tokens, -(-width // ops.LATE_COLUMNS)), float("nan"), device="cuda"), eps)
    got = x.clone()
    into = ops.LateResidual(got, gain, late)
    plain = torch.empty(tokens, width, dtype=torch.bfloat16, device="cuda")
    if few:
        for splits in (1, 2, 4, 8):
            got.copy_(x)
            late.parts.fill_(float("nan"))
            ops.gemm_decode(ops.DecodeWeight(w1), a, None, bias, error, splits, None, into)
            ops.gemm_decode(ops.DecodeWeight(w1), a, plain, bias, error, splits)
            assert torch.equal(got, x + plain.float())
    else:
        ops.gemm_skinny(w1, a, None, bias, None, None, into)
        ops.gemm_skinny(w1, a, plain, bias)
    # the stream is what the norm kernel makes of the plain product: the same bits; the rows are its values times the gain
    assert torch.equal(got, x + plain.float())
    assert torch.equal(late.rows, bf16(got * gain.float()))
    squares = torch.nn.functional.pad(got.double() ** 2, (0, -width % 16)).view(tokens, -1, 16).sum(-1)
    assert ((late.parts.double() - squares).abs() <= squares * 16 * 2.0 ** -24).all()

    # the products behind: against 64 bits of the same bfloat16 rows, rounded once (gate and up: before the activation too)
    if width % 32 and not few:
        return
    n = 48
    w2 = bf16(rand(2 * n, width) * width ** -0.5)
    factor = 1 / (got.double().square().mean(-1, keepdim=True) + eps).sqrt()
    sums = (late.rows.double() @ w2.double().T) * factor
    slack = 1e-5 * (late.rows.double().abs() @ w2.double().abs().T) * factor         # 32-bit sums
    half = 2.0 ** -8
    y = torch.empty(tokens, 2 * n, dtype=torch.bfloat16, device="cuda")
    act = torch.empty(tokens, n, dtype=torch.bfloat16, device="cuda")
    if few:
        ops.gemm_decode(ops.DecodeWeight(w2), late.rows, y, None, error, 1, late)
        ops.gemm_decode(ops.DecodeWeight(w2, True), late.rows, act, None, error, 1, late)
    else:
        ops.gemm_skinny(w2, late.rows, y, None, None, late)
        ops.gemm_skinny_swiglu(w2, late.rows, act, late)
    assert ((y.double() - sums).abs() <= slack + half * sums.abs()).all()
    gate, up = sums[:, :n], sums[:, n:]
    want = gate * torch.sigmoid(gate) * up
    bound = 1.2 * (half * gate.abs() + slack[:, :n]) * up.abs() + 1.1 * (half * up.abs() + slack[:, n:]) * gate.abs() + half * want.abs()
    assert ((act.double() - want).abs() <= bound + 1e-6).all()
    assert int(error.item()) == 0


def test_rotated_projection_of_pending_rows():
    """The fused q, k, v product over rows with a pending norm against the same product over the normed rows."""
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    tokens, width, heads, kv_heads, dim, page = 5, 96, 4, 2, 32, 16
    n = (heads + 2 * kv_heads) * dim
    w, bias, v = bf16(rand(n, width) * width ** -0.5), bf16(rand(n)), rand(tokens, width) * 2
    late = ops.LateRows(bf16(v), v.square().view(tokens, -1, 16).sum(-1).contiguous(), 1e-6)
    normed = late.rows.double() * (1 / (v.double().square().mean(-1, keepdim=True) + 1e-6).sqrt())
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    table, error = rand(64, dim), ints([0])
    rows = []
    for x, norm in ((late.rows, late), (bf16(normed), None)):
        pages = torch.zeros(4, 2, kv_heads, page, dim, dtype=torch.bfloat16, device="cuda")
        out = torch.zeros(tokens, n, dtype=torch.bfloat16, device="cuda")
        ops.gemm_skinny_qkv_rope(w, x, out, bias, ints([0, 5, 63, 7, 9]), table, ints([3, 17, 40, -1, 63]), pages[:, 0], pages[:, 1],
                                 pages.stride(0), page, heads, kv_heads, dim, error, norm)
        rows.append(torch.cat([out.flatten(), pages.flatten()]).double())
    assert int(error.item()) == 0
    # two roundings of a row to bfloat16 (2^-9 of a value at most, each way), summed over a row of 96: well below these
    assert ((rows[0] - rows[1]).abs().max() / rows[1].square().mean().sqrt()) < 0.06
    assert ((rows[0] - rows[1]).norm() / rows[1].norm()) < 6e-3


@pytest.mark.parametrize("tokens", [1, 8, 16])
def test_step_with_and_without(tokens):
    """A decoder's step with pending norms and with the norm kernels: the same logits up to roundings to bfloat16."""
    from from_scratch_inference_engine_b200 import LoadedModel, ModelRunner, StepEntry
    from from_scratch_inference_engine_b200.config import config_from_dict
    from from_scratch_inference_engine_b200.parts.model import tensor_specs
    generator = torch.Generator(device="cuda").manual_seed(tokens)
    config = config_from_dict(dict(
        architectures=["Qwen2ForCausalLM"], model_type="qwen2", num_hidden_layers=3, hidden_size=192,
        num_attention_heads=6, num_key_value_heads=2, head_dim=32, intermediate_size=416, vocab_size=300,
        rope_theta=1e4, tie_word_embeddings=True, max_position_embeddings=64))
    weights = {}
    for spec in tensor_specs(config.build_spec()):
        if not spec.optional:
            t = torch.randn(spec.shape, generator=generator, device="cuda") * 0.05
            weights[spec.name] = bf16(t + 1 if spec.init == "gain" else t)
    rows = {}
    for late in (True, False):
        model = LoadedModel.from_tensors(config, {k: v.clone() for k, v in weights.items()}, "bfloat16", "cuda:0", max_positions=64)
        model.runtime.late_norms = late
        assert bool(model.model.blocks[1].late_norm(tokens)) == late
        runner = ModelRunner(model.model, model.runtime, page_size=16, num_pages=64, max_requests=16)
        handles = [runner.cache.open(r) for r in range(tokens)]
        got = [runner.step([StepEntry(handles[0], list(range(tokens)), [tokens - 1])]).clone()]        # a short prompt
        for turn in range(3):                                                                         # and captured steps
            entries = [StepEntry(h, [(7 * r + turn) % 300], [0]) for r, h in enumerate(handles)]
            got.append(runner.step(entries).clone())
        rows[late] = torch.cat(got).double()
        runner.raise_on_device_error()
    assert (rows[True] - rows[False]).norm() / rows[False].norm() < 2e-2


@pytest.mark.parametrize("few", [False, True])
@pytest.mark.parametrize("tokens,inner,width", [(1, 8, 32), (9, 72, 96), (16, 130, 512), (8, 8960, 64)])
def test_gated_product_with_bias(tokens, inner, width, few):
    """The bits of the stacked product with its bias and the SwiGLU kernel behind it."""
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(inner)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda").to(torch.bfloat16)
    x, w, bias = rand(tokens, width), rand(2 * inner, width) * width ** -0.5, rand(2 * inner)
    both, got = (torch.empty(tokens, n, dtype=torch.bfloat16, device="cuda") for n in (2 * inner, inner))
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    if few:
        for splits in (1, 2):
            ops.gemm_decode(ops.DecodeWeight(w), x, both, bias, error, splits)
            ops.gemm_decode(ops.DecodeWeight(w, True), x, got, bias, error, splits)
            assert torch.equal(got, ops.swiglu(both, torch.empty_like(got)))
    else:
        ops.gemm_skinny(w, x, both, bias)
        ops.gemm_skinny_swiglu(w, x, got, None, bias)
        assert torch.equal(got, ops.swiglu(both, torch.empty_like(got)))
    assert int(error.item()) == 0
