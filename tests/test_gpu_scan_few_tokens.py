"""The scan that takes the activation itself, chunks of long prompts chained eight at a time, gated norm with a row in registers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim,vdim", [(4, 128, 128), (3, 10, 24), (2, 20, 33), (1, 256, 64)])
def test_scan_of_projections_as_they_are(heads, dim, vdim, dtype):
    """The bits of silu_rows and the scan behind it."""
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(dim)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    counts = (1, 20, 3)
    tokens, width = sum(counts), heads * (2 * dim + vdim)
    proj, state, decay = rand(tokens, width + 8).to(dtype), rand(4, heads, dim, vdim), torch.rand(heads, device="cuda")
    results = []
    for silu in (True, False):
        mine, out = state.clone(), torch.empty(tokens, heads * vdim, device="cuda")
        act = proj if silu else ops.silu_rows(proj, width, torch.empty(tokens, width, device="cuda"))
        ops.lightning_scan(act, 0, heads * dim, 2 * heads * dim, ints([0, 1, 21]), ints(list(counts)), ints([2, 0, 3]), 3, mine,
                           decay, out, heads, dim, vdim, silu=silu)
        results.append((out, mine))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("kind", ["head", "token", "row"])
@pytest.mark.parametrize("chunk,counts", [(4, (4, 35, 1)), (8, (64, 65, 7)), (1, (17, 8, 9))])
def test_chunks_chained_eight_at_a_time(chunk, counts, kind):
    """Against the walk token by token: sums in another order, 32-bit."""
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(sum(counts))
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    heads, dim, vdim, tokens = 2, 24, 40, sum(counts)
    starts = [sum(counts[:i]) for i in range(len(counts))]
    proj, state = rand(tokens, heads * (2 * dim + vdim)), rand(3, heads, dim, vdim)
    shape = {"head": (heads,), "token": (tokens, heads), "row": (tokens, heads * dim)}[kind]
    decay = torch.rand(shape, generator=generator, device="cuda") * 0.5 + 0.5
    given = {"head": {}, "token": {"decay_tok": decay}, "row": {"decay_row": decay}}[kind]
    items, rows = zip(*[(i, r) for i, n in enumerate(counts) for r in range(0, n, chunk)])
    results = []
    for chunks in ({}, dict(seg_item=ints(items), seg_row0=ints(rows), num_segs=len(items), seg_tokens=chunk,
                            chunk_states=torch.empty(len(items) * heads * dim * (vdim + 1), device="cuda"))):
        mine, out = state.clone(), torch.empty(tokens, heads * vdim, device="cuda")
        ops.lightning_scan(proj, 0, heads * dim, 2 * heads * dim, ints(starts), ints(list(counts)), ints([1, 0, 2]), 3, mine,
                           decay if kind == "head" else None, out, heads, dim, vdim, **given, **chunks)
        results.append((out, mine))
    for got, want in zip(*results):
        assert ((got - want).abs() <= 2e-5 * want.abs().max()).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [8, 264, 2048, 8192, 8200, 36])
def test_gated_norm_rows(width, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(width)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    o, proj, gain = rand(3, width), rand(3, width + 16).to(dtype), rand(width)
    got = ops.gated_rmsnorm(o, proj, 16, gain, 1e-6, torch.empty(3, width, device="cuda", dtype=dtype))
    want = o.double() / (o.double().square().mean(-1, keepdim=True) + 1e-6).sqrt() * gain * torch.sigmoid(proj[:, 16:].double())
    assert ((got.double() - want).abs() <= 1e-5 * (1 + want.abs()) + (2.0 ** -8 * want.abs() if dtype is torch.bfloat16 else 0)).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [8, 130, 264, 500, 512, 700, 1024, 1025, 1300, 1700, 2000, 2048, 2049, 4096])
def test_gated_norm_rows_are_the_general_kernels(width, dtype):
    """The row in registers leaves the bits of the kernel for rows of any width."""
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(width)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    o, proj, gain = rand(40, width), rand(40, width + 16).to(dtype), rand(width)
    got, want = (ops.gated_rmsnorm(o, proj, 16, gain, 1e-6, torch.empty(40, width, device="cuda", dtype=dtype), general=general)
                 for general in (False, True))
    assert torch.equal(got, want)
