"""The scan of one token per request against the walk of any number of tokens: the same bits, and the state at once or after the wait."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# head sizes that the step kernel takes (four and eight rows a thread, rows and columns that end inside) and some that it does
# not (up to 32 rows, more than 128, columns or a state off the 16 bytes); shared q and k; a padding entry; every decay
@pytest.mark.parametrize("kind", ["silu", "silu16", "head", "token", "row", "row16"])
@pytest.mark.parametrize("heads,dim,vdim,share,gap", [(16, 128, 128, 1, 0), (4, 33, 36, 1, 4), (6, 64, 256, 3, 0), (3, 100, 20, 1, 8),
                                                      (2, 32, 32, 1, 0), (1, 136, 64, 1, 0), (2, 64, 33, 1, 0), (2, 64, 32, 1, 3)])
def test_one_token_per_request(heads, dim, vdim, share, gap, kind):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(heads * dim)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    items, qk = 4, heads // share * dim
    dtype = torch.bfloat16 if kind.endswith("16") else torch.float32
    state, proj = rand(5, heads * dim * vdim + gap), rand(items + 1, 2 * qk + heads * vdim + 8).to(dtype)
    decay = torch.rand({"silu": heads, "head": heads, "token": (items + 1) * heads, "row": (items + 1) * heads * dim}[kind.replace("16", "")],
                       generator=generator, device="cuda")
    given = {"token": {"decay_tok": decay}, "row": {"decay_row": decay}}.get(kind.replace("16", ""), {})
    results = []
    for rows, early in ((items, False), (items, True), (items + 1, False)):    # a row more than requests: the general walk
        mine, out = state.clone(), torch.full((items + 1, heads * vdim), float("nan"), device="cuda")
        torch.cuda.synchronize()
        ops.lightning_scan(proj[:rows], 0, qk, 2 * qk, ints([0, 1, 2, 3]), ints([1] * items), ints([2, -1, 0, 4]), items, mine,
                           None if given else decay, out, heads, dim, vdim, share=share, out_scale=0.5, silu=kind.startswith("silu"),
                           early=early, **given)
        results.append((out.nan_to_num(7e7), mine))
    for got in results[:2]:
        assert torch.equal(got[0], results[2][0]) and torch.equal(got[1], results[2][1])
