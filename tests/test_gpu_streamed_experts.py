"""The products that stream the matrices of experts with few rows (lists of tiles of 16 rows) against plain
64-bit products, at the edges of tiles, items and slots along k; in bfloat16 they give the tiled products' bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# experts, top, tokens, hidden, inner, experts that are met (None: any)
SIZES = [
    (5, 1, 1, 32, 32, None),          # a single row, a quarter of a slot
    (4, 2, 3, 64, 96, None),          # items of 32 and 16 columns that end inside
    (7, 3, 16, 288, 40 * 4, None),    # two whole slots and a quarter, one and a quarter
    (3, 1, 17, 1056, 96, [1]),        # one expert meets 17 rows: a full tile and a tile of one row
    (2, 1, 40, 512, 2080, [0]),       # three tiles of one expert, many items per block
    (64, 6, 8, 2048, 1408, None),     # a routed layer of a decode step
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mode", ["gated", "plain"])
@pytest.mark.parametrize("experts,top,tokens,hidden,inner,met", SIZES)
def test_streamed_expert_products(experts, top, tokens, hidden, inner, met, mode, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    torch.manual_seed(experts * 1000 + tokens)
    gated = mode == "gated"
    pairs, tile = tokens * top, ops.moe_few_tile_rows()
    w1 = torch.randn(experts, (2 if gated else 1) * inner, hidden, device="cuda").to(dtype) * hidden ** -0.5
    w2 = torch.randn(experts, hidden, inner, device="cuda").to(dtype) * inner ** -0.5
    x = torch.randn(tokens, hidden + 8, device="cuda").to(dtype)[:, :hidden]        # rows with a gap between them
    ids = torch.stack([torch.randperm(experts)[:top] for _ in range(tokens)]).int().cuda()
    if met is not None:
        ids.fill_(met[0])
    assert ops.moe_few_fits(x, hidden, inner)
    lists = ops.moe_align(ids, pairs, experts, torch.zeros(ops.moe_lists_size(pairs, experts, tile),
                                                           dtype=torch.int32, device="cuda"), tile)
    act = torch.full((pairs, inner), float("nan"), device="cuda", dtype=dtype)
    out = torch.full((pairs, hidden), float("nan"), device="cuda", dtype=dtype)
    ops.moe_product(x, w1, act, lists, pairs, top, gated, "silu" if gated else "relu2", first=True, tile=tile)
    ops.moe_product(act, w2, out, lists, pairs, top, False, tile=tile)

    if dtype is torch.bfloat16:
        wide = ops.moe_align(ids, pairs, experts, torch.zeros(ops.moe_lists_size(pairs, experts), dtype=torch.int32,
                                                              device="cuda"))
        tiled_act, tiled = torch.empty_like(act), torch.empty_like(out)
        ops.moe_product(x, w1, tiled_act, wide, pairs, top, gated, "silu" if gated else "relu2", first=True)
        ops.moe_product(act, w2, tiled, wide, pairs, top, False)
        assert torch.equal(act, tiled_act) and torch.equal(out, tiled)

    order = lists[1].long()
    expert = ids.view(-1).long()[order]
    rows = x.double()[order // top]
    first = torch.einsum("ph,pih->pi", rows, w1.double()[expert]).to(dtype).double()
    if gated:
        want_act = torch.nn.functional.silu(first[:, :inner]) * first[:, inner:]
    else:
        want_act = torch.relu(first) ** 2
    # a value next to a rounding edge may round the other way before the activation, which f and the other
    # factor (up to about 5 each) carry on: a few units of the storage type; 32-bit sums over k <= 2,080
    # random terms differ by about 1e-6
    tolerance = 3e-2 if dtype is torch.bfloat16 else 1e-5
    scale = want_act.abs().max()
    assert float((act.double() - want_act).abs().max()) <= tolerance * float(scale)
    want = torch.empty(pairs, hidden, dtype=torch.float64, device="cuda")
    want[order] = torch.einsum("pi,phi->ph", act.double(), w2.double()[expert])
    tolerance = 8e-3 if dtype is torch.bfloat16 else 1e-5           # one rounding of the result: 2^-8 of it at most
    assert float((out.double() - want).abs().max()) <= tolerance * float(want.abs().max())


def test_no_expert_is_met():
    """Every choice names an identity expert: no tile, and the products leave everything as it was."""
    from from_scratch_inference_engine_b200.kernels import ops
    tile = ops.moe_few_tile_rows()
    ids = torch.full((4, 2), 3, dtype=torch.int32, device="cuda")
    lists = ops.moe_align(ids, 8, 3, torch.zeros(ops.moe_lists_size(8, 3, tile), dtype=torch.int32, device="cuda"), tile)
    for dtype in (torch.bfloat16, torch.float32):
        act = torch.full((8, 64), 7.0, device="cuda", dtype=dtype)
        ops.moe_product(torch.ones(4, 32, device="cuda", dtype=dtype), torch.ones(3, 64, 32, device="cuda", dtype=dtype),
                        act, lists, 8, 2, False, "relu2", first=True, tile=tile)
        assert float(act.min()) == 7.0 and float(act.max()) == 7.0
