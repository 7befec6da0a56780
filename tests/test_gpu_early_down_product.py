"""The experts' second product that asks for its matrices before the first has finished: the bits of the one that waits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# fewer items than blocks, one slot and more than the five that are asked for ahead, items that end inside, a last item of a
# block asked for ahead together with the next
@pytest.mark.parametrize("experts,top,tokens,hidden,inner", [(5, 1, 1, 32, 32), (4, 2, 3, 64, 96), (7, 3, 16, 288, 160),
                                                             (2, 1, 40, 512, 2080), (64, 6, 8, 2048, 1408), (128, 8, 8, 4096, 128)])
def test_matrices_before_the_wait(experts, top, tokens, hidden, inner):
    from from_scratch_inference_engine_b200.kernels import ops
    torch.manual_seed(experts + tokens)
    pairs, tile, dtype = tokens * top, ops.moe_few_tile_rows(), torch.bfloat16
    w1 = torch.randn(experts, 2 * inner, hidden, device="cuda").to(dtype) * hidden ** -0.5
    w2 = torch.randn(experts, hidden, inner, device="cuda").to(dtype) * inner ** -0.5
    x = torch.randn(tokens, hidden, device="cuda").to(dtype)
    ids = torch.stack([torch.randperm(experts)[:top] for _ in range(tokens)]).int().cuda()
    lists = ops.moe_align(ids, pairs, experts, torch.zeros(ops.moe_lists_size(pairs, experts, tile), dtype=torch.int32,
                                                           device="cuda"), tile)
    outs = []
    for early in (False, True, True):
        act = torch.full((pairs, inner), float("nan"), device="cuda", dtype=dtype)
        out = torch.full((pairs, hidden), float("nan"), device="cuda", dtype=dtype)
        ops.moe_product(x, w1, act, lists, pairs, top, True, first=True, tile=tile)
        ops.moe_product(act, w2, out, lists, pairs, top, False, tile=tile, early=early)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]) and not torch.isnan(outs[0]).any()
