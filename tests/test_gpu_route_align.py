"""Choice and lists of a step of routed experts in one launch against the two launches: the same bits, the same rows per expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens: one, some and as many as the block has warps; experts at the edges of 32 per lane, one group of one, groups
# kept whole, more groups than lanes, identity experts; ties; every kind of scores
@pytest.mark.parametrize("scores,group_score", [("sigmoid", "top2"), ("softmax", "max"), ("chosen_softmax", "top2")])
@pytest.mark.parametrize("tokens,routed,experts,top,groups,keep", [
    (1, 1, 1, 1, 1, 1), (3, 6, 4, 2, 3, 2), (8, 64, 64, 6, 8, 4), (32, 32, 32, 32, 1, 1), (17, 33, 30, 4, 1, 1),
    (32, 256, 256, 8, 64, 3), (5, 130, 130, 7, 10, 10), (31, 80, 65, 32, 40, 20)])
def test_one_launch_is_the_two(tokens, routed, experts, top, groups, keep, scores, group_score):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(tokens * 1000 + routed)
    logits = torch.randn(tokens, routed, generator=generator, device="cuda") * 3
    logits[0, routed // 2:] = logits[0, 0].item()                                  # ties
    correction, bias = (torch.randn(routed, generator=generator, device="cuda") for _ in range(2))
    if scores == "chosen_softmax":
        correction = None
    assert tokens <= ops.MOE_ROUTE_ALIGN_TOKENS == ops.routed().fsie_moe_route_align_tokens()
    assert ops.moe_route_align_fits(tokens, routed, top)
    pairs = tokens * top
    for tile in (ops.moe_tile_rows(), ops.moe_few_tile_rows()):
        ids, want_ids = (torch.full((tokens, top), -7, dtype=torch.int32, device="cuda") for _ in range(2))
        weights, want_weights = (torch.full((tokens, top), float("nan"), device="cuda") for _ in range(2))
        lists, want_lists = (torch.full((ops.moe_lists_size(pairs, experts, tile),), -7, dtype=torch.int32, device="cuda")
                             for _ in range(2))
        ops.moe_route(None, None, correction, want_ids, want_weights, top, groups, keep, 2.5, scores, True,
                      logits=logits, group_score=group_score, bias=bias)
        want = ops.moe_align(want_ids, pairs, experts, want_lists, tile)
        got = ops.moe_route_align(logits, bias, correction, ids, weights, top, groups, keep, 2.5, scores, True, group_score,
                                  experts, lists, tile)
        assert torch.equal(ids, want_ids) and torch.equal(weights, want_weights)
        assert torch.equal(got[0], want[0]) and torch.equal(got[4], want[4])           # offsets, number of tiles
        tiles, rows = int(want[4].item()), int(want[0][-1].item())
        assert torch.equal(got[2][:tiles], want[2][:tiles]) and torch.equal(got[3][:tiles], want[3][:tiles])
        # an expert's rows in any order, and nothing behind the lists' ends
        assert [sorted(got[1][a:b].tolist()) for a, b in zip(want[0][:-1].tolist(), want[0][1:].tolist())] == \
            [sorted(want[1][a:b].tolist()) for a, b in zip(want[0][:-1].tolist(), want[0][1:].tolist())]
        assert (got[1][rows:] == -7).all() and (got[2][tiles:] == -7).all()
        assert int((ids.view(-1) < experts).sum().item()) == rows
