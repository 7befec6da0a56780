"""The state-space mixer's preparation of steps of one token per request in one launch against the two launches, and its gated
norm with a row in registers against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# taps that the one launch takes and one more; channels that end inside a block of 1,024; a head size that is no multiple of
# 8; requests in another order than their tokens; a padding entry; no bias
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,vdim,extra,taps,order", [(64, 64, 256, 4, (0, 1, 2, 3, 4)), (3, 8, 16, 2, (4, 1, 0, 2, 3)),
                                                         (2, 24, 40, 3, (0, 1, 2, 4, 3)), (2, 8, 16, 5, (0, 1, 2, 3, 4)),
                                                         (3, 12, 20, 4, (0, 1, 2, 3, 4))])
def test_one_launch_is_the_two(heads, vdim, extra, taps, order, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(heads * 100 + taps)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    items, inner = 5, heads * vdim
    channels, matrix = inner + extra, 32
    ld = -(-(inner + channels + heads) // 8) * 8
    proj = rand(items, ld).to(dtype)
    conv, bias = rand(channels, taps), rand(channels) if taps != 3 else None
    dt_bias, a_log = rand(heads), rand(heads)
    slots = [3, -1, 0, 5, 1]
    state = rand(6, -(-(matrix + (taps - 1) * channels) // 8) * 8)
    results = []
    for move in (True, False):
        act = torch.full((items, channels + inner), float("nan"), device="cuda")
        decay = torch.full((items, heads), float("nan"), device="cuda")
        mine = state.clone()
        lists = (ints(list(order)), ints([1] * items), ints(slots), items)
        ops.ssd_prep(proj, inner, inner + channels, *lists, mine, matrix, conv, bias, dt_bias, a_log, heads, vdim, act, decay,
                     conv_wt=conv.t().contiguous(), move_tails=move, one_each=move)
        if not move:
            ops.ssd_tails(proj, inner, channels, taps, *lists, mine, matrix)
        results.append((act, decay, mine))
    for got, want in zip(*results):
        assert torch.equal(got.nan_to_num(7e7), want.nan_to_num(7e7))
    assert torch.isnan(results[0][0]).any(1).tolist() == [order.index(t) == 1 for t in range(items)]      # the padding entry's
    assert torch.equal(results[0][2][:, :matrix], state[:, :matrix])


# as many tokens as requests, but not one each: a request's second token, and requests without any
@pytest.mark.parametrize("counts", [(2, 0), (0, 2), (1, 0, 3, 0)])
def test_as_many_tokens_as_requests(counts):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(len(counts))
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    heads, vdim, taps, items = 3, 8, 4, len(counts)
    inner = heads * vdim
    channels = inner + 16
    proj, conv = rand(items, 2 * inner + 24), rand(channels, taps)
    bias, dt_bias, a_log, state = rand(channels), rand(heads), rand(heads), rand(items, (taps - 1) * channels)
    lists = (ints([sum(counts[:i]) for i in range(items)]), ints(list(counts)), ints(list(range(items))), items)
    act, decay, mine = torch.full((items, channels + inner), float("nan"), device="cuda"), torch.empty(items, heads, device="cuda"), state.clone()
    call = lambda **given: ops.ssd_prep(proj, inner, inner + channels, *lists, mine, 0, conv, bias, dt_bias, a_log, heads, vdim, act,
                                        decay, conv_wt=conv.t().contiguous(), move_tails=True, **given)
    call()
    t = 0
    for i, n in enumerate(counts):
        history = torch.cat([state[i].view(taps - 1, channels), proj[t:t + n, inner:inner + channels]]).double()
        assert torch.equal(mine[i].double().view(taps - 1, channels), history[n:])
        for r in range(n):
            want = torch.nn.functional.silu((history[r:r + taps] * conv.t().double()).sum(0) + bias.double())
            assert ((act[t + r, :channels].double() - want).abs() <= 1e-5 * (1 + want.abs())).all()
        t += n
    with pytest.raises(ops.KernelError):                      # said to be one each, and not as many
        ops.ssd_prep(proj[:1], inner, inner + channels, *lists, mine, 0, conv, bias, dt_bias, a_log, heads, vdim, act, decay,
                     conv_wt=conv.t().contiguous(), move_tails=True, one_each=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,vdim,parts", [(64, 64, 1), (4, 8, 2), (3, 24, 1), (64, 128, 1), (65, 128, 1), (3, 12, 1),
                                              (25, 40, 1), (16, 64, 1), (16, 64, 2), (31, 64, 1), (40, 50, 1), (9, 40, 1),
                                              (26, 50, 1), (34, 50, 1), (50, 64, 1)])
def test_gated_norm(heads, vdim, parts, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(heads + vdim)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    tokens, inner = 3, heads * vdim
    o, act, proj = rand(tokens, inner), rand(tokens, inner + 8), rand(tokens, inner + 16).to(dtype)
    skip, gain = rand(heads), rand(inner)
    y = ops.ssd_gate_norm(o, act, proj, 8, skip, gain, torch.empty(tokens, inner, device="cuda", dtype=dtype), vdim, parts, 1e-5)
    z = proj[:, 8:8 + inner].double()
    v = (o.double() + skip.double().repeat_interleave(vdim) * act[:, :inner].double()) * z * torch.sigmoid(z)
    norm = v.view(tokens, parts, -1)
    want = (norm / (norm.square().mean(-1, keepdim=True) + 1e-5).sqrt()).view(tokens, inner) * gain.double()
    # the row in registers leaves the bits of the kernel for rows of any width
    general = ops.ssd_gate_norm(o, act, proj, 8, skip, gain, torch.empty_like(y), vdim, parts, 1e-5, general=True)
    assert torch.equal(y, general)
    # a few roundings of numbers of the order of one, times the gain, then one to the storage type
    assert ((y.double() - want).abs() <= 2e-5 * (1 + want.abs()) + (2.0 ** -8 * want.abs() if dtype is torch.bfloat16 else 0)).all()
