"""Kernels that read in front of their wait for the kernel before them: the kernel before is one of this package's, still running
while the next is scheduled, and the last that it writes - over NaN - is an operand of that one.  With `early` the operand that is
read behind the wait, without it each of those that are read in front."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32
STRIDE = 4096 * 256            # elements that cast_rows' blocks write at a time


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def written_late(values):
    """`values` again, as the last elements that a launch of cast_rows over 24 strides writes."""
    from from_scratch_inference_engine_b200.kernels import ops
    total = 24 * STRIDE
    source = torch.zeros(total, device="cuda")
    source[total - values.numel():] = values.flatten().float()
    target = torch.full((total,), float("nan"), device="cuda", dtype=values.dtype)
    torch.cuda.synchronize()
    ops.cast_rows(source, target)
    return target[total - values.numel():].view(values.shape)


class Case:
    def __init__(self, seed):
        generator = torch.Generator(device="cuda").manual_seed(seed)
        self.rand = lambda *shape, dtype=F32: torch.randn(shape, generator=generator, device="cuda").to(dtype)

    def check(self, tensors, behind, in_front, call):
        """`behind`: the operands that the kernel reads behind its wait, `in_front`: those in front.  call(get, early) asks
        for its operands by get(names) when everything else is in place, launches and gives its results."""
        want = call(lambda *names: [tensors[name] for name in names], False)
        for names, early in ((behind, True), (in_front, False)):
            for late in names:
                got = call(lambda *asked: [written_late(tensors[name]) if name == late else tensors[name] for name in asked], early)
                for a, b in zip(got, want):
                    assert torch.equal(a.nan_to_num(7e4), b.nan_to_num(7e4)), (late, early)


@pytest.mark.parametrize("rows", [1, 5, 16])
def test_float32_product(rows):
    from from_scratch_inference_engine_b200.kernels import ops
    case = Case(rows)
    t = dict(x=case.rand(rows, 1540), w=case.rand(300, 1540))

    def call(get, early):
        out = torch.full((rows, 300), float("nan"), device="cuda")
        x, w = get("x", "w")
        return (ops.gemm_f32(x, w, None, out, kind="rows", early=early),)
    case.check(t, ["x"], ["w"], call)


@pytest.mark.parametrize("tokens,k", [(3, 64), (8, 512), (16, 1024), (2, 1032)])
def test_product_per_head(tokens, k):
    from from_scratch_inference_engine_b200.kernels import ops
    case = Case(k)
    t = dict(x=case.rand(tokens, 4 * k, dtype=BF16), w=case.rand(4, 72, k, dtype=BF16))

    def call(get, early):
        out = torch.full((tokens, 4 * 72), float("nan"), device="cuda", dtype=BF16)
        x, w = get("x", "w")
        return (ops.head_product(x, 4 * k, k, w, out, 4 * 72, 72, tokens, early=early),)
    case.check(t, ["x"], ["w"], call)


def test_norms():
    from from_scratch_inference_engine_b200.kernels import ops
    case, rows, width = Case(1), 3, 2048
    t = dict(x=case.rand(rows, width), d=case.rand(rows, width, dtype=BF16), gain=case.rand(width), bias=case.rand(width),
             streams=case.rand(rows, 4, width), mix=case.rand(4, 4), spread=case.rand(4), gather=case.rand(4),
             scale=case.rand(width), proj=case.rand(rows, width + 64, dtype=BF16), act=case.rand(rows, width + 8),
             skip=case.rand(width // 64))
    out = lambda: torch.full((rows, width), float("nan"), device="cuda", dtype=BF16)

    def rows_of(get, early):
        y = out()
        x, gain = get("x", "gain")
        return (ops.layernorm_rows(x, gain, 1e-6, y, early=early),)
    case.check(t, ["x"], ["gain"], rows_of)

    def added(get, early):
        y, x = out(), t["x"].clone()
        d, gain = get("d", "gain")
        ops.add_layernorm(x, d, gain, 1e-6, y, early=early)
        return x, y
    case.check(t, ["d"], ["gain"], added)

    def summed(get, early):
        y, x = out(), t["x"].clone()
        d, gain, bias = get("d", "gain", "bias")
        ops.sum_layernorm(x, [d], gain, bias, 1e-6, y, early=early)
        return x, y
    case.check(t, ["d"], ["gain", "bias"], summed)

    def over_streams(get, early):
        y, x = out(), t["streams"].clone()
        d, mix, spread, gather, gain, bias, scale = get("d", "mix", "spread", "gather", "gain", "bias", "scale")
        ops.stream_norm(x, None, d, mix, spread, gather, gain, bias, 1e-6, y, delta_scale=scale, early=early)
        return x, y
    case.check(t, ["d"], ["mix", "spread", "gather", "gain", "bias", "scale"], over_streams)

    def gated(get, early):
        y = out()
        x, proj, gain = get("x", "proj", "gain")
        return (ops.gated_rmsnorm(x, proj, 64, gain, 1e-6, y, early=early),)
    case.check(t, ["x", "proj"], ["gain"], gated)

    def state_space(get, early):
        y = out()
        x, act, proj, skip, gain = get("x", "act", "proj", "skip", "gain")
        return (ops.ssd_gate_norm(x, act, proj, 0, skip, gain, y, 64, 1, 1e-6, early=early),)
    case.check(t, ["x", "act", "proj"], ["skip", "gain"], state_space)


def test_preparations_of_single_tokens():
    from from_scratch_inference_engine_b200.kernels import ops
    case, items, heads, vdim, taps = Case(2), 4, 8, 64, 4
    inner = heads * vdim
    channels = inner + 256
    t = dict(proj=case.rand(items, inner + channels + heads), state=case.rand(items, 3 * channels), conv=case.rand(channels, taps),
             conv_b=case.rand(channels), dt_bias=case.rand(heads), a_log=case.rand(heads))
    t["conv_t"] = t["conv"].t().contiguous()
    lists = (ints(list(range(items))), ints([1] * items), ints([2, 0, 3, 1]), items)

    def state_space(get, early):
        state, act, decay = t["state"].clone(), torch.zeros(items, channels + inner, device="cuda"), torch.zeros(items, heads, device="cuda")
        proj, conv_t, conv_b, dt_bias, a_log = get("proj", "conv_t", "conv_b", "dt_bias", "a_log")
        ops.ssd_prep(proj, inner, inner + channels, *lists, state, 0, t["conv"], conv_b, dt_bias, a_log, heads, vdim, act, decay,
                     conv_wt=conv_t, move_tails=True, one_each=True, early=early)
        return state, act, decay
    case.check(t, ["proj"], ["conv_t", "conv_b", "dt_bias", "a_log"], state_space)

    width = 8 * 128 + 2 * 256
    t = dict(proj=case.rand(items, width), conv=case.rand(width, taps), q_gain=case.rand(1024), k_gain=case.rand(256),
             table=case.rand(64, 128), tails=case.rand(items, taps - 1, width))
    error = ints([0])

    def rows(get, early):
        tails, pages, q = t["tails"].clone(), torch.zeros(4, 2 * 2 * 16 * 128, device="cuda"), torch.zeros(items, 1024, device="cuda")
        pos0, slot_of = ints([5, 9, 0, 33]), ints([3, 20, 40, 60])
        proj, conv, q_gain, k_gain, table = get("proj", "conv", "q_gain", "k_gain", "table")
        ops.conv_norm_rotate(proj, items, lists[0], pos0, lists[2], tails, conv, taps, q_gain, k_gain, table, 128,
                             slot_of, pages[:, :4096], pages[:, 4096:], pages.stride(0), 16, q, 8, 2, 128, 128, True,
                             1e-6, error, lists[1], one_each=True, early=early)
        return tails, pages, q
    case.check(t, ["proj"], ["conv", "q_gain", "k_gain", "table"], rows)


# one token each (the kernel for that) and a longer portion (the walk)
@pytest.mark.parametrize("counts", [(1, 1, 1), (1, 9, 2)])
def test_scans(counts):
    from from_scratch_inference_engine_b200.kernels import ops
    case, heads, dim, vdim, tokens, items = Case(3), 4, 64, 64, sum(counts), len(counts)
    t = dict(proj=case.rand(tokens, heads * (2 * dim + vdim)), state=case.rand(4, heads, dim, vdim), decay=torch.rand(heads, device="cuda"))
    starts = [sum(counts[:i]) for i in range(items)]

    def call(get, early):
        out, kept = torch.full((tokens, heads * vdim), float("nan"), device="cuda"), t["state"].clone()
        lists = ints(starts), ints(list(counts)), ints([2, 0, 3])
        proj, state, decay = get("proj", "state", "decay")
        if state is t["state"]:
            state = kept
        ops.lightning_scan(proj, 0, heads * dim, 2 * heads * dim, *lists, items, state, decay, out, heads, dim, vdim, silu=True, early=early)
        return out, state
    case.check(t, ["proj"], ["state", "decay"], call)


def attention_inputs(case, dtype, kv_heads, dim, page, contexts, total_late):
    """Pages whose last ones hold every request's newest keys: what a launch of cast_rows over `total_late` elements ends with."""
    per_page = 2 * kv_heads * page * dim
    old = [[] for _ in contexts]
    count = 0
    for i, n in enumerate(contexts):
        for _ in range((n - 1) // page):
            old[i].append(count)
            count += 1
    pages_total = -(-(count * per_page + total_late) // per_page)
    pages = torch.empty(pages_total * per_page, device="cuda", dtype=dtype)
    pages[:count * per_page] = case.rand(count * per_page).to(dtype)
    newest = case.rand(len(contexts) * per_page).to(dtype)
    tables = torch.full((len(contexts), max(len(o) for o in old) + 1), -1, dtype=torch.int32)
    for i, o in enumerate(old):
        row = o + [pages_total - len(contexts) + i]
        tables[i, :len(row)] = torch.tensor(row, dtype=torch.int32)
    return pages, newest, tables.cuda(), per_page


# a first tile of older keys only, one with the newest among them, a request of one token; keys in one block and split
@pytest.mark.parametrize("nsplit", [1, 3])
@pytest.mark.parametrize("form", ["float32", "mma_few", "auto"])
def test_attention(form, nsplit):
    from from_scratch_inference_engine_b200.kernels import ops
    case, heads, kv_heads, dim, page = Case(4), 8, 2, 64, 16
    dtype = F32 if form == "float32" else BF16
    contexts = (200, 10, 97, 1)
    pages, newest, tables, per_page = attention_inputs(case, dtype, kv_heads, dim, page, contexts, 24 * STRIDE)
    half = per_page // 2
    k_pages, v_pages = pages.view(-1, per_page)[:, :half], pages.view(-1, per_page)[:, half:]
    items = len(contexts)
    q = case.rand(items, heads * dim, dtype=dtype)
    lists = ints(list(range(items))), ints([1] * items), ints([n - 1 for n in contexts])
    tile_item, tile_row0, scale, error = ints(list(range(items))), ints([0] * items), torch.full((heads,), 0.125, device="cuda"), ints([0])

    def call(q, early):
        out = torch.full((items, heads * dim), float("nan"), device="cuda", dtype=dtype)
        parts = [torch.full((nsplit * items * heads * n,), float("nan"), device="cuda") for n in (dim, 2)] if nsplit > 1 else [None, None]
        torch.cuda.synchronize()
        return lambda: (ops.attention_generic(
            q, q.stride(0), k_pages, v_pages, per_page, page, tables, tile_item, tile_row0, items, *lists, out, items, heads, kv_heads,
            dim, 0, 0.125, nsplit, *parts, rows16=True, early=early) if dtype is F32 else ops.scaled_attention(
            q, q.stride(0), scale, k_pages, v_pages, per_page, page, dim, dim, False, tables, tile_item, tile_row0, items, *lists,
            tile_item, out, items, heads, kv_heads, 0, error, nsplit, *parts, form=form, early=early))

    pages[-newest.numel():] = newest
    want = call(q, False)()
    assert not torch.isnan(want).any()
    # the queries late
    late = torch.full((24 * STRIDE,), float("nan"), device="cuda", dtype=dtype)
    source = torch.zeros(24 * STRIDE, device="cuda")
    source[-q.numel():] = q.flatten().float()
    go = call(late[-q.numel():].view_as(q), True)
    ops.cast_rows(source, late)
    assert torch.equal(go(), want)
    # the newest keys late
    source.zero_()
    source[-newest.numel():] = newest.float()
    pages[-24 * STRIDE:].fill_(float("nan"))
    go = call(q, True)
    ops.cast_rows(source, pages[-24 * STRIDE:])
    assert torch.equal(go(), want)
    # without `early` all keys may be that new: the older ones as well, by a launch over all pages
    everything = pages.float().clone()
    pages.fill_(float("nan"))
    go = call(q, False)
    ops.cast_rows(everything, pages)
    assert torch.equal(go(), want)


@pytest.mark.parametrize("nsplit", [1, 2])
def test_mixed_heads(nsplit):
    from from_scratch_inference_engine_b200.kernels import ops
    case, heads, kv_heads, dim, page = Case(5), 8, 2, 64, 16
    pages = case.rand(16, 2 * kv_heads * page * dim)
    tables = torch.arange(16, dtype=torch.int32, device="cuda").view(2, 8)
    t = dict(q=case.rand(2, heads * dim), talk=case.rand(heads, heads))
    half, one, error = kv_heads * page * dim, ints([0, 1]), ints([0])

    def call(get, early):
        out = torch.full((2, heads * dim), float("nan"), device="cuda")
        stats, parts = torch.empty(2 * nsplit * 128, device="cuda"), torch.empty(nsplit * 2 * heads * dim, device="cuda")
        zero, qlen, pos0 = ints([0, 0]), ints([1, 1]), ints([110, 3])
        q, talk = get("q", "talk")
        ops.talking_attention(q, pages[:, :half], pages[:, half:], 2 * half, page, tables, one, zero, 2, one, qlen, pos0, one, talk, out,
                              heads, kv_heads, dim, dim, 0, 0, 1, 0.125, error, nsplit, stats if nsplit > 1 else None,
                              parts if nsplit > 1 else None, early=early)
        return (out,)
    case.check(t, ["q"], ["talk"], call)


def test_lists_of_the_second_product():
    """Without `early` the lists may be the last launch's."""
    from from_scratch_inference_engine_b200.kernels import ops
    case, experts, top, tokens, hidden, inner = Case(6), 64, 6, 8, 512, 256
    pairs, tile = tokens * top, ops.moe_few_tile_rows()
    w, act = case.rand(experts, hidden, inner, dtype=BF16), case.rand(pairs, inner, dtype=BF16)
    ids = torch.stack([torch.randperm(experts)[:top] for _ in range(tokens)]).int().cuda()
    outs = []
    for wait in (True, False):
        room = torch.zeros(ops.moe_lists_size(pairs, experts, tile), dtype=torch.int32, device="cuda")
        out = torch.full((pairs, hidden), float("nan"), device="cuda", dtype=BF16)
        torch.cuda.synchronize()
        lists = ops.moe_align(ids, pairs, experts, room, tile)
        if wait:
            torch.cuda.synchronize()
        outs.append(ops.moe_product(act, w, out, lists, pairs, top, False, tile=tile))
    assert torch.equal(*outs) and not torch.isnan(outs[0]).any()
