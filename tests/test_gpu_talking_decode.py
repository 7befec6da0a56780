"""Mixed-heads attention and its preparation for steps of one token per request: keys split over blocks and not against
64 bits, and the row in one go against the general kernel, to the bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def device(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


# one key; the edges of a tile of 64 keys and of more tiles than ranges; a window with kept first tokens, kept ones alone; a
# padding entry; one head per key/value head and eight; rows that no 16-byte copy takes; columns that are no multiple of 64 or 32;
# values with a buffer of their own and without; more than 32 ranges
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,page,window,keep,lengths,splits", [
    (16, 4, 128, 128, 16, 1024, 4, (1, 64, 65, 916), 15), (4, 4, 8, 40, 16, 0, 0, (255, 256, 257, 513), 5),
    (8, 1, 72, 24, 8, 100, 3, (1, 99, 103, 700), 2), (6, 2, 252, 90, 32, 33, 64, (63, 200, 0, 32), 3),
    (64, 8, 64, 136, 16, 1, 2, (5, 1, 2, 300), 2), (5, 1, 13, 7, 16, 0, 0, (31, 33, 2600, 40), 41)])
def test_split_over_blocks(heads, kv_heads, dim, vdim, page, window, keep, lengths, splits, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(heads * 100 + dim)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    items, group = len(lengths), heads // kv_heads
    blocks = -(-max(lengths) // page) + 1
    keys, values = rand(items * blocks, kv_heads, page, dim).to(dtype), rand(items * blocks, kv_heads, page, vdim).to(dtype)
    width = kv_heads * page * (dim + vdim)
    pages = torch.cat([keys.flatten(1), values.flatten(1)], dim=1).contiguous()
    k_pages, v_pages = pages[:, :kv_heads * page * dim], pages[:, kv_heads * page * dim:]
    tables = torch.randperm(items * blocks, generator=generator, device="cuda").int().view(items, blocks)
    q, talk = rand(items, heads * dim), rand(heads, heads) * heads ** -0.5
    scale = dim ** -0.5
    pos0, slots = device([max(n - 1, 0) for n in lengths]), device([-1 if n == 0 else i for i, n in enumerate(lengths)])
    qstart, qlen, error = device(list(range(items))), device([1] * items), device([0])
    assert ops.talking_attention_key_tile(heads, kv_heads, dim, vdim, dtype) > 0
    outs = []
    for nsplit in (1, splits):
        out = torch.full((items, heads * vdim), float("nan"), device="cuda", dtype=dtype)
        stats = torch.full((items * nsplit * 128,), float("nan"), device="cuda")
        parts = torch.full((nsplit * items * heads * vdim,), float("nan"), device="cuda")
        ops.talking_attention(q, k_pages, v_pages, width, page, tables, device(list(range(items))), device([0] * items), items,
                              qstart, qlen, pos0, slots, talk, out, heads, kv_heads, dim, vdim, window, keep, 1, scale, error,
                              nsplit, stats if nsplit > 1 else None, parts if nsplit > 1 else None)
        outs.append(out)
    assert int(error.item()) == 0
    for i, n in enumerate(lengths):
        if n == 0:
            assert torch.isnan(outs[0][i]).all()             # a padding entry writes nothing
            continue
        seen = [j for j in range(n) if window == 0 or n - 1 - j < window or j < keep]
        rows = [(int(tables[i, j // page]), j % page) for j in seen]
        k = torch.stack([keys[p, :, s] for p, s in rows]).double()                 # [keys, kv heads, dim]
        v = torch.stack([values[p, :, s] for p, s in rows]).double()
        s = torch.einsum("hd,jhd->hj", q[i].view(heads, dim).double(), k.repeat_interleave(group, 1)) * scale
        mixed = talk.double() @ torch.softmax(s, dim=1)
        want = torch.einsum("hj,jhv->hv", mixed, v.repeat_interleave(group, 1)).flatten()
        size = torch.einsum("hj,jhv->hv", talk.double().abs() @ torch.softmax(s, dim=1), v.abs().repeat_interleave(group, 1)).flatten()
        # 32-bit: a score of dim products moves its weight by dim 2^-24 of the products' sum (up to 64 here), then sums over
        # keys and heads; the result rounded to the storage type
        bound = size * (dim + heads + 64) * 64 * 2.0 ** -24 + (want.abs() + size * 1e-3) * (2.0 ** -8 if dtype is torch.bfloat16 else 0.0)
        for out in outs:
            assert ((out[i].double() - want).abs() <= bound).all()


def test_a_page_that_was_given_back():
    """Its keys count as zeros and the step fails, with keys split over blocks as in one."""
    from from_scratch_inference_engine_b200.kernels import ops
    pages = torch.randn(4, 2 * 8 * 16, device="cuda")
    one, outs = device([0]), []
    for nsplit in (1, 2):
        error, out = device([0]), torch.empty(1, 16, device="cuda")
        ops.talking_attention(torch.ones(1, 16, device="cuda"), pages[:, :128], pages[:, 128:], 256, 16, device([[2, -1, 0, 3]]), one, one,
                              1, one, device([1]), device([60]), one, torch.ones(2, 2, device="cuda"), out, 2, 1, 8, 8, 0, 0, 1, 0.3, error,
                              nsplit, torch.empty(256, device="cuda"), torch.empty(32, device="cuda"))
        assert int(error.item()) == 3
        outs.append(out)
    assert torch.allclose(*outs, rtol=1e-4, atol=1e-5)


# tokens of one request each (tails move in the launch), as many tokens as requests but not one each, and longer portions; before the sequence's start; taps 2 to
# 4 and a count the row form does not take; without keys of its own; a refused position; a padding entry
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,taps,rot,qlens", [
    (16, 4, 128, 128, 4, 128, (1, 1, 1, 1)), (16, 4, 128, 128, 4, 64, (1, 5, 2, 30)), (2, 1, 16, 24, 4, 10, (2, 0, 1, 1)), (2, 1, 16, 24, 2, 10, (1, 1, 1, 1)),
    (3, 1, 40, 8, 3, 0, (1, 1, 3, 1)), (4, 2, 8, 8, 5, 4, (1, 1, 1, 1)), (4, 0, 24, 8, 4, 24, (1, 1, 1, 1))])
def test_rows_in_one_go(heads, kv_heads, dim, vdim, taps, rot, qlens, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(dim + taps)
    rand = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    has_kv, kvh, page, items = kv_heads > 0, max(kv_heads, 1), 16, len(qlens)
    width = heads * dim + (kvh * (dim + vdim) if has_kv else 0)
    tokens, starts = sum(qlens), [sum(qlens[:i]) for i in range(items)]
    pos0 = [0, 1, 40, 7]
    slots = [2, 0, -1, 3]
    proj, conv_w, q_gain, k_gain = rand(tokens, width).to(dtype), rand(width, taps), rand(heads * dim), rand(kvh * dim)
    tails = rand(5, taps - 1, width)
    tails[2], tails[0, :-1] = 0.0, 0.0                        # nothing before the sequence starts
    table = rand(64, max(rot, 1))
    error = device([0])
    pages = torch.zeros(8, kvh * page * (dim + vdim), device="cuda", dtype=dtype)
    slot_of = device([16 * i + 3 if i != 1 else -1 for i in range(tokens)]) if tokens <= 8 else device([-1] * tokens)

    def run(proj, pages, tails, qlen):
        q = torch.full((tokens, heads * dim), float("nan"), device="cuda")
        ops.conv_norm_rotate(proj, items, device(starts), device(pos0), device(slots), tails, conv_w, taps, q_gain,
                             k_gain if has_kv else None, table, rot, slot_of if has_kv else None,
                             pages[:, :kvh * page * dim] if has_kv else None, pages[:, kvh * page * dim:] if has_kv else None,
                             pages.stride(0), page, q, heads, kv_heads, dim, vdim, has_kv, 1e-6, error, qlen,
                             one_each=qlen is not None and set(qlens) == {1})
        return q
    got_pages, got_tails = pages.clone(), tails.clone()
    got = run(proj, got_pages, got_tails, device(list(qlens)))
    # the general kernel takes what does not start on 16 bytes: the same projection four bytes further on
    shifted = torch.empty(proj.numel() + 8, device="cuda", dtype=dtype)[8 // proj.element_size() // 2:][:proj.numel()].view_as(proj)
    shifted.copy_(proj)
    assert shifted.data_ptr() % 16
    want_pages, want_tails = pages.clone(), tails.clone()
    want = run(shifted, want_pages, want_tails, None)
    ops.conv_tails(proj, device(starts), device(list(qlens)), device(slots), items, want_tails, taps)
    assert torch.equal(got_tails, want_tails) and int(error.item()) == 0
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got.nan_to_num(7e7), want.nan_to_num(7e7)) and torch.equal(got_pages, want_pages)
    run(proj, got_pages, got_tails, None)
    assert int(error.item()) == 0
    pos0[3] = 64                                              # beyond the table
    run(proj, got_pages, got_tails, None)
    assert int(error.item()) == (2 if rot else 0)


@pytest.mark.parametrize("width", [3, 264, 1000, 2048, 2049, 4096, 4097])
@pytest.mark.parametrize("dtype", DTYPES)
def test_layer_norm_rows(width, dtype):
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(width)
    src, gain, x = (torch.randn(shape, generator=generator, device="cuda") * 3 + 1.5 for shape in ((5, width), (width,), (5, width)))
    norm = lambda v: torch.nn.functional.layer_norm(v.double(), (width,), eps=1e-6) * gain.double()
    rows, half = device([4, 0, 2]), 2.0 ** -8 if dtype is torch.bfloat16 else 0.0
    want = norm(src)[rows.long()]
    got = ops.layernorm_rows(src, gain, 1e-6, torch.empty(3, width, device="cuda", dtype=dtype), rows=rows)
    assert ((got.double() - want).abs() <= (1e-5 + half) * (1 + want.abs())).all()
    delta, copy, sum_ = src.to(dtype), torch.empty(5, width, device="cuda", dtype=dtype), x.clone()
    ops.add_layernorm(sum_, delta, gain, 1e-6, copy)
    want = x.double() + norm(delta)
    assert ((sum_.double() - want).abs() <= 1e-5 * (1 + want.abs())).all()      # the sum stays 32-bit
    assert torch.equal(copy, sum_.to(dtype))


# every number of values a thread, one to eight, with each number of threads; rows that end inside
@pytest.mark.parametrize("width", [3, 130, 264, 500, 512, 700, 1024, 1025, 1300, 1700, 2000, 2048, 2049, 4096])
@pytest.mark.parametrize("dtype", DTYPES)
def test_layer_norm_rows_are_the_general_kernels(width, dtype):
    """The row in registers leaves the bits of the kernel for rows of any width."""
    from from_scratch_inference_engine_b200.kernels import ops
    generator = torch.Generator(device="cuda").manual_seed(width)
    src, gain, x = (torch.randn(shape, generator=generator, device="cuda") * 3 + 1.5 for shape in ((40, width), (width,), (40, width)))
    results = []
    for general in (False, True):
        y, copy = (torch.full((40, width), float("nan"), device="cuda", dtype=dtype) for _ in range(2))
        sum_ = x.clone()
        ops.layernorm_rows(src, gain, 1e-6, y, general=general)
        ops.add_layernorm(sum_, src.to(dtype), gain, 1e-6, copy, general=general)
        results.append((y, sum_, copy))
    assert all(torch.equal(a, b) for a, b in zip(*results))
