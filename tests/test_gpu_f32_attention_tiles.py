"""float32 attention of prompts in tiles of 32 rows x 64 keys: contexts, portions and windows at the edges of both."""

import pytest
import torch

from test_gpu_kernels import PagedCase, assert_rows_close, ops  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,window,nsplit", [(6, 1, 0, 1), (4, 4, 64, 1), (12, 2, 65, 3), (7, 1, 0, 2)])
def test_tiles(ops, hd, heads, kv_heads, window, nsplit):  # noqa: F811
    items = [(0, 63), (0, 64), (0, 65), (63, 2), (127, 33), (64, 1), (190, 31)]
    case = PagedCase(torch.float32, heads, kv_heads, hd, 8, items, window=window, seed=hd + window)
    assert_rows_close(case.run(ops, nsplit), case.want, case, torch.float32)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,window,nsplit", [(2, 2, 0, 1), (6, 1, 0, 1), (12, 2, 40, 1), (7, 1, 0, 2)])
def test_values_that_a_row_does_not_see(ops, hd, heads, kv_heads, window, nsplit):  # noqa: F811
    """An infinite value and a NaN key of the last token reach none of the rows before it."""
    new = 140
    case = PagedCase(torch.float32, heads, kv_heads, hd, 8, [(0, new)], window=window, seed=hd)
    want = case.run(ops, nsplit)
    page, offset = int(case.tables[0, (new - 1) // 8]), (new - 1) % 8
    case.pages[page, 0, 0, :, offset] = float("nan")
    case.pages[page, 0, 1, :, offset] = float("inf")
    got = case.run(ops, nsplit)
    assert torch.equal(got[:-1], want[:-1])
    assert not torch.isfinite(got[-1]).any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,rows16", [(64, False), (128, True), (96, False)])
def test_more_splits_than_the_merge_stages(ops, hd, rows16, dtype):  # noqa: F811
    """4,096 splits' maxima and sums fit the merge's shared memory; it takes more, with the same bits (each split has a tile or none)."""
    case = PagedCase(dtype, 4, 2, hd, 8, [(300, 1), (0, 3)], seed=hd)
    most, more = (case.run(ops, nsplit, rows16 and dtype is torch.float32) for nsplit in (4096, 4097))
    assert_rows_close(more, case.want, case, dtype)
    assert torch.equal(most, more)
