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
