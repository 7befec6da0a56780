"""Which float32 products go to the tensor cores: the rule on sizes, without a GPU."""

import pytest

from from_scratch_inference_engine_b200.engine.runtime import f32_split_pays


@pytest.mark.parametrize("rows,n,k,split", [
    # few rows: FFMA up to 16, then only against enough columns and a k over which the error is no larger
    (1, 17920, 1536, False), (16, 151936, 1536, False), (17, 17920, 1536, True), (48, 17920, 1536, True),
    (17, 4096, 4096, False), (48, 1536, 8960, False), (17, 17920, 508, False), (48, 17920, 512, True),
    # many rows: a short k stays with FFMA, which is one launch and sums as exactly
    (49, 192, 192, True), (49, 64, 16, False), (2048, 64, 16, False), (2048, 1024, 96, False), (49, 16, 128, True),
    (2048, 4096, 48, True), (2048, 4096, 32, False), (300, 16384, 48, True), (49, 16384, 64, False), (8192, 8192, 4, False),
    (1668, 1536, 8960, True), (49, 37888, 3584, True)])
def test_route(rows, n, k, split):
    assert f32_split_pays(rows, n, k, 148) is split
