"""Which products a step's routed rows take: the rule on sizes, without a GPU."""

import pytest
import torch

from from_scratch_inference_engine_b200.parts.routed_experts import streaming_pays


@pytest.mark.parametrize("dtype,pairs,experts,streams", [
    (torch.bfloat16, 48, 64, True), (torch.bfloat16, 768, 64, True),
    (torch.bfloat16, 1020, 64, False), (torch.bfloat16, 1278, 64, False),    # slower where tokens share their experts
    (torch.bfloat16, 320, 16, True), (torch.bfloat16, 322, 16, False), (torch.bfloat16, 1536, 128, True),
    (torch.float32, 2048, 64, True), (torch.float32, 2050, 64, False), (torch.float32, 512, 16, True)])
def test_route(dtype, pairs, experts, streams):
    assert streaming_pays(dtype, pairs, experts) is streams
