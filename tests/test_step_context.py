"""What a step's context says of its requests' lengths (no GPU needed)."""
import types

import numpy as np
import pytest
import torch

from from_scratch_inference_engine_b200.engine.context import StepContext


class Ring:
    def stage(self, host, device, out=None):
        return torch.from_numpy(host.copy())


# as many tokens as requests is not one token each
@pytest.mark.parametrize("q_len,one_each", [((1, 1, 1), True), ((2, 0, 1), False), ((0, 2), False), ((1, 4), False)])
def test_one_token_each(q_len, one_each):
    starts, pos0 = [sum(q_len[:i]) for i in range(len(q_len))], [5 + 10 * i for i in range(len(q_len))]
    ctx = StepContext(types.SimpleNamespace(device="cpu"), Ring(), {}, None, [0] * sum(q_len), starts, q_len, pos0,
                      list(range(len(q_len))), [(4, [list(range(8)) for _ in q_len])])
    assert ctx.one_each is one_each
    want = np.concatenate([np.arange(p, p + n) for p, n in zip(pos0, q_len)])
    assert ctx.positions.tolist() == want.tolist()
