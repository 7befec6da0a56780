"""Host side of sampling: when the kernel for short lists is launched; and that the check which the GPU tests use on
sampled tokens refuses a token beside the right one."""

import numpy as np

from from_scratch_inference_engine_b200.sampling.sampler import SamplingParams, any_short_list
from sampling_ranks import cumulative, kept, ranks


def test_short_lists_are_launched_for_rows_that_have_one():
    random = lambda k: SamplingParams(temperature=0.8, top_k=k, top_p=0.9)
    assert not any_short_list([SamplingParams()], 104)                       # the default: no top_k
    assert not any_short_list([random(0), random(105), random(50000)], 104)
    assert not any_short_list([SamplingParams(temperature=0.0, top_k=40)], 104)
    assert any_short_list([random(0), random(104)], 104) and any_short_list([random(1)], 104)
    assert not any_short_list([], 104)


def test_the_check_refuses_neighbours():
    rng = np.random.default_rng(3)
    refused = passed = 0
    for t in (0.8, 2.0):
        for k in (2, 40, 104):
            for p in (1.0, 0.95, 0.2):
                row = (rng.standard_normal(4096) * 3).astype(np.float32)
                run = cumulative(row, kept(row, k), t)
                want, may = ranks(run, p, rng.random())
                assert want in may
                for beside in (want - 1, want + 1):
                    refused += beside not in may
                    passed += beside in may
    assert passed <= 1 and refused >= 35
