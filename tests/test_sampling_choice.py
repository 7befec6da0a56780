"""Host side of sampling: when the kernel for short lists is launched."""

from from_scratch_inference_engine_b200.sampling.sampler import SamplingParams, any_short_list


def test_short_lists_are_launched_for_rows_that_have_one():
    random = lambda k: SamplingParams(temperature=0.8, top_k=k, top_p=0.9)
    assert not any_short_list([SamplingParams()], 104)                       # the default: no top_k
    assert not any_short_list([random(0), random(105), random(50000)], 104)
    assert not any_short_list([SamplingParams(temperature=0.0, top_k=40)], 104)
    assert any_short_list([random(0), random(104)], 104) and any_short_list([random(1)], 104)
    assert not any_short_list([], 104)
