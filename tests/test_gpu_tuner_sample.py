"""The BSE tuner times the FP64 kernel that the whole list runs, not one with more threads for a shorter list."""

import dataclasses

import pytest

pytestmark = pytest.mark.gpu


def test_sample_fills_the_device():
    """The sample is as long as the list or fills the SMs' threads with CTAs of one warp, the smallest there are."""
    import torch

    from dgamore_b200 import autotune, synthetic
    from dgamore_b200.pipeline import LadderPass

    cfg = dataclasses.replace(synthetic.CONFIGS["c1"], nk=(16, 16, 1), niw=30, niv=20, niv_shell=0)
    lp = LadderPass(synthetic.make_inputs(cfg))
    lp.pre_bse()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sample = autotune.tune_bse(lp, force=True).sample_items
    assert sample == lp.n_items or sample * 32 > sms * 256
