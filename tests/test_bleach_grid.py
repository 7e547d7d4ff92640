"""Start of the single-exponential bleach fit: eight and two traces per block
give the same parameters bit for bit, at trace counts around the blocks and
trace lengths around the 32 points of a row."""
import numpy as np
import pytest
import torch

from imaging_fcs_1_52_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


def bleach_params(stack):
    t, h, w = stack.shape
    cfg = engine.FCSConfig(width=w, height=h, frames=t, background=100, bleach=_lib.BLEACH_SINGLE_EXP, do_fit=False, q=2)
    plan = engine.Plan(cfg)
    plan.execute(torch.from_numpy(stack.view(np.int16)).cuda(), plan.alloc_device_outputs())
    torch.cuda.synchronize()
    return np.asarray(plan.bleach_params()).reshape(h, w, -1)


@pytest.mark.parametrize("frames", [200, 255, 257, 999, 1000, 1031, 2500])
def test_eight_and_two_traces_per_block_agree(frames):
    w, h = 53, 46                                 # 2,438 traces: eight per block
    rng = np.random.default_rng(frames)
    rate = np.exp(rng.uniform(-1.0, 2.5, (h, w)))
    t = (np.arange(frames) + 0.5) / frames
    mean = 200.0 * np.exp(-rate * t[:, None, None]) + 30.0
    stack = (100 + rng.poisson(mean)).astype(np.uint16)
    stack[:, 0, 1] = 100                          # an empty trace
    big = bleach_params(stack)
    assert np.isfinite(big[2:, :, 12]).all()
    for rows, cols in ((1, 1), (1, 2), (3, 1), (5, 53)):
        small = bleach_params(np.ascontiguousarray(stack[:, :rows, :cols]))
        np.testing.assert_array_equal(small.view(np.int32), big[:rows, :cols].view(np.int32))
    # the fitted rate (parameter 5, 1/s) against the truth where the curve bends within the trace
    sel = (rate > 1.0) & (np.arange(h)[:, None] > 0)
    rel = big[..., 5][sel] * (frames * cfg_frametime()) / rate[sel] - 1
    assert np.median(np.abs(rel)) <= 0.1


def cfg_frametime():
    return engine.FCSConfig(width=1, height=1, frames=100).frametime
