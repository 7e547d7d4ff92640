"""Lag-major outputs of calcACF at pixel and lag counts around the 32 x 32
tiles that turn them, against the FP64 oracle."""
import numpy as np
import pytest

import oracle
from imaging_fcs_1_52_gb300._lib import ACFParameters
from imaging_fcs_1_52_gb300.gpufit_imfcs import GpufitImFCS
from tests.helpers import ACF_TOL, acf_deviation
from tests.synth import brownian_stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,q", [(1, 1, 8), (31, 1, 2), (4, 8, 8), (11, 3, 3), (13, 5, 6)])
def test_outputs_are_lag_major(w, h, q):
    raw = brownian_stack(w, h, 3000, seed=w, density=2.0, cps=3e4)
    ch = 17 + 8 * (q - 1)
    p = ACFParameters(width=w, height=h, win_star=w, hin_star=h, w_temp=w, h_temp=h, pixbinX=1, pixbinY=1,
                      binningX=1, binningY=1, firstframe=1, lastframe=3000, framediff=3000, cfXDistance=0,
                      cfYDistance=0, correlatorp=16, correlatorq=q, frametime=1e-3, background=100, chanum=ch,
                      isNBcalculation=0, bleachcorr_gpu=0, bleachcorr_order=0, nopit=1000, ave=3)
    outs = [np.zeros((ch, h, w)), np.zeros((ch, h, w)), np.zeros((h, w)), np.zeros((h, w)), np.zeros((2, h, w))]
    GpufitImFCS.calcACF(raw.astype(np.float32) - 100, *outs, None, np.zeros(ch), np.zeros(ch, np.int32), p)
    ref = oracle.run(raw, out_w=w, out_h=h, background=100, q=q, do_fit=False)
    assert acf_deviation({"acf": outs[0].reshape(ch, -1).T}, ref) <= ACF_TOL
    np.testing.assert_array_equal(outs[4][0].ravel(), ref["blocked_ind"])


@pytest.mark.parametrize("p_corr,q", [(16, 8), (32, 8)])
def test_memory_answer_counts_the_plan(p_corr, q):
    """isACFmemorySufficient turns to no where the input, the outputs (lag-major
    copies too) and the plan's scratch -- affine in the frames up to the
    segments' rounding: 5 % -- reach nine tenths of the free memory."""
    import torch
    from imaging_fcs_1_52_gb300 import engine
    w = h = 512
    ch = p_corr + (q - 1) * p_corr // 2 + 1

    def params(frames):
        return ACFParameters(width=w, height=h, win_star=w, hin_star=h, w_temp=w, h_temp=h, pixbinX=1, pixbinY=1,
                             binningX=1, binningY=1, firstframe=1, lastframe=frames, framediff=frames, cfXDistance=0,
                             cfYDistance=0, correlatorp=p_corr, correlatorq=q, frametime=1e-3, background=100,
                             chanum=ch, isNBcalculation=0, bleachcorr_gpu=0, bleachcorr_order=0, nopit=1000,
                             ave=frames // 1000)

    def need(frames):
        plan = engine.Plan(engine.FCSConfig(width=w, height=h, frames=frames, p=p_corr, q=q, do_fit=False))
        return plan.scratch_bytes + w * h * (frames * 4 + 4 * 8 * ch)

    torch.cuda.empty_cache()
    n1, n2 = need(12000), need(24000)
    free = torch.cuda.mem_get_info()[0]
    per_frame = (n2 - n1) / 12000
    expected = 24000 + (0.9 * free - n2) / per_frame
    lo, hi = 12000, 4 * int(expected)
    assert GpufitImFCS.isACFmemorySufficient(params(lo)) and not GpufitImFCS.isACFmemorySufficient(params(hi))
    while hi - lo > 200:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if GpufitImFCS.isACFmemorySufficient(params(mid)) else (lo, mid)
    assert abs(lo / expected - 1) <= 0.05
