"""Polynomial bleach fit of every order, at trace lengths around a warp's rows;
fits with one, two and three free parameters (the epilogue has the usual counts
at compile time, the others at run time)."""
import numpy as np
import pytest
import torch

import oracle
from imaging_fcs_1_52_gb300 import _lib, engine
from tests.helpers import run_both
from tests.synth import brownian_stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("frames", [300, 1000, 3100])
def test_coefficients_match_least_squares(order, frames):
    """Legendre coefficients against an FP64 least-squares fit of the averaged
    trace (whole numbers: the mean is truncated, as the oracle's is).  Bound: the trace's FP32 rounding (2^-24 of its largest value) times
    a projection row's sum of magnitudes (below 1.3 (2 order + 1)), and the
    coefficient's own rounding: below 2e-6 of the largest value."""
    st = brownian_stack(5, 4, frames, seed=order, density=6.0, cps=1e5)
    cfg = engine.FCSConfig(width=5, height=4, frames=frames, background=100, q=3, do_fit=False,
                           bleach=_lib.BLEACH_POLYNOMIAL, poly_order=order)
    plan = engine.Plan(cfg)
    plan.execute(torch.from_numpy(st.view(np.int16)).cuda(), plan.alloc_device_outputs())
    torch.cuda.synchronize()
    got = np.asarray(plan.bleach_params())[:, :order + 1].astype(np.float64)
    n = min(frames, 1000)
    y = np.stack([oracle.intensity_trace(st, p % 5, p // 5, bckg=100)[0] for p in range(20)], axis=1)
    want = np.polynomial.legendre.legfit(np.linspace(-1.0, 1.0, n), y, order).T
    assert np.max(np.abs(got - want) / np.abs(y).max(axis=0)[:, None]) <= 2e-6


@pytest.mark.parametrize("free", [(1, 0, 0), (1, 1, 0), (1, 1, 1)], ids=["N", "ND", "NDG"])
def test_free_parameter_counts_match_oracle(free):
    st = brownian_stack(6, 4, 6000, seed=3, density=3.0, cps=1e5)
    mask = (free[0], free[1], 0, 0, free[2]) + (0,) * 6
    cfg = engine.FCSConfig(width=6, height=4, frames=6000, background=100, free_mask=mask)
    gpu, ref = run_both(st, cfg)
    np.testing.assert_array_equal(gpu["fitted"], ref["fitted"])
    both = gpu["fitted"] == 1
    assert both.sum() >= 12
    np.testing.assert_allclose(gpu["fitres"][both][:, 0], ref["fitres"][both][:, 0], rtol=1e-4)
