"""GLS covariance, Cholesky factor and whitened fit at matrix sizes around the
factorisation's panels of 8 columns and the warps' 32 (lags 24 to 72), against
the FP64 oracle; tolerances of the GLS parity tests."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import _lib, engine
from tests.helpers import FIT_TOL, run_both
from tests.synth import brownian_stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [2, 3, 4, 5, 6, 7, 8])
def test_matrix_sizes_match_oracle(q):
    st = brownian_stack(6, 5, 9000, seed=61, density=3.0, cps=1e5)
    cfg = engine.FCSConfig(width=6, height=5, frames=9000, background=100, q=q, gls=True)
    gpu, ref = run_both(st, cfg)
    np.testing.assert_array_equal(gpu["blocked_ind"], ref["blocked_ind"])
    n1 = cfg.chanum - 1
    g, r = gpu["covmats"].reshape(-1, n1, n1), ref["covmats"].reshape(-1, n1, n1)
    fin = np.isfinite(r).all(axis=(1, 2))
    assert fin.sum() >= 15
    scale = np.abs(r[fin]).max(axis=(1, 2), keepdims=True)
    assert np.max(np.abs(g[fin] - r[fin]) / scale) <= 1e-4
    if q < 5:
        return                # lag times too short for the fit to be determined at FIT_TOL
    both = (gpu["fitted"] == 1) & (ref["fitted"] == 1)
    assert both.sum() >= 0.8 * (ref["fitted"] == 1).sum()
    for i in (0, 1):
        err = np.abs(gpu["fitres"][both, i] / ref["fitres"][both, i] - 1)
        assert both.sum() == 0 or err.max() <= FIT_TOL, (i, err.max())


def test_covariances_with_non_finite_lags_repeat():
    """Pixels most of whose lags are not finite (a polynomial bleach curve
    through zero) get the same covariance entries whatever ran before them."""
    w = h = 40
    st = brownian_stack(w, h, 6000, seed=5, density=3.0, cps=1e5)
    t = np.arange(6000)[:, None, None] / 6000.0
    st = (100 + (st - 100.0) * np.maximum(0.0, 1.0 - 1.1 * t)).astype(np.uint16)
    cfg = engine.FCSConfig(width=w, height=h, frames=6000, background=100, gls=True, bleach=_lib.BLEACH_POLYNOMIAL,
                           poly_order=5)
    bright = engine.FCSConfig(width=w, height=h, frames=6000, background=100, gls=True)
    first = engine.run_host(st, cfg)["covmats"]
    assert not np.isfinite(first).all()
    for _ in range(3):
        engine.run_host(st, bright)
        np.testing.assert_array_equal(engine.run_host(st, cfg)["covmats"], first)


def test_exported_covariances_are_copied_whole():
    """The covariance leaves before the factorisation overwrites it in place,
    whatever order a block's warps run in: with the GPU full every matrix is
    symmetric bit for bit (the two copies of an entry are read by different
    threads) and equals the one of a small grid over the same pixels."""
    w, h, rows = 64, 48, 2
    st = engine.simulate(w, h, 5000, steps_per_frame=1, density=4.0, seed=7)
    outs = []
    for kw in ({}, {"map_y0": 20, "out_h": rows}):
        plan = engine.Plan(engine.FCSConfig(width=w, height=h, frames=5000, background=100, gls=True, do_fit=False, **kw))
        o = plan.alloc_device_outputs()
        plan.execute(st, o)
        outs.append(o["covmats"].cpu().numpy())
    full, part = outs
    assert np.isfinite(full).all(axis=(1, 2)).sum() >= 0.9 * w * h
    np.testing.assert_array_equal(full, full.transpose(0, 2, 1))
    np.testing.assert_array_equal(full.reshape(h, w, *full.shape[1:])[20:20 + rows].reshape(part.shape), part)
