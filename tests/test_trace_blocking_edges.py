"""Averaged trace and blocking transform at their edges, against the FP64
oracle: raw sums by 16-byte, 4-byte and 2-byte loads, a region narrow enough
for the one-pass trace, binned and displaced windows of the raw sums, frame
counts around a blocking segment's and a sixteen-product step's end, and
recordings whose upper blocking levels span 2 to 32 segments.  Tolerances of
the correlator's parity tests."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import _lib, engine
from tests.helpers import ACF_TOL, acf_deviation, run_both
from tests.synth import bleach_stack
from tests.test_gpu_correlator import check_acf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,frames,kw", [
    (16, 3, 4000, {}),
    (10, 3, 4000, {}),
    (9, 5, 4321, {}),
    (16, 4, 4000, {"first": 3, "num": 3500, "map_y0": 1, "out_h": 2}),
    (40, 4, 4000, {"map_x0": 7, "out_w": 6}),
    (22, 9, 4000, {"binx": 3, "biny": 2, "pixbinx": 1, "pixbiny": 2, "cfx": 1, "cfy": -1, "map_y0": 1, "out_h": 3}),
], ids=["vec8", "vec2", "vec1", "vec8-rows", "narrow", "windows-ccf"])
def test_trace_forms(w, h, frames, kw):
    # the polynomial correction makes every output depend on the trace
    st = bleach_stack(w, h, frames, seed=51, fluct=0.05)
    cfg = engine.FCSConfig(width=w, height=h, frames=frames, background=100, do_fit=False,
                           bleach=_lib.BLEACH_POLYNOMIAL, poly_order=4, **kw)
    gpu, ref = run_both(st, cfg)
    np.testing.assert_array_equal(gpu["blocked_ind"], ref["blocked_ind"])
    np.testing.assert_array_equal(np.isfinite(gpu["acf"]), np.isfinite(ref["acf"]))
    assert acf_deviation(gpu, ref) <= ACF_TOL


@pytest.mark.parametrize("frames,kw", [(4097, {}), (4098, {}), (4112, {"cfx": 1}), (4113, {}), (4353, {}), (17000, {}),
                                       (33025, {})])
def test_blocking_edges(frames, kw):
    st = bleach_stack(5, 4, frames, amp=300.0, tau1=1e6, frac2=0.0, corr_frames=6.0, seed=52)
    cfg = engine.FCSConfig(width=5, height=4, frames=frames, background=100, do_fit=False, **kw)
    gpu, ref = run_both(st, cfg)
    check_acf(gpu, ref)
