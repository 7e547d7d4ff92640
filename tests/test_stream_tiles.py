"""GPU parity of the streaming pass at the edges of its tiles and boxes: rows
that are not whole TMA granules (word-aligned copies, one run per frame where
the tile is as wide as the frame), outputs wider than a tile, windows whose
column sums are staged, displaced windows on either side, frame counts that
end inside a box.  Checked against the FP64 oracle: block index and flag
exactly, finiteness per lag exactly, the ACF within the correlator tests'
tolerance (the blocked variance of these short stacks has one or two blocks
at the top lags and says nothing about the streaming pass)."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import _lib, engine
from tests.helpers import ACF_TOL, acf_deviation, run_both
from tests.synth import bleach_stack, brownian_stack

pytestmark = pytest.mark.gpu


def check(gpu, ref):
    np.testing.assert_array_equal(gpu["blocked_ind"], ref["blocked_ind"])
    np.testing.assert_array_equal(gpu["blocked_ok"], ref["blocked_ok"])
    np.testing.assert_array_equal(np.isfinite(gpu["acf"]), np.isfinite(ref["acf"]))
    assert acf_deviation(gpu, ref) <= ACF_TOL


@pytest.mark.parametrize("w,h,frames,kw", [
    (21, 9, 2500, {}),
    (129, 2, 2305, {}),
    (264, 2, 2304, {}),
    (23, 12, 2400, {"binx": 5, "biny": 5, "pixbinx": 1, "pixbiny": 1}),
    (41, 17, 2311, {"binx": 3, "biny": 4, "pixbinx": 2, "pixbiny": 3, "cfx": 2, "cfy": 1}),
    (40, 24, 2400, {"binx": 5, "biny": 5, "pixbinx": 5, "pixbiny": 5}),
    (24, 16, 2400, {"binx": 3, "biny": 3, "pixbinx": 1, "pixbiny": 1, "cfx": -2, "cfy": -1, "map_x0": 2, "map_y0": 1,
                    "out_w": 18, "out_h": 11}),
    (19, 11, 2700, {"first": 133, "num": 2431, "cfx": 1, "cfy": -1, "map_y0": 1, "out_h": 9}),
], ids=["run21", "tiles129", "tiles264", "cols-odd", "cols-odd-ccf", "cols-step5", "cols-ccf-neg", "run-range"])
def test_tiles_no_bleach(w, h, frames, kw):
    st = brownian_stack(w, h, frames, seed=21, density=2.0, cps=3e4)
    cfg = engine.FCSConfig(width=w, height=h, frames=frames, background=100, do_fit=False, **kw)
    gpu, ref = run_both(st, cfg)
    check(gpu, ref)


@pytest.mark.parametrize("order", [3, 4, 7, 8])
def test_padded_basis_rows(order):
    # order + 1 below, at and above a whole float4
    st = bleach_stack(13, 6, 2600, seed=22, fluct=0.05)
    cfg = engine.FCSConfig(width=13, height=6, frames=2600, background=100, do_fit=False, q=6,
                           bleach=_lib.BLEACH_POLYNOMIAL, poly_order=order)
    gpu, ref = run_both(st, cfg)
    check(gpu, ref)
