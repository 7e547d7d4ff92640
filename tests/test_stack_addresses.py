"""A uint16 stack at any address: 16-byte aligned (TMA boxes, 16-byte trace
loads), 4-byte (cp.async, 4-byte loads) and 2-byte (plain loads) give the same
bits."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,kw", [
    (24, 10, {"bleach": _lib.BLEACH_SINGLE_EXP}),
    (21, 10, {"bleach": _lib.BLEACH_POLYNOMIAL, "poly_order": 5}),
    (32, 12, {"binx": 2, "biny": 2, "cfx": 2, "bleach": _lib.BLEACH_DOUBLE_EXP}),
    (24, 16, {"binx": 5, "biny": 5, "pixbinx": 1, "pixbiny": 1, "cfy": 1, "first": 3, "num": 4000}),
], ids=["exp", "poly-odd", "bin-ccf-exp2", "overlap-range"])
def test_stack_addresses_give_the_same_bits(w, h, kw):
    import torch
    frames = 4100
    st = engine.simulate(w, h, frames, steps_per_frame=1, density=4.0, cps=1e5, tau_bleach=20.0, seed=9)
    cfg = engine.FCSConfig(width=w, height=h, frames=frames, background=100, **kw)
    plan = engine.Plan(cfg)
    outs = []
    for shift in (0, 2, 1):                   # elements of two bytes
        buf = torch.zeros(st.numel() + 8, dtype=torch.int16, device="cuda")
        view = buf[shift:shift + st.numel()]
        view.copy_(st.view(torch.int16).flatten())
        assert view.data_ptr() % 16 == 2 * shift
        o = plan.alloc_device_outputs()
        plan.execute(view.view(torch.uint16).view(frames, h, w), o)
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    assert np.isfinite(outs[0]["acf"]).all(axis=1).mean() > 0.5
    for o in outs[1:]:
        for k in o:
            np.testing.assert_array_equal(o[k], outs[0][k], err_msg=k)
