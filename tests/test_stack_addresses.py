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


@pytest.mark.parametrize("w,h,kw", [
    (33, 3, {"bleach": _lib.BLEACH_POLYNOMIAL}), (25, 4, {"bleach": _lib.BLEACH_POLYNOMIAL}),
    (101, 1, {"cfx": 1, "bleach": _lib.BLEACH_SINGLE_EXP}), (25, 44, {"out_w": 8}), (43, 9, {"out_w": 14}),
    (5, 16, {"binx": 3, "biny": 1}), (5, 17, {"binx": 3, "biny": 1}), (11, 64, {"binx": 5, "biny": 5, "pixbiny": 1}),
    (21, 20, {"binx": 2, "biny": 3, "pixbinx": 1, "pixbiny": 1, "cfy": 1}),
], ids=["99-pixels", "100-pixels", "one-row-ccf", "third-of-rows", "third-of-rows-2", "16-rows", "17-rows", "narrow-overlap",
        "run-ccf"])
def test_either_side_of_the_staging_rule(w, h, kw):
    """Frames whose rows are not 16-byte aligned are staged by cp.async or read
    with plain loads, by their shape; a stack at an odd address always takes
    the plain loads.  Same bits."""
    import torch
    frames = 2900
    st = engine.simulate(w, h, frames, steps_per_frame=1, density=4.0, cps=1e5, tau_bleach=20.0, seed=9)
    plan = engine.Plan(engine.FCSConfig(width=w, height=h, frames=frames, background=100, do_fit=False, **kw))
    buf = torch.zeros(st.numel() + 1, dtype=torch.int16, device="cuda")
    buf[1:].copy_(st.view(torch.int16).flatten())
    outs = []
    for stack in (st, buf[1:].view(torch.uint16).view(frames, h, w)):
        o = plan.alloc_device_outputs()
        plan.execute(stack, o)
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    for k in outs[0]:
        np.testing.assert_array_equal(outs[1][k], outs[0][k], err_msg=k)
