"""Averaged trace of binned windows, by every form it takes: sums of a window's
rows by 16-, 4- and 2-byte loads, in one part and in several (a recording's
level-0 stream holds fewer sums than its points), windows with gaps, a frame
range and displaced columns, overlapping windows, and the one-pass kernel for
few frames a point.  The centre a plan without bleach correction subtracts is
the mean of the trace: against numpy within the rounding of a sum of 1000
values by 32 lanes (37 roundings of 2^-24: 2.2e-6).  Scratch follows the
output pixels, not the raw ones."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import engine

pytestmark = pytest.mark.gpu


def traces(st, cfg):
    nopit = min(cfg.num, 1000)
    ave = cfg.num // nopit
    out = []
    for dx, dy in ((0, 0), (cfg.cfx, cfg.cfy))[:1 + bool(cfg.cfx or cfg.cfy)]:
        for y in range(cfg.out_h):
            for x in range(cfg.out_w):
                x0, y0 = (cfg.map_x0 + x) * cfg.pixbinx + dx, (cfg.map_y0 + y) * cfg.pixbiny + dy
                w = st[cfg.first:cfg.first + nopit * ave, y0:y0 + cfg.biny, x0:x0 + cfg.binx].astype(np.int64)
                s = (w - cfg.background).sum(axis=(1, 2)).reshape(nopit, ave).sum(axis=1)
                out.append(np.trunc(s / ave))
    return np.array(out)


@pytest.mark.parametrize("w,h,frames,kw", [
    (24, 13, 4100, {"binx": 3, "biny": 4}),
    (22, 13, 4100, {"binx": 3, "biny": 4}),
    (21, 12, 3500, {"binx": 2, "biny": 3}),
    (32, 20, 4200, {"binx": 3, "biny": 2, "pixbinx": 4, "pixbiny": 5, "first": 7, "num": 4001, "map_x0": 1, "map_y0": 1,
                    "out_w": 6, "out_h": 2, "cfx": 2}),
    (64, 64, 4000, {"binx": 16, "biny": 16}),
    (40, 40, 2100, {"binx": 5, "biny": 5, "q": 6}),
    (40, 40, 2100, {"binx": 8, "biny": 8, "q": 6}),
    (40, 40, 1900, {"binx": 4, "biny": 4, "q": 6}),
    (26, 18, 1900, {"binx": 5, "biny": 5, "pixbinx": 1, "pixbiny": 1, "q": 6}),
    (24, 16, 4100, {"binx": 2, "biny": 3, "cfy": 2}),
    (32, 32, 20000, {"pixbinx": 2, "pixbiny": 2, "out_w": 16, "out_h": 16}),
    (32, 8, 1900, {"out_w": 16, "q": 6}),
    (40, 40, 10500, {"binx": 8, "biny": 8, "pixbinx": 4, "pixbiny": 4}),
    (40, 40, 2500, {"binx": 8, "biny": 8, "pixbinx": 4, "pixbiny": 4}),
], ids=["rows8", "rows2", "rows1", "rows-gaps-range-cfx", "rows-parts", "rows-two-frames", "one-pass-parts",
        "one-pass-short", "overlap", "cfy", "one-pass-sparse", "one-pass-half",
        "overlap-parts", "one-pass-overlap"])
def test_centre_is_the_mean_of_the_trace(w, h, frames, kw):
    rng = np.random.default_rng(81)
    st = rng.integers(100, 60000, (frames, h, w), dtype=np.uint16)
    cfg = engine.FCSConfig(width=w, height=h, frames=frames, background=100, do_fit=False, **kw)
    plan = engine.Plan(cfg)
    plan.execute_host(st)
    ref = traces(st, cfg).mean(axis=1)
    got = plan.bleach_params()[:, 12]
    assert np.abs(got / ref - 1).max() <= 2.2e-6


def test_bright_windows_above_a_high_background():
    """The raw values of a point's frames add up to more than 2^31, those above
    the background do not."""
    rng = np.random.default_rng(82)
    st = rng.integers(58900, 59200, (600_000, 8, 16), dtype=np.uint16)
    cfg = engine.FCSConfig(width=16, height=8, frames=600_000, background=59000, binx=8, biny=8, do_fit=False)
    plan = engine.Plan(cfg)
    plan.execute_host(st)
    assert np.abs(plan.bleach_params()[:, 12] / traces(st, cfg).mean(axis=1) - 1).max() <= 2.2e-6


def test_scratch_follows_the_output_pixels():
    one = engine.Plan(engine.FCSConfig(width=16, height=16, frames=3000, do_fit=False))
    for b in (2, 16):
        binned = engine.Plan(engine.FCSConfig(width=16 * b, height=16 * b, frames=3000, binx=b, biny=b, do_fit=False))
        assert binned.scratch_bytes == one.scratch_bytes
