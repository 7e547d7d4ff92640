"""Pair kernels of the level chain with a pair's lags in one block and dealt out
to several: small and large grids give a pixel the same outputs, bit for bit."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import engine
from tests.synth import brownian_stack

pytestmark = pytest.mark.gpu

W, H = 70, 66          # 73 blocks of pixels: whole


@pytest.fixture(scope="module")
def stack():
    one = brownian_stack(14, 11, 9000, seed=8, density=3.0, cps=1e5)
    return np.ascontiguousarray(np.tile(one, (1, H // 11, W // 14 + 1))[:, :, :W])


@pytest.mark.parametrize("kw", [dict(), dict(cfx=1, cfy=1), dict(q=7), dict(q=5), dict(gls=True)],
                         ids=["auto", "cross", "q7", "q5", "gls"])
@pytest.mark.parametrize("w,h", [(1, 1), (9, 7), (13, 11)])
def test_small_and_large_grids_agree(stack, kw, w, h):
    dx, dy = kw.get("cfx", 0), kw.get("cfy", 0)
    out = []
    for cw, ch in ((W, H), (w + dx, h + dy)):
        st = np.ascontiguousarray(stack[:, :ch, :cw])
        cfg = engine.FCSConfig(width=cw, height=ch, frames=9000, background=100, do_fit=False, **kw)
        r = engine.run_host(st, cfg)
        out.append([np.asarray(r[k]).reshape(ch - dy, cw - dx, -1)[:h, :w] for k in ("acf", "var", "blocked_ind")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("kw", [dict(), dict(fitstart=2, fitend=40), dict(p=32, q=5),
                                dict(cst=engine.model_constants(sz_um=1.0))], ids=["plain", "range", "p32", "spim"])
def test_few_and_many_fits_agree(stack, kw):
    """More than 4,096 fits and few take different instances of the fit kernel."""
    out = []
    for w, h in ((W, H), (14, 11)):
        cfg = engine.FCSConfig(width=w, height=h, frames=9000, background=100, **kw)
        r = engine.run_host(np.ascontiguousarray(stack[:, :h, :w]), cfg)
        out.append([np.asarray(r[k]).reshape(h, w, -1)[:11, :14] for k in ("fitres", "chi2", "fitted", "iterations")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))
