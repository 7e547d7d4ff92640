"""Fits whose model or data leave the finite range: dead pixels (a zero curve
of variance zero: infinite weights), noise that sends D far negative
(4 D tau + s^2 < 0 gives a NaN model), initial values outside the model's
domain.  What becomes of such a fit depends on its own curve alone: a grid
above 4,096 fits and the two rows of it that hold those pixels, which the
other form of the fit kernel takes, agree bit for bit, and dead pixels stay
unfitted."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import engine
from tests.synth import brownian_stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("init", [(1, 1e-12, 0), (1, -1e-12, 0), (1e-3, 1e-9, 0), (-1, 1e-12, 0), (1e6, 1e-12, 0),
                                  (1, 1e-6, 0), (1, 1e25, 0)], ids=str)
def test_results_do_not_depend_on_other_fits(init):
    import torch
    w, h, frames = 65, 64, 2600
    rng = np.random.default_rng(5)
    st = rng.poisson(200, (frames, h, w)).astype(np.uint16)
    st[:, ::3, ::3] = 500                      # dead: no variance
    dead = np.zeros((h, w), bool)
    dead[::3, ::3] = True
    dev = torch.from_numpy(st.view(np.int16)).cuda().view(torch.uint16)
    n, d, g = init
    outs = []
    for kw in ({}, {"map_y0": 30, "out_h": 2}):
        plan = engine.Plan(engine.FCSConfig(width=w, height=h, frames=frames, init=(n, d, 0, 0, g, 0, 0, 0, 0, 0, 0),
                                            **kw))
        o = plan.alloc_device_outputs()
        plan.execute(dev, o)
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    full, part = outs
    assert (full["var"][dead.ravel()] == 0).all()
    assert not full["fitted"][dead.ravel()].any()
    assert np.isnan(full["fitres"][dead.ravel()][:, [0, 1, 4]]).all()
    assert np.isfinite(full["fitres"][full["fitted"] == 1]).all()
    for k in ("fitted", "iterations", "fitres", "chi2"):
        np.testing.assert_array_equal(full[k][30 * w:32 * w], part[k], err_msg=k)


@pytest.mark.parametrize("gls", [False, True])
def test_bayes_terms_beside_failed_fits(gls):
    """Pixels without a fit (dead: no factorisation either) get the failed
    fits' probabilities, 0 / 0 as the oracle's, and leave their neighbours'
    as they are."""
    st = brownian_stack(8, 6, 6000, seed=21, density=2.0, cps=3e4)
    st[:, 2:4, ::2] = 300
    dead = np.zeros((6, 8), bool)
    dead[2:4, ::2] = True
    outs = [engine.run_host(st, engine.FCSConfig(width=8, height=6, frames=6000, background=100, gls=gls, bayes=True,
                                                 **kw)) for kw in ({}, {"map_y0": 2, "out_h": 2})]
    full, part = (o["bayes_prob"] for o in outs)
    assert np.isnan(full[dead.ravel()]).all()
    assert np.isfinite(full[~dead.ravel()]).all(axis=1).sum() >= 30
    np.testing.assert_array_equal(full[2 * 8:4 * 8], part)
