"""The specialised two-component fit against the general fit kernel, bit for
bit: a held flow of 1e-300 is zero in the fit's FP32 parameters, so both solve
the same problem, but only an exactly zero one selects the specialisation."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import engine
from tests.synth import brownian_stack

pytestmark = pytest.mark.gpu

FREE = (1, 1, 0, 0, 1, 1, 1, 0, 0, 0, 0)


@pytest.fixture(scope="module")
def stack():
    def d_map(x, y):
        return np.where(np.random.default_rng(4).random(len(x)) < 0.3, 5.0, 0.5)
    return brownian_stack(13, 9, 6000, seed=22, density=2.0, cps=3e4, d_map=d_map)


@pytest.mark.parametrize("case", [dict(), dict(fitstart=3, fitend=8), dict(fitend=31), dict(fitend=32),
                                  dict(fitend=33), dict(fitend=64), dict(fitend=65), dict(p=32, q=5), dict(p=32, q=6),
                                  dict(max_iter=0), dict(max_iter=7),
                                  dict(binx=2, biny=1, cst=engine.model_constants(binx=2, biny=1)),
                                  dict(cst=engine.model_constants(sz_um=0.9)),
                                  dict(map_w=1, map_h=1)],
                         ids=lambda c: "-".join(f"{k}{v}" if np.ndim(v) == 0 else k for k, v in c.items()) or "plain")
def test_matches_general_kernel(stack, case):
    case = dict(case)
    w, h = case.pop("map_w", 13), case.pop("map_h", 9)
    st = np.ascontiguousarray(stack[:, :h, :w])
    out = []
    for vx in (0.0, 1e-300):
        cfg = engine.FCSConfig(width=w, height=h, frames=6000, background=100, free_mask=FREE,
                               init=(1.0, 1e-12, vx, 0, 0, 0.3, 1e-13, 0, 0, 0, 0), **case)
        out.append(engine.run_host(st, cfg))
    for key in ("fitres", "chi2", "fitted", "iterations"):
        a, b = out[0][key], out[1][key]
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32), err_msg=key)
