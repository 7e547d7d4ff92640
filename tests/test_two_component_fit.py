"""The specialised fits of the plain one- and two-component models against the
general fit kernel, bit for bit.  Plans: a held flow of 1e-300 is zero in the
fit's FP32 parameters, so both solve the same problem, but only an exactly zero
one selects the specialisation.  The Gpufit entry point: one more fit with a
window offset sends its whole batch to the general kernel."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import engine
from imaging_fcs_1_52_gb300.gpufit_imfcs import FitModel, FitResult, GpufitImFCS, Model
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


@pytest.mark.parametrize("npts", [3, 4, 31, 32, 33, 64, 65, 72, 95, 96, 97])
@pytest.mark.parametrize("tol,iters,kw,weighted", [(1e-16, 500, {}, True), (1e-4, 500, {}, False), (1e-16, 3, {}, True),
                                                   (1e-16, 500, dict(sz_um=1.0), True),
                                                   (1e-16, 500, dict(binx=2), True)],
                         ids=["plain", "loose-unweighted", "few-iterations", "spim", "rectangular"])
def test_gpufit_call_matches_general_kernel(npts, tol, iters, kw, weighted):
    rng = np.random.default_rng(npts)
    n = 40
    tau = 1e-3 * 1.09 ** np.arange(npts)
    N, D = np.exp(rng.uniform(-1, 3, n)), np.exp(rng.uniform(-1.5, 1.5, n))
    y = 1 / N[:, None] / (1 + 4 * D[:, None] * tau / 0.06) + rng.normal(0, 0.01, (n, npts)) / N[:, None]
    y[1, 0] = np.nan
    y[2] = 0.0
    out = []
    for extra in (0, 1):
        fm = FitModel(n + extra, npts, weighted, Model.ACF_1D, tolerance=tol, maxNumberIterations=iters,
                      parametersToFit=[i in (0, 1, 4) for i in range(20)], userInfoSize=4 * npts)
        fm.data[:] = np.concatenate([y, y[:extra]]).astype(np.float32).ravel()
        if weighted:
            fm.weights[:] = np.repeat(1e4 * np.concatenate([N, N[:extra]]) ** 2, npts)
        fm.userInfo[:] = tau
        init = fm.initialParameters.reshape(n + extra, 20)
        init[:, 0], init[:, 1] = 1.0, 1e-12
        init[:, 11:] = engine.model_constants(**kw)
        init[n:, 11:] = engine.model_constants(cfx=1, **kw)
        out.append(GpufitImFCS.fit(fm, FitResult(n + extra, 20)))
    for key in ("parameters", "states", "chiSquares", "numberIterations"):
        a, b = np.asarray(getattr(out[0], key)), np.asarray(getattr(out[1], key))
        np.testing.assert_array_equal(a.view(np.int32), b[:a.size].view(np.int32), err_msg=key)
