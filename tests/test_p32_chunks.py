"""P = 32 correlator at its edges: pixel counts above one scratch chunk give the
results of the pixels alone, and frame counts around a segment's and a step's
end agree with the oracle (tolerances of the correlator's parity tests)."""
import numpy as np
import pytest

from imaging_fcs_1_52_gb300 import engine
from tests.helpers import run_both
from tests.helpers import ACF_TOL, acf_deviation
from tests.synth import brownian_stack
from tests.test_gpu_correlator import check_acf

pytestmark = pytest.mark.gpu


def test_pixel_chunks_match_a_part_of_the_pixels():
    # 1,600 pixels x 50,000 frames: two chunks (512 MB hold some 1,300 pixels)
    st = engine.simulate(40, 40, 50000, steps_per_frame=1, density=4.0, seed=5)
    outs = []
    for kw in ({}, {"map_y0": 30, "out_h": 10}):
        plan = engine.Plan(engine.FCSConfig(width=40, height=40, frames=50000, background=100, p=32, do_fit=False, **kw))
        o = plan.alloc_device_outputs()
        plan.execute(st, o)
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
        if not kw:
            assert plan.kernel_launches() > 10      # three correlator kernels per chunk
    for k in outs[1]:
        np.testing.assert_array_equal(outs[0][k][-400:], outs[1][k], err_msg=k)


@pytest.mark.parametrize("frames,q,kw", [(8192, 8, {}), (8193, 8, {"cfx": 1}), (8207, 7, {}), (4100, 6, {"cfy": -1, "map_y0": 1, "out_h": 4}),
                                         (3000, 2, {})])
def test_segment_edges_match_oracle(frames, q, kw):
    st = brownian_stack(6, 5, frames, seed=31, density=3.0, cps=3e4)
    cfg = engine.FCSConfig(width=6, height=5, frames=frames, background=100, p=32, q=q, do_fit=False, **kw)
    gpu, ref = run_both(st, cfg)
    check_acf(gpu, ref)


@pytest.mark.parametrize("q,kw", [(2, {}), (4, {"cfx": 1}), (5, {})], ids=["q2", "q4-ccf", "q5"])
def test_gls_products_match_oracle(q, kw):
    """GLS takes up to 96 fit lags, P = 32 with Q <= 5 among them: the
    covariance comes from the products the P = 32 kernels hand over."""
    st = brownian_stack(6, 5, 9000, seed=61, density=3.0, cps=1e5)
    cfg = engine.FCSConfig(width=6, height=5, frames=9000, background=100, p=32, q=q, gls=True, **kw)
    gpu, ref = run_both(st, cfg)
    np.testing.assert_array_equal(gpu["blocked_ind"], ref["blocked_ind"])
    assert acf_deviation(gpu, ref) <= ACF_TOL
    n1 = cfg.chanum - 1
    g, r = gpu["covmats"].reshape(-1, n1, n1), ref["covmats"].reshape(-1, n1, n1)
    fin = np.isfinite(r).all(axis=(1, 2))
    assert fin.sum() >= 15
    scale = np.abs(r[fin]).max(axis=(1, 2), keepdims=True)
    assert np.max(np.abs(g[fin] - r[fin]) / scale) <= 1e-4
