"""Level chain at the edges of its 16-sample steps and of its segments: sample
counts around whole steps at every level, levels that end the chain as a pair's
first level, segments of two samples at the top level, and every tile at a
frame count that no segment divides.  Against the FP64 oracle with the
correlator tests' tolerances."""
import pytest

from imaging_fcs_1_52_gb300 import engine
from tests.helpers import ACF_TOL, acf_deviation, oracle_kwargs, run_both
from tests.synth import brownian_stack
from tests.test_gpu_correlator import check_acf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,q,kw", [
    (8192, 8, {}), (8191, 8, {}), (8193, 8, {"cfx": 1}), (8223, 7, {}), (8208, 7, {"cfy": 1}), (4111, 6, {}),
    (4097, 5, {"cfx": -1, "map_x0": 1, "out_w": 5}), (4095, 5, {}),
])
def test_step_edges_match_oracle(frames, q, kw):
    st = brownian_stack(6, 5, frames, seed=41, density=3.0, cps=3e4)
    cfg = engine.FCSConfig(width=6, height=5, frames=frames, background=100, q=q, do_fit=False, **kw)
    gpu, ref = run_both(st, cfg)
    check_acf(gpu, ref)


def test_tiles_agree_at_a_ragged_frame_count():
    import oracle
    st = brownian_stack(7, 5, 9001, seed=42, density=3.0, cps=3e4)
    cfg = engine.FCSConfig(width=7, height=5, frames=9001, background=100, do_fit=False)
    ref = oracle.run(st, **oracle_kwargs(cfg))
    for tile in ((32, 0, 0), (64, 1, 3), (32, 2, 4)):
        plan = engine.Plan(cfg)
        plan.set_corr_tile(*tile)
        assert acf_deviation(plan.execute_host(st), ref) <= ACF_TOL, tile
