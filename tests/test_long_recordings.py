"""Recordings of 0.6 to 1.9 million frames against the FP64 oracle (tolerances of
the correlator's parity tests): the monitors' scans take fewer pixels a block
from 1.1 million frames on, and at Q <= 4 the P = 32 level streams have more
spans than a grid has rows from 524,288 on."""
import numpy as np
import pytest
from scipy.signal import lfilter

from imaging_fcs_1_52_gb300 import engine
from tests.helpers import run_both
from tests.test_gpu_correlator import check_acf

pytestmark = pytest.mark.gpu


def correlated_counts(width, height, frames, seed, corr_frames=20.0, level=300.0, fluct=0.2):
    """Poisson counts of an AR(1) process of unit variance per pixel."""
    rng = np.random.default_rng(seed)
    rho = np.exp(-1.0 / corr_frames)
    z = lfilter([np.sqrt(1 - rho * rho)], [1, -rho], rng.normal(0, 1, (frames, height * width)), axis=0)
    counts = rng.poisson(level * np.maximum(0.0, 1 + fluct * z)) + 100
    return counts.astype(np.uint16).reshape(frames, height, width)


@pytest.mark.parametrize("frames,p,q,kw", [(600_003, 32, 4, {}), (1_300_000, 16, 8, {}),
                                           (1_200_000, 32, 8, {"cfx": 1, "out_w": 2}),
                                           (1_900_000, 16, 5, {"cfx": 1, "out_w": 2})])
def test_long_recordings(frames, p, q, kw):
    st = correlated_counts(3, 2, frames, seed=71)
    cfg = engine.FCSConfig(width=3, height=2, frames=frames, background=100, p=p, q=q, do_fit=False, **kw)
    gpu, ref = run_both(st, cfg)
    check_acf(gpu, ref)
