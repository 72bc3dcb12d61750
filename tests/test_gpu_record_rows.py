"""Grain records that the row kernel reads from global memory.  Four rows of 256
grains need 72 KB of staging (damping, anisotropy and exchange records and six
rows of moments, 16 B a grain), more than a quarter of an SM, which is a block's
share in row shape 3; so nothing is staged there, and a layer whose records are
all equal is read through its first one.  Row shape 0 stages its one row."""
import numpy as np
import pytest

from helpers import random_m
from mrm_b200 import FP32, GpuSim, media

pytestmark = pytest.mark.gpu

STEPS, DT = 50, 1e-13
# a step rotates by at most gamma H dt ~ 0.05 rad, rounded to a few ulp in each
# of its two stages: 8 ulp a step
TOL = STEPS * 8 * 2.0**-24


def _medium(vary):
    med = media.mh_medium(256, ny=8, boundary=1, seed=3, temperature=0.0)
    lay, rng = med.layers[0], np.random.default_rng(8)
    if "records" in vary:
        lay.ms = lay.ms * rng.uniform(0.8, 1.2, lay.N)
        lay.alpha_scale = rng.uniform(0.5, 1.5, lay.N)
    if "exchange" in vary:
        lay.hx = lay.hx * rng.uniform(0.5, 1.5, lay.hx.size)
    return med


@pytest.mark.parametrize("row", [0, 3])
def test_uploads_of_equal_and_of_varying_records(oracle, gpulib, row):
    """One handle through uploads of every kind, each following another."""
    gpu = None
    for k, vary in enumerate(["", "records", "exchange", "", "records exchange", ""]):
        med = _medium(vary)
        orc = oracle.OracleSim(med)
        if gpu is None:
            gpu = GpuSim(med, precision=FP32, tensor=orc.n2d)
            gpu.set_shape(row, 0, 1)
        else:
            gpu.upload_medium(med)
        m = random_m(med.layers[0].N, 5 + k)
        orc.set_state(0, m)
        gpu.set_state(0, m)
        gpu.set_time(0.0)
        so, sg = orc.step(STEPS, DT), gpu.step(STEPS, DT)
        assert np.abs(gpu.get_state(0) - orc.get_state(0)).max() < TOL, (k, vary)
        assert np.allclose(sg["mave"], so["mave"], rtol=0, atol=TOL)
    gpu.close()
