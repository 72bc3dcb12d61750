"""Which column kernel and shape the runs of a batch get."""
import numpy as np
import pytest

from mrm_b200 import FP32, GpuSim, media
from mrm_b200.batch import Batch

pytestmark = pytest.mark.gpu


def test_long_two_layer_columns_leave_the_one_layer_runs_alone(gpulib):
    """Column shape 2 takes a one-layer run's components in turn.  A two-layer run
    with 1024-point columns, too long for that shape's groups, does not change
    the one-layer runs' kernel (its blocks per SM) or any result."""
    one = [media.mh_medium(256, seed=5 + i, temperature=300.0) for i in range(4)]
    two = media.two_layer_medium(24, 512, seed=9)
    occ = []
    for meds in (one, one + [two]):
        b = Batch(FP32)
        runs = [b.add(m, dt=1e-13, steps=12, thermal_seed=3 + i) for i, m in enumerate(meds)]
        runs[0].set_shape(1, 2, 1)
        b.step(12)
        occ.append(b.occupancy()[1])
        for i, (r, m) in enumerate(zip(runs, meds)):
            g = GpuSim(m, precision=FP32, thermal_seed=3 + i)
            g.set_shape(1, 0, 1)
            g.step(12, 1e-13)
            for l in range(m.n_lay):
                assert np.array_equal(r.get_state(l), g.get_state(l)), (i, l)
            g.close()
        b.close()
    assert occ[0] == occ[1] > 2, occ
