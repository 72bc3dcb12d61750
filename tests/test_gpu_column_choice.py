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


def _images(med):
    """A soft underlayer: its image terms make the tensor asymmetric, which the
    in-place column kernel takes."""
    med.sul_mu, med.space_to_sul = 50.0, 2e-7
    return med


def _step_all(meds, n=8):
    b = Batch(FP32)
    same, runs = {}, []
    for i, m in enumerate(meds):
        key = (m.nx, m.ny, m.n_lay)
        runs.append(b.add(m, dt=1e-13, steps=n, thermal_seed=7, tensor_from=same.get(key)))
        same.setdefault(key, runs[-1])
    b.step(n)
    b.stats(runs)
    shape, out = runs[0].get_shape(), [[r.get_state(l) for l in range(m.n_lay)] for r, m in zip(runs, meds)]
    b.close()
    return shape, out


def test_tuned_shapes_follow_the_column_kernel(gpulib):
    """One column per task is all a batch of the register kernel has to time (it
    does not use the number); a batch of the in-place kernel with the same sizes
    times its own, and one column per task is never the fastest there (81 or 68 us
    a launch against 62 with two)."""
    med = media.mh_medium(256, seed=3)
    assert _step_all([med] * 16)[0][2] == 1
    assert _step_all([_images(media.mh_medium(256, seed=3))] * 16)[0][2] > 1


def test_tuned_shapes_that_do_not_fit_are_tuned_again(gpulib):
    """Short in-place columns are fastest at many columns per task; the same
    batch with its long two-layer run on the in-place kernel as well has no
    shared memory for that many."""
    short = _images(media.mh_medium(128, seed=3))
    sym = media.two_layer_medium(24, 512, seed=9, temperature=0.0)
    asym = _images(media.two_layer_medium(24, 512, seed=9, temperature=0.0))
    _step_all([short] * 32 + [sym])
    _, out = _step_all([short] * 32 + [asym])
    g = GpuSim(asym, precision=FP32, thermal_seed=7)
    g.step(8, 1e-13)
    for l in range(2):
        assert np.array_equal(out[-1][l], g.get_state(l)), l
    g.close()


@pytest.mark.parametrize("layers,ny,most", [(2, 48, 2), (2, 100, 2), (1, 400, 3), (1, 512, 4)])
def test_row_blocks_spread_over_the_sms(gpulib, layers, ny, most):
    """Runs of the in-place column kernel: no more row blocks fit an SM than an
    even spread of the launch needs, at least two."""
    med = media.two_layer_medium(437, ny, seed=4) if layers == 2 else _images(media.mh_medium(437, ny=ny, seed=4))
    b = Batch(FP32)
    r = b.add(med, dt=1e-13, steps=10)
    r.set_shape(0, 2, 2)
    b.step(10)
    b.stats([r])
    assert b.occupancy()[0] == most
    b.close()


def test_row_blocks_of_a_small_run_keep_their_room(gpulib):
    """65 column tasks leave more than half of the SMs to the row blocks."""
    b = Batch(FP32)
    r = b.add(_images(media.mh_medium(64, seed=4)), dt=1e-13, steps=10)
    r.set_shape(0, 2, 1)
    b.step(10)
    b.stats([r])
    assert b.occupancy()[0] == 4
    b.close()


@pytest.mark.parametrize("runs,row", [(1, 0), (8, 2)])
def test_rows_per_block_without_the_tuner(gpulib, runs, row):
    """Rows of 128 grains go two to a block where there are enough of them."""
    med = media.mh_medium(128, seed=4, temperature=300.0)
    b = Batch(FP32)
    rs = []
    for i in range(runs):
        rs.append(b.add(med, dt=1e-13, steps=8, thermal_seed=3, tensor_from=rs[0] if rs else None))
    rs[0].set_autotune(False)
    b.step(8)
    b.stats(rs)
    assert rs[0].get_shape()[0] == row
    g = GpuSim(med, precision=FP32, thermal_seed=3)
    g.step(8, 1e-13)
    assert np.array_equal(rs[-1].get_state(0), g.get_state(0))
    g.close()
    b.close()


def test_column_shape_without_the_tuner(gpulib):
    """Shape 1 of the register column kernel, shape 0 of the in-place one."""
    for med, col in ((media.mh_medium(32, seed=4), 1), (_images(media.mh_medium(32, seed=4)), 0),
                     (media.two_layer_medium(8, 500, seed=4), 1), (media.two_layer_medium(8, 20, seed=4), 0)):
        g = GpuSim(med, precision=FP32)
        g.set_autotune(False)
        g.step(8, 1e-13)
        assert g.get_shape()[1] == col
        g.close()


@pytest.mark.parametrize("nx,ny,row,col", [(200, 250, 4, 1), (40, 500, 4, 1), (600, 200, 3, 2), (1000, 140, 2, 2)])
def test_blocks_of_two_layer_runs_spread_over_the_sms(gpulib, nx, ny, row, col):
    """Two-layer runs on the register column kernel: one column block to an SM where
    there are no more tasks than SMs; row blocks as for the in-place kernel."""
    med = media.two_layer_medium(nx, ny, seed=4, temperature=300.0)
    b = Batch(FP32)
    r = b.add(med, dt=1e-13, steps=10, thermal_seed=3)
    r.set_shape(0, 1, 1)
    b.step(10)
    b.stats([r])
    assert b.occupancy() == (row, col)
    g = GpuSim(med, precision=FP32, thermal_seed=3)
    g.set_shape(1, 0, 1)
    g.step(10, 1e-13)
    for l in range(2):
        assert np.array_equal(r.get_state(l), g.get_state(l))
    g.close()
    b.close()
