"""Batches whose runs end, start late or are parked while their neighbours step:
with more column tasks than persistent blocks a block meets tasks without work
in a row, ahead of, between and after tasks with work.  Every run has to stay
bit for bit what it is alone."""
import numpy as np
import pytest

from helpers import random_m
from mrm_b200 import FP32, GpuSim, media
from mrm_b200.batch import Batch

pytestmark = pytest.mark.gpu

DT = 1e-13


def _alone(med, seed, steps, shape=None):
    g = GpuSim(med, precision=FP32, thermal_seed=seed)
    if shape:
        g.set_shape(*shape)
    if steps:
        g.step(steps, DT)
    out = [g.get_state(l) for l in range(med.n_lay)]
    g.close()
    return out


def _same(run, med, want):
    for l in range(med.n_lay):
        assert np.array_equal(run.get_state(l), want[l]), (med.nx, med.ny, l)


# (1024 x 256 x 2: 513 column tasks of 512 points a run, 148 persistent blocks or
# twice that; 256 x 512 x 2: 1024-point columns)
@pytest.mark.parametrize("nx,ny", [(1024, 256), (256, 512)])
@pytest.mark.parametrize("shape", [None, (1, 0, 1), (1, 1, 1), (1, 2, 1)])
def test_two_layer_budgets_and_delay(gpulib, nx, ny, shape):
    meds = [media.head_write_medium(nx, ny, seed=3 + i, prbs_seed=i + 1) for i in range(4)]
    b = Batch(FP32)
    first, runs = None, []
    for i, (m, k) in enumerate(zip(meds, [3, 5, 40, 12])):  # two that end early in front, a delayed one behind
        runs.append(b.add(m, dt=DT, steps=k, thermal_seed=20 + i, tensor_from=first))
        first = first or runs[0]
    runs[3].delay(28)
    if shape:
        runs[0].set_shape(*shape)
    b.step(40)
    b.stats(runs)  # (waits, and reports a device error)
    assert [r.get_time()[1] for r in runs] == [3, 5, 40, 12]
    for i, (r, m, k) in enumerate(zip(runs, meds, [3, 5, 40, 12])):
        _same(r, m, _alone(m, 20 + i, k, shape))
    # the ended runs stay where they are
    b.runs[2].set_run(DT, 46)
    b.step(20)
    b.stats(runs)
    for i, (r, m, k) in enumerate(zip(runs, meds, [3, 5, 46, 12])):
        _same(r, m, _alone(m, 20 + i, k, shape))
    b.close()


def test_field_of_one_run_with_the_others_parked(gpulib):
    meds = [media.two_layer_medium(1024, 256, seed=5 + i, temperature=0.0) for i in range(3)]
    b = Batch(FP32)
    runs = []
    for i, m in enumerate(meds):
        runs.append(b.add(m, dt=DT, steps=8, tensor_from=runs[0] if runs else None))
        for l in range(2):
            runs[i].set_state(l, random_m(m.layers[l].N, 60 + 2 * i + l))
    for i in (2, 0, 1):
        g = GpuSim(meds[i], precision=FP32)
        for l in range(2):
            g.set_state(l, random_m(meds[i].layers[l].N, 60 + 2 * i + l))
        for l in range(2):
            assert np.array_equal(runs[i].eval_field(0.0, l), g.eval_field(0.0, l)), (i, l)
        g.close()
    b.close()


# One layer, column shapes 0 and 1 (components side by side) and 2 (in turn):
# 513 tasks a run of 256-point columns in shape 1, 257 in shape 0; mixed
# lengths change the block's tables between tasks.
@pytest.mark.parametrize("shape", [(1, 0, 1), (1, 1, 1), (1, 2, 1)])
@pytest.mark.parametrize("rows", [[100, 100, 100, 100, 100, 100, 100, 100], [512, 512, 512], [100, 60, 250, 33, 250, 100, 100, 60]])
def test_one_layer_budgets(gpulib, shape, rows):
    meds = [media.mh_medium(1000, ny=ny, seed=40 + i, temperature=300.0) for i, ny in enumerate(rows)]
    steps = 20
    ends = [2 if i < len(rows) // 2 else 7 if i == len(rows) - 1 else steps for i in range(len(rows))]
    b = Batch(FP32)
    runs = [b.add(m, dt=DT, steps=k, thermal_seed=70 + i) for i, (m, k) in enumerate(zip(meds, ends))]
    runs[0].set_shape(*shape)
    b.step(steps)
    b.stats(runs)
    for i, (r, m, k) in enumerate(zip(runs, meds, ends)):
        _same(r, m, _alone(m, 70 + i, k, shape))
    # parked runs between stepping ones
    for i in range(0, len(rows), 2):
        runs[i].set_run(DT, ends[i], active=False)
    for i in range(1, len(rows), 2):
        runs[i].set_run(DT, steps + 5)
    b.step(25)
    b.stats(runs)
    for i, (r, m, k) in enumerate(zip(runs, meds, ends)):
        _same(r, m, _alone(m, 70 + i, k if i % 2 == 0 else min(steps + 5, k + 25), shape))
    b.close()


@pytest.mark.parametrize("ny", [128, 512])
def test_parked_in_place_runs_beside_others(gpulib, ny):
    """The in-place column kernel's launch covers only its own runs (here a
    32-point one); with those parked, the launches behind it still follow the
    row kernel of the runs that step: one with demag in the register column
    kernel, one without demag."""
    small, big = media.mh_medium(40, ny=16, seed=90, temperature=300.0), media.mh_medium(256, ny=ny, seed=91, temperature=300.0)
    bare = media.mh_medium(1024, ny=512, seed=92, temperature=300.0)
    b = Batch(FP32)
    r0 = b.add(small, dt=DT, steps=40, thermal_seed=1)
    r1 = b.add(big, dt=DT, steps=40, thermal_seed=2)
    r2 = b.add(bare, dt=DT, steps=40, thermal_seed=3, demag=False)
    r0.set_run(DT, 40, active=False)
    b.step(40)
    b.stats([r1, r2])
    _same(r0, small, _alone(small, 1, 0))
    _same(r1, big, _alone(big, 2, 40))
    g = GpuSim(bare, precision=FP32, thermal_seed=3, demag=False)
    g.step(40, DT)
    _same(r2, bare, [g.get_state(0)])
    g.close()
    b.close()
