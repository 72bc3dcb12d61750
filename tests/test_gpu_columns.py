"""FP32 column and row kernels at the edges of their splits: every column
length of the register column kernels in every compiled shape, odd row and
column counts (a last column without a partner, rows beyond the tile), padded
and periodic columns, one and two layers; tensors whose layer pairs are not
symmetric (they take the general column kernel); and layers whose grain
records differ from grain to grain (uniform ones are read once)."""
import numpy as np
import pytest

from helpers import random_m, rel_l2
from mrm_b200 import FP32, FP64, GpuSim, media

pytestmark = pytest.mark.gpu

# Relative L2 of an FP32 demag field: forward and inverse transforms of at most
# 2^10 points each way are 40 levels of butterflies, each rounded to 2^-24 of
# the values it adds.
DEMAG_TOL = 40 * 2.0**-24


def _medium(nx, ny, layers, boundary, **kw):
    med = media.two_layer_medium(nx, ny, boundary=boundary, temperature=0.0) if layers == 2 else \
        media.mh_medium(nx, ny=ny, boundary=boundary, **kw)
    return med


def _convolve(T, med, ms):
    """The convolution with the real-space tensor T[source, observation, 3a + b]
    in FP64 (demag.f90:33-135; T carries 1/(px py))."""
    py, px = T.shape[-2:]
    N = np.fft.rfft2(T)
    src = np.zeros((med.n_lay, 3, med.ny, med.nx))
    for l, lay in enumerate(med.layers):
        m32 = ms[l].astype(np.float32).astype(np.float64)
        src[l] = (lay.ms[:, None] * m32).reshape(med.ny, med.nx, 3).transpose(2, 0, 1)
    M = np.fft.rfft2(src, s=(py, px))
    H = np.einsum("soabyx,sbyx->oayx", N.reshape(med.n_lay, med.n_lay, 3, 3, *N.shape[-2:]), M)
    h = np.fft.irfft2(H, s=(py, px))[..., :med.ny, :med.nx] * (px * py)
    return h.transpose(0, 2, 3, 1).reshape(med.n_lay, -1, 3)


def _demag_check(med, shapes):
    ref = GpuSim(med, precision=FP64, demag=False)
    T = ref.download_tensor()
    ref.close()
    ms = [random_m(med.layers[0].N, 30 + l) for l in range(med.n_lay)]
    want = _convolve(T, med, ms)
    gpu = GpuSim(med, precision=FP32, tensor=T)
    for shape in shapes:
        gpu.set_shape(*shape)
        for l, m in enumerate(ms):
            gpu.set_state(l, m)
        for l in range(med.n_lay):
            assert rel_l2(gpu.eval_field(0.0, l), want[l]) < DEMAG_TOL, (shape, l)
    gpu.close()


@pytest.mark.parametrize("nx,ny,layers,boundary", [
    (9, 17, 1, 1), (16, 32, 1, 1), (33, 33, 1, 1), (12, 64, 2, 1), (20, 75, 1, 1), (5, 129, 1, 1), (7, 256, 2, 1),
    (9, 257, 1, 1), (6, 300, 2, 1), (16, 64, 1, 0), (8, 128, 2, 0), (32, 256, 1, 0), (4, 512, 1, 0),
])
def test_column_lengths_and_shapes(gpulib, nx, ny, layers, boundary):
    _demag_check(_medium(nx, ny, layers, boundary), [(0, 0, 1), (0, 1, 1), (1, 2, 2), (2, 0, 4)])


@pytest.mark.parametrize("ny", [20, 40, 130])
def test_asymmetric_tensor(gpulib, ny):
    """The soft-underlayer image makes N_xz and N_zx differ in sign."""
    med = _medium(24, ny, 1, 1)
    med.sul_mu, med.space_to_sul = 50.0, 2e-7
    _demag_check(med, [(0, 0, 1), (1, 2, 1)])


@pytest.mark.parametrize("vary", ["ms", "exchange", "both", "none"])
def test_grain_records(oracle, gpulib, vary):
    med = _medium(32, 16, 1, 1, seed=3)
    lay = med.layers[0]
    rng = np.random.default_rng(8)
    if vary in ("ms", "both"):
        lay.ms = lay.ms * rng.uniform(0.8, 1.2, lay.N)
        lay.alpha_scale = rng.uniform(0.5, 1.5, lay.N)
    if vary in ("exchange", "both"):
        lay.hx = lay.hx * rng.uniform(0.5, 1.5, lay.hx.size)
    orc = oracle.OracleSim(med)
    orc.set_state(0, random_m(lay.N, 5))
    steps, dt = 50, 1e-13
    so = orc.step(steps, dt)
    for row in range(5):
        gpu = GpuSim(med, precision=FP32, tensor=orc.n2d)
        gpu.set_shape(row, 0, 1)
        gpu.set_state(0, random_m(lay.N, 5))
        sg = gpu.step(steps, dt)
        # a step rotates by at most gamma H dt ~ 0.05 rad, rounded to a few ulp
        # in each of its two stages: 8 ulp a step
        assert np.abs(gpu.get_state(0) - orc.get_state(0)).max() < steps * 8 * 2.0**-24, row
        assert np.allclose(sg["mave"], so["mave"], rtol=0, atol=steps * 8 * 2.0**-24)
        gpu.close()


def test_small_asymmetric_part(gpulib):
    """Two layers with 512-point columns and a tensor of N_zz on the diagonal
    with a small N_xz = -N_zx: moments along x see N_zx alone, so its sign shows
    in H_z at full precision however small it is."""
    med = _medium(8, 256, 2, 1)
    gpu = GpuSim(med, precision=FP32)
    px, py = gpu.fft_grid()
    T = np.zeros((2, 2, 9, py, px))
    T[:, :, 8, 0, 0] = 1.0 / (px * py)
    # |N_xz - N_zx| is 1.2e-7 of the largest value in the spectrum
    e = 3e-8 / (px * py)
    T[:, :, 2, 0, 1], T[:, :, 2, 0, -1] = e, -e
    T[:, :, 6] = -T[:, :, 2]
    gpu.upload_tensor(T)
    rng = np.random.default_rng(6)
    ms = [np.outer(rng.choice([-1.0, 1.0], lay.N), [1.0, 0.0, 0.0]) for lay in med.layers]
    want = _convolve(T, med, ms)
    for l, m in enumerate(ms):
        gpu.set_state(l, m)
    for l in range(2):
        assert rel_l2(gpu.eval_field(0.0, l)[:, 2], want[l][:, 2]) < DEMAG_TOL
    gpu.close()
