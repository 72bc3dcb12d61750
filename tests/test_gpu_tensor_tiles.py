"""The device tensor at the edges of the tensor kernel's tiles: first, last and
half-way slots, grids smaller than a tile, unequal cell sides (no shared y
lattice), unequal layer thicknesses, periodic images and the SUL / head image
terms, against quadruple precision."""
import ctypes as C

import numpy as np
import pytest

from mrm_b200 import FP64, GpuSim
from mrm_b200 import media

pytestmark = pytest.mark.gpu


def _offsets(f, n, nimg):
    """Every offset that wraps onto slot f of n, with its periodic images
    (tensor_element.f90:233-257)."""
    if f == n // 2:
        return [-n // 2 - n * k for k in range(nimg + 1)] + [n // 2 + n * k for k in range(nimg + 1)]
    i = 0 if f == 0 else (-f if f <= n // 2 else n - f)
    return [i + n * k for k in range(-nimg, nimg + 1)]


def _slot(oracle, med, px, py, dz_s, dz_o, rz, fi, fj, nimg):
    pts = [(i, j) for j in _offsets(fj, py, nimg) for i in _offsets(fi, px, nimg)]
    ix = np.array([p[0] for p in pts], np.int32)
    iy = np.array([p[1] for p in pts], np.int32)
    out = np.zeros(9)
    ip = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))  # noqa: E731
    oracle.lib().orc_volume_averaged_n_q(len(pts), ip(ix), ip(iy), med.dx, med.dy, rz, med.dx, med.dy, dz_s, med.dx, dz_o,
                                         1.0 / (med.dx * med.dy * dz_o * px * py), out.ctypes.data_as(C.POINTER(C.c_double)))
    return out.reshape(3, 3)


@pytest.mark.parametrize("nx,ny,boundary,images,ratio,dz,sul_mu,head_mu", [
    (4, 2, 0, 0, 1.0, [10e-7], 1.0, 1.0),
    (8, 32, 0, 2, 1.0, [10e-7], 50.0, 1.0),
    (16, 16, 0, 1, 0.75, [10e-7], 1.0, 20.0),
    (5, 9, 1, 0, 1.25, [8e-7, 4e-7], 1.0, 1.0),
    (17, 8, 1, 0, 1.0, [8e-7, 4e-7], 3.0, 4.0),
])
def test_tensor_tiles(oracle, gpulib, nx, ny, boundary, images, ratio, dz, sul_mu, head_mu):
    med = media.two_layer_medium(nx, ny, boundary=boundary) if len(dz) == 2 else media.mh_medium(nx, ny=ny, boundary=boundary)
    med.dy = ratio * med.dx
    med.images, med.sul_mu, med.head_mu, med.space_to_sul, med.fly_height = images, sul_mu, head_mu, 5e-7, 6e-7
    gpu = GpuSim(med, precision=FP64)
    T = gpu.download_tensor()
    px, py = gpu.fft_grid()
    gpu.close()
    nimg = images if boundary == 0 else 0
    nl = len(dz)
    # heights above the SUL and depths below the head of the layers' mid-planes
    bottom = np.array([5e-7 + sum(dz[l + 1:]) for l in range(nl)])
    depth = np.array([6e-7 + sum(dz[:l]) + 0.5 * dz[l] for l in range(nl)])
    edge = lambda n: sorted({f for f in (0, 1, 6, 7, 8, 9, n // 2 - 1, n // 2, n // 2 + 1, n - 1) if 0 <= f < n})  # noqa: E731
    sign = np.array([[-1.0] * 3, [-1.0] * 3, [1.0] * 3])
    for ks in range(nl):
        for ko in range(nl):
            zs, zo = bottom[ks] + 0.5 * dz[ks], bottom[ko] + 0.5 * dz[ko]
            for fi in edge(px):
                for fj in edge(py):
                    q = _slot(oracle, med, px, py, dz[ks], dz[ko], zs - zo, fi, fj, nimg)
                    if sul_mu > 1.0:
                        f = (sul_mu - 1.0) / (sul_mu + 1.0)
                        q = q + f * sign * _slot(oracle, med, px, py, dz[ks], dz[ko], -(zs + zo), fi, fj, nimg)
                    if head_mu > 1.0:
                        f = (head_mu - 1.0) / (head_mu + 1.0)
                        q = q + f * sign * _slot(oracle, med, px, py, dz[ks], dz[ko], depth[ks] + depth[ko], fi, fj, nimg)
                    got = T[ks, ko, :, fj, fi].reshape(3, 3).T
                    # double-double values rounded once to FP64; the bound of the other slots' tests
                    assert np.abs(got - q).max() <= 1e-11 * np.abs(q).max(), (ks, ko, fi, fj)
