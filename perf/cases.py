"""The timed cases of the grain-dynamics path, through its public entry points.

A pass is what a host program does between two of its own actions: it advances
its run (or its batch of runs) by the steps of one sampling interval and takes
the sampled magnetisation and the state, or it builds the demag tensor of a new
geometry, or it reads a written track back.  Media are the synthetic ones of
mrm_b200.media with the sizes of the benchmark, its workloads and the tests.

The state and field of an FP32 run are FP32 numbers, which the accessors hand
out widened to double; they are kept as FP32 here, so each output has the
precision its run has.
"""
import math

import numpy as np
import torch

from mrm_b200 import FP32, FP64, GpuSim, media
from mrm_b200.batch import Batch

DT = 1e-13  # s, the benchmark's fixed step
READBACK = dict(zoff=1e-7, dzobs=1e-7, num_images=0)  # slab 1 nm above the media, 1 nm thick


def listed():
    return [
        # the smallest run a server takes: launch latency is all there is
        dict(name="mh 32x32 fp32", kind="run", medium="mh", nx=32, ny=32, fp=32, temperature=300.0, llg_type=-3, steps=100),
        # the CPU-sized M(H) loop in full precision, no thermal field
        dict(name="mh 64x64 fp64 T0", kind="run", medium="mh", nx=64, ny=64, fp=64, temperature=0.0, llg_type=-3, steps=100),
        # a rectangular sample off every power of two, the semi-implicit midpoint push
        dict(name="mh 200x75 fp32 midpoint", kind="run", medium="mh", nx=200, ny=75, fp=32, temperature=300.0, llg_type=-2, steps=100),
        # the drop-in single run at the headline size, sampled for its M(H) curve
        dict(name="mh 256x256 fp32", kind="run", medium="mh", nx=256, ny=256, fp=32, temperature=300.0, llg_type=-3, steps=200),
        # the same in full precision: the run that an FP32 result is judged by
        dict(name="mh 256x256 fp64", kind="run", medium="mh", nx=256, ny=256, fp=64, temperature=300.0, llg_type=-3, steps=50),
        # the largest request that a server takes
        dict(name="mh 512x512 fp32", kind="run", medium="mh", nx=512, ny=512, fp=32, temperature=300.0, llg_type=-3, steps=100),
        # a two-layer track under the moving write head
        dict(name="write 1024x256x2 fp32", kind="run", medium="write", nx=1024, ny=256, fp=32, temperature=300.0, llg_type=-3, steps=50),
        # heat-assisted layer below its Curie temperature, variable |m|
        dict(name="llb 256x256 fp32", kind="run", medium="llb", nx=256, ny=256, fp=32, temperature=600.0, llg_type=-3, steps=100),
        # seeds of one medium advanced together: an ensemble over the thermal noise
        dict(name="batch 32 of 256x256", kind="batch", runs=32, lo=256, hi=256, llg_type=-3, steps=200),
        # realisations of all sizes advanced together, a server's call
        dict(name="batch 64 of 32..256", kind="batch", runs=64, lo=32, hi=256, llg_type=-3, steps=100),
        # the tensor of a new geometry and the first demag field with it: what every new run waits for
        dict(name="tensor 256x256", kind="tensor", nx=256, ny=256, fp=32),
        # the readback field of a written two-layer track
        dict(name="readback 1024x256x2", kind="readback", nx=1024, ny=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(rng, grains, most):
    return max(10, min(200, int(most / grains), _log_int(rng, 20, 200)))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["batch"] * 2 + ["tensor", "readback"])
    if kind == "readback":  # the off-plane field takes powers of two
        return dict(kind=kind, nx=2 ** rng.randint(7, 10), ny=2 ** rng.randint(6, 8))
    if kind == "tensor":
        return dict(kind=kind, nx=_log_int(rng, 32, 512), ny=_log_int(rng, 32, 512), fp=rng.choice([32, 32, 64]))
    if kind == "batch":
        runs, lo = _log_int(rng, 4, 64), 32 * rng.randint(1, 6)
        hi = 32 * rng.randint(lo // 32, 8)
        return dict(kind=kind, runs=runs, lo=lo, hi=hi, llg_type=-3, steps=_steps(rng, runs * hi * hi, 2e8))
    medium = rng.choice(["mh", "mh", "mh", "write", "llb"])
    if medium == "write":
        nx, ny = _log_int(rng, 128, 1024), _log_int(rng, 32, 256)
        return dict(kind=kind, medium=medium, nx=nx, ny=ny, fp=32, temperature=round(rng.uniform(250.0, 350.0), 1),
                    llg_type=rng.choice([-3, -3, -2]), steps=_steps(rng, 2 * nx * ny, 2e7))
    if medium == "llb":  # hot enough that the |m| relaxation is resolved by the step
        nx = _log_int(rng, 32, 256)
        return dict(kind=kind, medium=medium, nx=nx, ny=nx, fp=32, temperature=round(rng.uniform(560.0, 620.0), 1), llg_type=-3,
                    steps=_steps(rng, nx * nx, 5e6))
    fp = rng.choice([32, 32, 32, 64])
    hi = 512 if fp == 32 else 256
    nx, ny = _log_int(rng, 24, hi), _log_int(rng, 24, hi)
    return dict(kind=kind, medium=medium, nx=nx, ny=ny, fp=fp, temperature=rng.choice([0.0, 300.0, 350.0]),
                llg_type=rng.choice([-3, -3, -3, 2, -2]), steps=_steps(rng, nx * ny, 2e7 if fp == 32 else 3e6))


# ---------------- inputs ----------------

def _medium(case, seed):
    if case["medium"] == "write":
        return media.head_write_medium(case["nx"], case["ny"], seed=seed, prbs_seed=seed, temperature=case["temperature"])
    if case["medium"] == "llb":
        return media.llb_medium(case["nx"], seed=seed, temperature=case["temperature"])
    return media.mh_medium(case["nx"], ny=case["ny"], seed=seed, temperature=case["temperature"])


def _batch_media(case, seed):
    """One medium per run: with one size the same medium for every run (the
    runs differ by their thermal seed), else sides log-uniform in [lo, hi]
    rounded to multiples of 32, their first the largest."""
    n, lo, hi = case["runs"], case["lo"], case["hi"]
    if lo == hi:
        return [media.mh_medium(lo, seed=seed, temperature=300.0)] * n
    rng = np.random.default_rng(seed)
    # the sizes belong to the case, the media to the seed
    sides = np.exp(np.random.default_rng(n * 1000003 + lo * 1009 + hi).uniform(math.log(lo), math.log(hi), n))
    sides = [hi] + [max(32, int(round(s / 32.0)) * 32) for s in sides[1:]]
    return [media.mh_medium(s, seed=seed + 1 + i, temperature=300.0, k_sigma=-rng.uniform(0.03, 0.10)) for i, s in enumerate(sides)]


def _written(nx, ny, seed):
    """A written pattern: bits of 2..6 columns, transitions off by a column from row to row, moments a few degrees off the normal."""
    rng = np.random.default_rng(seed)
    edges = np.cumsum(rng.integers(2, 7, nx))
    col = np.searchsorted(edges, np.arange(nx)[None, :] + rng.integers(0, 2, (ny, nx)), side="right")
    up = np.where(col % 2 == 0, 1.0, -1.0).reshape(-1)
    th, ph = np.abs(rng.normal(0.0, 0.1, nx * ny)), rng.uniform(0.0, 2.0 * np.pi, nx * ny)
    return np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), up * np.cos(th)], axis=1)


def _pinned(n):
    t = torch.empty((n, 3), dtype=torch.float64, pin_memory=True)
    return t, t.numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        meds = _batch_media(case, seed)
        b = Batch(FP32, 0)
        first = {}
        runs = []
        for i, m in enumerate(meds):
            r = b.add(m, dt=DT, thermal_seed=seed + i, tensor_from=first.get(m.nx))
            first.setdefault(m.nx, r)
            runs.append(r)
        t, a = _pinned(sum(m.n_grains for m in meds))
        at = np.cumsum([0] + [m.n_grains for m in meds])
        return dict(case=case, batch=b, runs=runs, out=t, parts=[a[at[i]:at[i + 1]] for i in range(len(meds))])
    if kind == "run":
        med = _medium(case, seed)
        sim = GpuSim(med, precision=FP64 if case["fp"] == 64 else FP32, thermal_seed=seed)
        return dict(case=case, sim=sim, outs=[_pinned(l.N) for l in med.layers])
    if kind == "tensor":
        med = media.mh_medium(case["nx"], ny=case["ny"], seed=seed)
        med.m0 = [_written(case["nx"], case["ny"], seed)]
        return dict(case=case, sim=GpuSim(med, precision=FP64 if case["fp"] == 64 else FP32))
    med = media.head_write_medium(case["nx"], case["ny"], seed=seed, prbs_seed=seed)
    med.m0 = [_written(case["nx"], case["ny"], seed + l) for l in range(2)]
    return dict(case=case, sim=GpuSim(med, precision=FP32))


# ---------------- passes ----------------

def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"], case["llg_type"])
        st = b.stats(state["runs"])
        for r, a in zip(state["runs"], state["parts"]):
            r.get_state(0, a)
        return dict(m=state["out"].float(), mave=st["mave"].astype(np.float32), have=st["have"].astype(np.float32))
    sim = state["sim"]
    if case["kind"] == "tensor":
        sim.build_tensor()
        h = torch.from_numpy(sim.eval_field(0.0))
        return dict(h_demag=h if case["fp"] == 64 else h.float())
    if case["kind"] == "readback":
        return dict(h=sim.off_field(**READBACK))
    keep = (lambda t: t.clone()) if case["fp"] == 64 else (lambda t: t.float())
    st = sim.step(case["steps"], DT, case["llg_type"])
    out = dict(mave=keep(torch.from_numpy(st["mave"].copy())), have=keep(torch.from_numpy(st["have"].copy())))
    for l, (t, a) in enumerate(state["outs"]):
        sim.get_state(l, a)
        out["m%d" % l] = keep(t)
    if case["medium"] == "llb":
        out["mag"] = keep(torch.from_numpy(sim.get_mag(0)))
    return out


# ---------------- what a pass cannot do without ----------------

def _grid(n):
    p = 2
    while p < 2 * n:
        p *= 2
    return p


def _step_work(nx, ny, nl, fp, evals):
    """One time step: the state read and written, the grain parameters and exchange coefficients read; the transforms of the zero-padded
    real convolution, the 3x3 products, and about 150 operations a grain for the field, the noise and the push."""
    px, py = _grid(nx), _grid(ny)
    real = 4 if fp == 32 else 8
    n, half = nx * ny * nl, px // 2 + 1
    rows = 2 * 3 * nl * ny * 2.5 * px * math.log2(px)
    cols = 2 * 3 * nl * half * 5.0 * py * math.log2(py)
    prod = half * py * nl * nl * 9 * 4.0
    return n * 20 * real, evals * (rows + cols + prod + 150.0 * n)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        by = fl = 0.0
        for m in _batch_media(case, 0) if case["lo"] != case["hi"] else [_Size(case["lo"])] * case["runs"]:
            b, f = _step_work(m.nx, m.ny, 1, 32, 2)
            by, fl = by + case["steps"] * b + m.nx * m.ny * 24, fl + case["steps"] * f
        return dict(bytes=by, flops=fl)
    nx, ny = case["nx"], case["ny"]
    if kind == "run":
        nl = 2 if case["medium"] == "write" else 1
        b, f = _step_work(nx, ny, nl, case["fp"], 1 if case["llg_type"] == 2 else 2)
        return dict(bytes=case["steps"] * b + nx * ny * nl * 24, flops=case["steps"] * f)
    # a tensor: per corner of a cell about 15 logarithms, arctangents and roots of 20 operations for each of 2 (tensor) or 4 (readback)
    # heights on the grid of corner offsets, six components' differences, then their transforms
    if kind == "tensor":
        px, py, nl, z = _grid(nx), _grid(ny), 1, 2
    else:
        px, py, nl, z = nx, ny, 2, 4
    build = nl * (px * py * (z * 300.0 + 6 * 27 * 2) + 6 * 2.5 * px * py * math.log2(px * py))
    moved = nl * nx * ny * 24 + 3 * nx * ny * 8 + (6 * 4 * (px // 2 + 1) * py if kind == "tensor" else 0)
    return dict(bytes=moved, flops=build + 9.0 * nl * 2.5 * px * py * math.log2(px * py))


class _Size:
    def __init__(self, side):
        self.nx = self.ny = side


# ---------------- the values in 64 bits ----------------
#
# The same physics on plain torch in double precision: the volume-averaged
# dipole tensor (closed forms of uniformly magnetised cuboids near, Gauss
# quadrature of the dipole kernel far, where the closed forms cancel), a
# zero-padded FFT convolution, and the pushes written out.

def _g1(x, y, z, d):
    t = lambda v: torch.clamp(v, min=1e-300)  # noqa: E731
    a = torch.atan(y * z / torch.copysign(t(x.abs() * d), x))
    return x * y * z * a + 0.5 * y * (z * z - x * x) * torch.log(t(d - y)) + 0.5 * z * (y * y - x * x) * torch.log(t(d - z)) \
        + (y * y + z * z - 2 * x * x) * d / 6


def _g2(x, y, z, d):
    t = lambda v: torch.clamp(v, min=1e-300)  # noqa: E731
    at = lambda p, q, r: torch.atan(p * q / torch.copysign(t(r.abs() * d), r))  # noqa: E731
    return -x * y * z * torch.log(t(d + x)) + z * (z * z - 3 * x * x) * torch.log(t(d + y)) / 6 + y * (y * y - 3 * x * x) * torch.log(t(d + z)) / 6 \
        + y * y * x * at(z, x, y) / 2 + z * z * x * at(x, y, z) / 2 + x ** 3 * at(y, z, x) / 6 + y * z * d / 3


_PAIRS = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))


def _near(i, j, dx, dy, zs, zo, rz):
    """Six components for cell offsets i, j (tensors); rz: observation minus source, lengths in units of dx."""
    n = [torch.zeros_like(i) for _ in range(6)]
    for c in range(64):
        b = [(c >> k & 1) - 0.5 for k in range(6)]
        x, y, z = i * dx + (b[0] - b[1]) * dx, j * dy + (b[2] - b[3]) * dy, torch.full_like(i, rz + b[4] * zo - b[5] * zs)
        d = torch.sqrt(x * x + y * y + z * z)
        s = 1.0 if sum(c >> k & 1 for k in range(6)) % 2 == 0 else -1.0
        v = (_g1(x, y, z, d), _g1(y, z, x, d), _g1(z, x, y, d), _g2(z, x, y, d), _g2(y, z, x, d), _g2(x, y, z, d))
        for k in range(6):
            n[k] += s * torch.where(d > 0, v[k], torch.zeros_like(d))
    return [v / (dx * dy * zo) for v in n]


def _pieces(a, b, n):
    """Nodes and weights of the distribution of (uniform of width a) - (uniform of width b)."""
    x, w = np.polynomial.legendre.leggauss(n)
    lo, hi = abs(a - b) / 2, (a + b) / 2
    cuts = [-hi, -lo, lo, hi] if lo > 1e-12 * hi else [-hi, 0.0, hi]
    u, q = [], []
    for p0, p1 in zip(cuts, cuts[1:]):
        xx = 0.5 * (p1 - p0) * x + 0.5 * (p1 + p0)
        u += list(xx)
        q += list(0.5 * (p1 - p0) * w * np.minimum(min(a, b), hi - np.abs(xx)) / (a * b))
    return u, q


def _far(i, j, dx, dy, zs, zo, rz):
    n = [torch.zeros_like(i) for _ in range(6)]
    for ux, wx in zip(*_pieces(dx, dx, 4)):
        for uy, wy in zip(*_pieces(dy, dy, 4)):
            for uz, wz in zip(*_pieces(zo, zs, 4)):
                r = (i * dx + ux, j * dy + uy, torch.full_like(i, rz + uz))
                r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
                f = wx * wy * wz * dx * dy * zs * r2 ** -2.5
                for k, (a, b) in enumerate(_PAIRS):
                    n[k] += f * (3 * r[a] * r[b] - (r2 if a == b else 0.0))
    return n


def _spectrum(px, py, dx, dy, zs, zo, rz):
    """Half spectrum of the six tensor components on the px x py grid (no images)."""
    unit = dx
    dx, dy, zs, zo, rz = 1.0, dy / unit, zs / unit, zo / unit, rz / unit
    dev = torch.device("cuda")
    f = lambda p: torch.arange(p, device=dev, dtype=torch.float64)  # noqa: E731
    total = [torch.zeros((py, px), device=dev, dtype=torch.float64) for _ in range(6)]
    # a slot half way round holds both of its offsets
    for sj in (0, 1):
        for si in (0, 1):
            i, j = f(px), f(py)
            i, j = torch.where(i > px // 2 - si, i - px, i), torch.where(j > py // 2 - sj, j - py, j)
            wi = torch.ones_like(i) if si == 0 else (i == -(px // 2)).double()
            wj = torch.ones_like(j) if sj == 0 else (j == -(py // 2)).double()
            ii, jj = i[None, :].expand(py, px), j[:, None].expand(py, px)
            near = (ii.abs() <= 7) & (jj.abs() <= 7)
            v = _far(torch.where(near, torch.full_like(ii, 8.0), ii), jj, dx, dy, zs, zo, rz)
            for k, w in enumerate(_near(ii[near], jj[near], dx, dy, zs, zo, rz)):
                v[k][near] = w
                total[k] += v[k] * wi[None, :] * wj[:, None]
    return torch.fft.rfft2(torch.stack(total))


_PAIR_OF = {(a, b): k for k, p in enumerate(_PAIRS) for a, b in (p, p[::-1])}


def _convolve(spec, src, ny, nx, py, px):
    """sum over b, layers s of N_ab(o, s) * M_b(s): src (R, L, 3, ny, nx) -> (R, O, 3, ny, nx); spec[o][s]: six half spectra."""
    s = torch.fft.rfft2(src, s=(py, px))
    out = []
    for row in spec:
        h = []
        for a in range(3):
            h.append(sum(n[_PAIR_OF[a, b]] * s[:, l, b] for l, n in enumerate(row) for b in range(3)))
        out.append(torch.stack(h, dim=1))
    return torch.fft.irfft2(torch.stack(out, dim=1), s=(py, px))[..., :ny, :nx]


def _heights(med):
    """z of each layer's centre, the last layer lowest."""
    z, out = 0.0, [0.0] * med.n_lay
    for l in reversed(range(med.n_lay)):
        out[l] = z + 0.5 * med.dz[l]
        z += med.dz[l] + med.il_space[l]
    return out


_M32 = 0xFFFFFFFF


def _signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _mulhi64(a, b):
    lo, hi = b & _M32, b >> 32
    al, ah = a & _M32, (a >> 32) & _M32
    t = ah * lo + ((al * lo >> 32) & _M32)
    u = al * hi + (t & _M32)
    return ah * hi + ((t >> 32) & _M32) + ((u >> 32) & _M32)


def _normals(fp, n, seed, step, layer):
    """Three standard normals per grain of the counter-based stream: Philox4x32-10 and 24-bit uniforms (FP32 runs) or Philox4x64-10 and 53-bit ones, Box-Muller."""
    g = torch.arange(n, device="cuda", dtype=torch.int64)
    full = lambda v: torch.full_like(g, _signed(v))  # noqa: E731
    if fp == 32:
        c = [g & _M32, full(step & _M32), full(step >> 32), full(layer)]
        k0, k1 = seed & _M32, (seed >> 32) ^ 0x6D726D
        for _ in range(10):
            p, q = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
            c = [((q >> 32) & _M32) ^ c[1] ^ k0, q & _M32, ((p >> 32) & _M32) ^ c[3] ^ k1, p & _M32]
            k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
        u = [((v >> 8).double() + 0.5) / 2.0 ** 24 for v in c]
        half = math.pi
    else:
        m0, m1 = 0xD2E7470EE14C6C93, 0xCA5A826395121157
        c = [g, full(step), full(layer), full(0)]
        k0, k1 = seed, 0x6D726D
        for _ in range(10):
            p, q = _mulhi64(c[0], m0), _mulhi64(c[2], m1)
            c = [q ^ c[1] ^ _signed(k0), c[2] * _signed(m1), p ^ c[3] ^ _signed(k1), c[0] * _signed(m0)]
            k0, k1 = (k0 + 0x9E3779B97F4A7C15) & (2 ** 64 - 1), (k1 + 0xBB67AE8584CAA73B) & (2 ** 64 - 1)
        u = [(((v >> 11) & (2 ** 53 - 1)).double() + 0.5) / 2.0 ** 53 for v in c]
        half = 0.0
    ra, rb = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    a, b = 2 * math.pi * u[1] - half, 2 * math.pi * u[3] - half
    return torch.stack([ra * torch.cos(a), ra * torch.sin(a), rb * torch.cos(b)])


def _cross(a, b):
    return torch.cross(a, b, dim=2)


def _dot(a, b):
    return (a * b).sum(2, keepdim=True)


class _Exact:
    """R runs of media with one geometry: fields (R, L, 3, ny, nx)."""

    def __init__(self, meds, seeds, fp):
        m = meds[0]
        self.med, self.meds, self.seeds, self.fp = m, meds, seeds, fp
        self.nx, self.ny, self.px, self.py, self.nl = m.nx, m.ny, _grid(m.nx), _grid(m.ny), m.n_lay
        z = _heights(m)
        self.spec = [[_spectrum(self.px, self.py, m.dx, m.dy, m.dz[s], m.dz[o], z[o] - z[s]) for s in range(self.nl)] for o in range(self.nl)]
        g = lambda f, c: torch.stack([torch.stack([torch.as_tensor(np.asarray(f(k, l), np.float64).reshape(self.ny, self.nx, c)).cuda()  # noqa: E731
                                                   for l, k in enumerate(x.layers)]) for x in meds]).permute(0, 1, 4, 2, 3).contiguous()
        self.m = torch.stack([torch.stack([torch.as_tensor(a.reshape(self.ny, self.nx, 3)).cuda() for a in x.m0]) for x in meds]).permute(0, 1, 4, 2, 3).contiguous()
        self.axis, self.hk, self.ms = g(lambda k, l: k.axis, 3), g(lambda k, l: k.hk[:, 0], 1), g(lambda k, l: k.ms, 1)
        self.vol, self.alpha = g(lambda k, l: k.vol, 1), g(lambda k, l: np.full(k.N, k.alpha), 1)
        self.gamma = m.layers[0].gamma
        self.hex = [float(k.hx[0]) if k.hx is not None else 0.0 for k in m.layers]
        if m.layers[0].llb:
            k = m.layers[0].llb
            self.mag = torch.ones_like(self.hk)
            self.spin, self.tc = k["spin"], g(lambda k, l: k.llb["tc"], 1)
            self.lam = g(lambda k, l: k.llb["lambda_ms"], 1) * (self.spin + 1) / self.spin

    def applied(self, l, t):
        k = self.med.layers[l]
        if k.head:
            h = k.head
            u = (torch.arange(self.nx, device="cuda", dtype=torch.float64) + 0.5) * self.med.dx - (h["x0"] + h["velocity"] * (t - h["t0"]))
            s = 1.0 if (h["pattern"] >> (math.floor((t - h["t0"]) / h["bit_time"]) % h["nbits"])) & 1 else -1.0
            a, b, z = u + 0.5 * h["gap"], u - 0.5 * h["gap"], h["z"]
            hx = s * h["hg"] / math.pi * (torch.atan(a / z) - torch.atan(b / z))
            hz = s * h["hg"] / (2 * math.pi) * torch.log((b * b + z * z) / (a * a + z * z))
            return torch.stack([hx, torch.zeros_like(hx), hz])[:, None, :]
        r = min(1.0, max(0.0, (t - k.t_start) / (k.t_end - k.t_start)))
        s = ((k.s_end - k.s_start) * r + k.s_start) * k.scale
        return torch.tensor(k.hdir, device="cuda", dtype=torch.float64)[:, None, None] * s

    def demag(self, m):
        return _convolve(self.spec, self.ms * m, self.ny, self.nx, self.py, self.px)

    def field(self, m, t):
        h = self.demag(m) + self.hk * _dot(m, self.axis) * self.axis
        for l in range(self.nl):
            n = m[:, l]
            h[:, l] += self.applied(l, t) + self.hex[l] * (n.roll(1, 2) + n.roll(-1, 2) + n.roll(1, 3) + n.roll(-1, 3))
            for o, c in ((l - 1, self.med.layers[l].uhx), (l + 1, self.med.layers[l].lhx)):
                if c is not None and 0 <= o < self.nl:
                    h[:, l] += float(c[2][0]) * m[:, o]
        return h

    def thermal(self, step):
        k = self.med.layers[0]
        if not k.thermal:
            return 0.0
        z = torch.stack([torch.stack([_normals(self.fp, self.nx * self.ny, s, step, l).reshape(3, self.ny, self.nx) for l in range(self.nl)]) for s in self.seeds])
        return z * torch.sqrt(2 * 1.380662e-16 * self.alpha * k.temperature / (self.gamma * self.ms * self.vol * DT))

    def heun(self, m, h, th):
        f = h + th
        t = _cross(m, f)
        return -self.gamma * DT / (1 + self.alpha ** 2) * (t + self.alpha * _cross(m, t))

    def implicit(self, m, f, dt):
        o = -0.5 * self.gamma * dt * f - self.alpha * m
        return m + 2 / (1 + _dot(o, o)) * _cross(m + _cross(m, o), o)

    def llb(self, m, mag, h, th):
        """d of the Landau-Lifshitz-Bloch Heun stage (|m| > 0)."""
        gk, T = 1.343427768e-4, self.med.layers[0].temperature
        e = h + self.lam * mag * m
        mh = torch.sqrt(_dot(e, e))
        e = e / mh
        x = gk * self.spin * mh / T
        lv, dlv = 1 / torch.tanh(x) - 1 / x, 1 / x ** 2 - 1 / torch.sinh(x) ** 2
        perp, par = self.alpha * (1 - self.lam * lv * T / (3 * mh * self.tc)), self.alpha * 2 * T / (3 * self.tc)
        th = th / torch.sqrt(self.alpha)
        tp = _dot(th, m) * m
        side = (th - tp) * torch.sqrt(torch.clamp(perp - par, min=0) / perp ** 2)
        q = -par * self.lam ** 2 / mh * self.gamma * DT * T * lv / (3 * dlv * self.tc) * (mag - lv * _dot(m, e))
        q = torch.copysign(torch.clamp(q.abs(), max=0.5), q)
        return -self.gamma * DT * (mag * _cross(m, h) + perp * _cross(m, _cross(m, h + side)) + tp * torch.sqrt(par)) + q * m

    def step(self, i, llg_type):
        unit = lambda v: v / torch.sqrt(_dot(v, v))  # noqa: E731
        t, m, th = i * DT, self.m, self.thermal(i)
        h = self.field(m, t)
        if self.med.layers[0].llb:
            d1 = self.llb(m, self.mag, h, th)
            w = m * self.mag + d1
            p = torch.sqrt(_dot(w, w))
            h = self.field(w / p, t + DT)
            w = m * self.mag + 0.5 * (d1 + self.llb(w / p, p, h, th))
            self.mag = torch.sqrt(_dot(w, w))
            self.m = w / self.mag
        elif llg_type == 2:
            self.m = self.implicit(m, h + th, DT)
        elif llg_type == -2:
            h = self.field(self.implicit(m, h + th, 0.5 * DT), t + 0.5 * DT)
            self.m = self.implicit(m, h + th, DT)
        else:
            d1 = self.heun(m, h, th)
            p = unit(m + d1)
            h = self.field(p, t + DT)
            self.m = unit(m + 0.5 * (d1 + self.heun(p, h, th)))
        self.h = h

    def mean(self, v):
        return (v * self.vol).sum((1, 3, 4)) / self.vol.sum((1, 3, 4))

    def grains(self, v, r, l):
        return v[r, l].permute(1, 2, 0).reshape(-1, v.shape[2])


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        e = _Exact([_medium(case, seed)], [seed], case["fp"])
        for i in range(case["steps"]):
            e.step(i, case["llg_type"])
        out = dict(mave=e.mean(e.m)[0], have=e.mean(e.h)[0], **{"m%d" % l: e.grains(e.m, 0, l) for l in range(e.nl)})
        if case["medium"] == "llb":
            out["mag"] = e.grains(e.mag, 0, 0)[:, 0]
        return out
    if kind == "batch":
        meds = _batch_media(case, seed)
        m, mave, have = [None] * len(meds), [None] * len(meds), [None] * len(meds)
        groups = {}
        for i, x in enumerate(meds):
            groups.setdefault(x.nx, []).append(i)
        for which in groups.values():
            for at in range(0, len(which), 8):
                part = which[at:at + 8]
                e = _Exact([meds[i] for i in part], [seed + i for i in part], 32)
                for i in range(case["steps"]):
                    e.step(i, case["llg_type"])
                for r, i in enumerate(part):
                    m[i], mave[i], have[i] = e.grains(e.m, r, 0), e.mean(e.m)[r], e.mean(e.h)[r]
        return dict(m=torch.cat(m), mave=torch.stack(mave), have=torch.stack(have))
    if kind == "tensor":
        med = media.mh_medium(case["nx"], ny=case["ny"], seed=seed)
        med.m0 = [_written(case["nx"], case["ny"], seed)]
        e = _Exact([med], [seed], case["fp"])
        return dict(h_demag=e.grains(e.demag(e.m), 0, 0))
    med = media.head_write_medium(case["nx"], case["ny"], seed=seed, prbs_seed=seed)
    nx, ny, z = case["nx"], case["ny"], _heights(med)
    top = z[0] + 0.5 * med.dz[0] + READBACK["zoff"] + 0.5 * READBACK["dzobs"]
    src = torch.stack([torch.as_tensor(_written(nx, ny, seed + l).astype(np.float32).astype(np.float64) * med.layers[l].ms[:, None]).reshape(ny, nx, 3).permute(2, 0, 1).cuda()
                       for l in range(2)])[None]
    spec = [[_spectrum(nx, ny, med.dx, med.dy, med.dz[l], READBACK["dzobs"], top - z[l]) for l in range(2)]]
    return dict(h=_convolve(spec, src, ny, nx, ny, nx)[0, 0])
