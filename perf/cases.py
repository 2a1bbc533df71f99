"""Performance cases of the solvers: what a reconstruction program has this
framework do, through the public classes.

kinds
  solve     FORWARD_SOLVER_CONVERGENT_BORN with the scalar Green's function:
            one forward solve of a set of illuminations, from host arrays
            (``solve``) or device arrays (``solve_device``)
  vector    the same with the dyadic Green's function (two polarisations in
            and out, three field components)
  gradient  one gradient of the inverse solver: new forward and adjoint
            potentials from the current RI in device memory, forward and
            adjoint solves, misfit (set_RI_device, gradient_device)
  fista     a whole BACKWARD_SOLVER_MULTI.solve of a few outer iterations
            (gradients, TV proximal steps, momentum)
  bpm       FORWARD_SOLVER_BPM: one beam-propagation solve

listed() gives the cases, draw() more of the same ranges, prepare() the
inputs and solver objects a program holds before the call, run() one call,
work() its unavoidable bytes and operations, exact() its outputs in double
precision written in plain torch.
"""
import math

import numpy as np
import torch

from inverse_solver_b200.backward import BACKWARD_SOLVER_MULTI
from inverse_solver_b200.bpm import FORWARD_SOLVER_BPM
from inverse_solver_b200.forward import FORWARD_SOLVER_CONVERGENT_BORN

N_BG = 1.3355          # water
WAVELENGTH = 0.532     # um
NA = 1.2
RES = 0.1              # um per voxel
DEFAULT_EDGE = 6.0     # boundary thickness in wavelengths: 12 voxels a side
WIDE_EDGE = 8.0331     # 16 voxels a side
STEP, TV, INNER = 0.01, 7.5e-3, 100


# --------------------------------------------------------------- the cases
def _case(name, kind, size, waves, **more):
    c = dict(name=name, kind=kind, nx=size[0], ny=size[1], nz=size[2], waves=waves, edge=DEFAULT_EDGE,
             ri_max=1.46, host=False, volume=False)
    c.update(more)
    return c


def listed():
    return [
        # one bead, one wave, everything back on the host: a first look at a
        # sample, the smallest call
        _case("solve_64_1", "solve", (64, 64, 64), 1, edge=WIDE_EDGE, host=True, volume=True),
        # the small and the large grids of a request loop of mixed sizes
        _case("solve_96x96x64_16", "solve", (96, 96, 64), 16),
        _case("solve_192x192x96_8", "solve", (192, 192, 96), 8),
        # a full scan of a cell: 49 illuminations
        _case("solve_128_49", "solve", (128, 128, 128), 49),
        # a camera's own crop: odd sizes, a rectangular field, few waves
        _case("solve_101x84x45_6", "solve", (101, 84, 45), 6, ri_max=1.40),
        # an RI grid whose padded lengths are prime
        _case("solve_103_16", "solve", (103, 103, 103), 16, ri_max=1.42),
        # polarised illumination (the reference's default mode)
        _case("vector_64_4", "vector", (64, 64, 64), 4, ri_max=1.40),
        # one gradient of the iterative reconstruction (odd z, as it needs)
        _case("gradient_128x128x129_16", "gradient", (128, 128, 129), 16, ri_max=1.42),
        # the same on the largest reconstruction grid with a stochastic subset
        _case("gradient_192x192x129_4", "gradient", (192, 192, 129), 4, ri_max=1.42),
        # a short whole reconstruction of a small sample, TV steps included
        _case("fista_64x64x61_8", "fista", (64, 64, 61), 8, ri_max=1.40),
        # the weak-scattering solver on a full scan and on another grid
        _case("bpm_128_49", "bpm", (128, 128, 128), 49, ri_max=1.40),
        _case("bpm_192x192x96_16", "bpm", (192, 192, 96), 16, ri_max=1.40),
    ]


def _largest_prime(n):
    p, m = 1, 2
    while n > 1:
        while n % m == 0:
            p, n = m, n // m
        m += 1
    return p


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edge_px(edge):
    return int(math.floor(edge * WAVELENGTH / N_BG / (2 * RES) + 0.5))


def _padded(c):
    return [n + 2 * _edge_px(c["edge"]) for n in (c["nx"], c["ny"], c["nz"])]


def draw(rng):
    """Half of the sizes are the round ones that programs choose (multiples
    of 8), the others any number; most fields are square."""
    kind = rng.choice(["solve"] * 6 + ["vector", "gradient", "gradient", "fista", "bpm", "bpm"])

    def length(lo, hi, roundish):
        n = _log_int(rng, lo, hi)
        return max(8, 8 * int(round(n / 8))) if roundish else n

    while True:
        roundish = rng.random() < 0.5
        c = _case("", kind, (0, 0, 0), 1, ri_max=round(rng.uniform(1.36, 1.46), 3))
        del c["name"]
        if kind == "solve":
            c["nx"] = length(32, 192, roundish)
            c["ny"] = c["nx"] if rng.random() < 0.75 else length(32, 192, roundish)
            c["nz"] = length(24, 129, roundish)
            c["waves"] = _log_int(rng, 1, 49)
            c["edge"] = rng.choice([DEFAULT_EDGE, DEFAULT_EDGE, WIDE_EDGE])
            c["host"] = rng.random() < 0.25
            c["volume"] = rng.random() < 0.25 and c["waves"] <= 4
        elif kind == "vector":
            c["nx"] = c["ny"] = 4 * _log_int(rng, 8, 24)
            c["nz"] = length(24, 80, roundish)
            c["waves"] = _log_int(rng, 1, 8)
        elif kind == "gradient":
            c["nx"] = c["ny"] = length(48, 192, roundish)
            c["nz"] = _log_int(rng, 12, 64) * 2 + 1
            c["waves"] = _log_int(rng, 1, 24)
        elif kind == "fista":
            c["nx"] = c["ny"] = length(40, 96, roundish)
            c["nz"] = _log_int(rng, 12, 36) * 2 + 1
            c["waves"] = _log_int(rng, 2, 12)
        else:
            c["nx"] = length(64, 256, roundish)
            c["ny"] = c["nx"] if rng.random() < 0.75 else length(64, 256, roundish)
            c["nz"] = length(16, 160, roundish)
            c["waves"] = _log_int(rng, 1, 49)
            if max(_largest_prime(c["nx"]), _largest_prime(c["ny"])) > 31:   # refused by the solver
                continue
        p = _padded(c)
        worst = max(_largest_prime(n) for n in p + [c["nx"], c["ny"]])
        if kind == "vector" and worst > 31:   # refused by the solver
            continue
        cost = c["waves"] * p[0] * p[1] * p[2] * {"gradient": 2, "fista": 6, "vector": 3}.get(kind, 1)
        if cost <= 152 ** 3 * (6 if worst > 31 else 24):
            return c


# -------------------------------------------------------------- the inputs
def _phantom(c, seed):
    """Spheres of random size, place and RI with one-voxel edges; the last
    one has the case's highest RI and covers at least one voxel fully, so
    the iteration count follows from the case alone."""
    rng = np.random.default_rng([seed, 1])
    size = np.array([c["nx"], c["ny"], c["nz"]])
    ri = np.full(size, N_BG)
    ax = [np.arange(n) for n in size]
    for k in range(8):
        last = k == 7
        r = rng.uniform(0.08, 0.3) * size.min()
        ctr = rng.uniform(r, size - 1 - r)
        n = c["ri_max"] if last else rng.uniform(N_BG, c["ri_max"])
        ctr = np.round(ctr) if last else ctr
        d = np.sqrt((ax[0][:, None, None] - ctr[0]) ** 2 + (ax[1][None, :, None] - ctr[1]) ** 2
                    + (ax[2][None, None, :] - ctr[2]) ** 2)
        cover = np.clip(r - d + 0.5, 0, 1)
        ri = ri * (1 - cover) + n * cover
    return ri.astype(np.float32)


def _waves(c, seed, pols=1):
    """Plane waves on the field's k-grid: normal incidence and directions
    spread over 90 % of the aperture, [nx, ny, pols, waves] complex64."""
    rng = np.random.default_rng([seed, 2])
    nx, ny = c["nx"], c["ny"]
    out = np.empty((nx, ny, pols, c["waves"]), np.complex64)
    x, y = np.arange(nx)[:, None] / nx, np.arange(ny)[None, :] / ny
    for k in range(c["waves"]):
        rho = 0.0 if k == 0 else 0.9 * math.sqrt(rng.uniform()) * NA / WAVELENGTH
        phi = rng.uniform(0, 2 * math.pi)
        i1, i2 = round(rho * math.cos(phi) * nx * RES), round(rho * math.sin(phi) * ny * RES)
        w = np.exp(2j * math.pi * (i1 * x + i2 * y))
        pol = rng.uniform(0, 2 * math.pi)
        for q in range(pols):
            out[:, :, q, k] = w * (1 if pols == 1 else (math.cos(pol), math.sin(pol))[q])
    return np.asfortranarray(out)


def _measured(c, seed, waves):
    """Measured fields: the waves behind a smooth phase and absorption."""
    rng = np.random.default_rng([seed, 3])
    x, y = np.linspace(-1, 1, c["nx"])[:, None], np.linspace(-1, 1, c["ny"])[None, :]
    g = np.zeros((c["nx"], c["ny"]))
    for _ in range(4):
        a, b, s = rng.uniform(-0.6, 0.6, 2).tolist() + [rng.uniform(0.2, 0.5)]
        g = g + np.exp(-((x - a) ** 2 + (y - b) ** 2) / s ** 2)
    screen = np.exp((0.8j - 0.1) * g)
    return np.asfortranarray((waves * screen[:, :, None, None]).astype(np.complex64))


def _params(cls, c):
    return cls.get_default_parameters(dict(
        size=[c["nx"], c["ny"], c["nz"]], wavelength=WAVELENGTH, NA=NA, RI_bg=N_BG, resolution=[RES] * 3))


def _solver(c, **flags):
    p = _params(FORWARD_SOLVER_CONVERGENT_BORN, c)
    p.update(vector_simulation=c["kind"] == "vector", boundary_thickness=[c["edge"]] * 3, **flags)
    return FORWARD_SOLVER_CONVERGENT_BORN(p)


def _up(a):
    """A host array on the GPU in column-major order (shape reversed)."""
    return torch.from_numpy(np.ascontiguousarray(a.transpose(*range(a.ndim - 1, -1, -1)))).cuda()


class _Start:
    """Initial guess of a reconstruction."""

    def __init__(self, ri):
        self.ri = ri

    def solve(self, input_field, output_field):
        return self.ri


def prepare(case, seed):
    c, kind = case, case["kind"]
    ri = _phantom(c, seed)
    waves = _waves(c, seed, 2 if kind == "vector" else 1)
    if kind in ("solve", "vector"):
        s = _solver(c, return_reflection=c["volume"], return_3D=c["volume"])
        s.set_RI(ri)
        if c["host"]:
            return dict(case=c, solver=s, waves=waves)
        fin = _up(waves)
        return dict(case=c, solver=s, fin=fin, trans=torch.empty_like(fin),
                    ref=torch.empty_like(fin) if c["volume"] else None,
                    vol=torch.empty((c["waves"], s.pole_num, c["nz"], c["ny"], c["nx"]), dtype=torch.complex64,
                                    device="cuda") if c["volume"] else None)
    if kind == "gradient":
        s = _solver(c, return_reflection=True, return_3D=True)
        start = (0.5 * (ri + np.float32(N_BG))).astype(np.complex64)
        return dict(case=c, solver=s, ri=_up(start), fin=_up(waves), meas=_up(_measured(c, seed, waves)),
                    grad=torch.empty((c["nz"], c["ny"], c["nx"]), dtype=torch.complex64, device="cuda"))
    if kind == "fista":
        fp = _params(FORWARD_SOLVER_CONVERGENT_BORN, c)
        fp.update(vector_simulation=False, boundary_thickness=[c["edge"]] * 3, return_reflection=True, return_3D=True)
        start = (0.5 * (ri + np.float32(N_BG))).astype(np.float32)
        bp = _params(BACKWARD_SOLVER_MULTI, c)
        bp.update(forward_solver=FORWARD_SOLVER_CONVERGENT_BORN, forward_solver_parameters=fp,
                  init_solver=_Start(start), step=STEP, tv_param=TV, inner_itt=INNER, itter_max=3,
                  use_non_negativity=True, nmin=N_BG, nmax=1.5)
        return dict(case=c, solver=BACKWARD_SOLVER_MULTI(bp), waves=waves, meas=_measured(c, seed, waves))
    s = FORWARD_SOLVER_BPM(_params(FORWARD_SOLVER_BPM, c))
    s.set_RI(ri)
    fin = _up(waves[:, :, 0])
    return dict(case=c, solver=s, fin=fin, trans=torch.empty_like(fin))


def run(state):
    c, s = state["case"], state["solver"]
    if c["kind"] in ("solve", "vector"):
        if c["host"]:
            return s.solve(state["waves"])
        s.solve_device(state["fin"], trans=state["trans"], ref=state["ref"], field3d=state["vol"])
        return state["trans"], state["ref"], state["vol"]
    if c["kind"] == "gradient":
        s.set_RI_device(state["ri"])
        s.set_RI_device(state["ri"], adjoint=True)
        err = s.gradient_device(state["fin"], state["meas"], state["grad"])
        return state["grad"], err
    if c["kind"] == "fista":
        return s.solve(state["waves"], state["meas"])
    s.solve_device(state["fin"], state["trans"])
    return state["trans"]


# ---------------------------------------------------------------- the work
def _born_iterations(c, ri_max):
    """Bornmax of the default setting: the padded diagonal over the step."""
    k = 2 * math.pi * N_BG / WAVELENGTH
    eps = 1.01 * k ** 2 * ((ri_max / N_BG) ** 2 - 1)
    diag = math.sqrt(sum((n * RES) ** 2 for n in _padded(c)))
    return 2 * math.ceil(diag / (2 * k / eps) / 2 + 1)


def work(case):
    """Inputs and outputs once; the transforms of the series (two 3D FFTs an
    iteration) or of the slices (two 2D FFTs a slice), 5 n log2 n each, with
    the products around them."""
    c = case
    plane, vol = c["nx"] * c["ny"], c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "bpm":
        n = plane * c["waves"]
        return {"bytes": 8 * (2 * n + vol), "flops": c["nz"] * n * (10 * math.log2(plane) + 30)}
    comps, pols = (3, 2) if c["kind"] == "vector" else (1, 1)
    p = _padded(c)
    n = p[0] * p[1] * p[2]
    mid = 0.5 * (c["ri_max"] + N_BG)
    solves = {"gradient": 2, "fista": 6}.get(c["kind"], 1)
    its = _born_iterations(c, c["ri_max"] if solves == 1 else mid)
    flops = solves * c["waves"] * comps * its * n * (10 * math.log2(n) + 40)
    tables = 2 * 4 * vol * solves            # refocusing and projection kernels on the doubled field
    io = 2 * plane * pols * c["waves"]
    if c["kind"] == "fista":
        flops += 3 * INNER * vol * 40
        return {"bytes": 8 * (tables + io + 2 * vol), "flops": flops}
    if c["kind"] == "gradient":
        return {"bytes": 8 * (tables + io + 2 * vol), "flops": flops}
    outs = c["waves"] * (vol * comps + plane * pols) if c["volume"] else 0
    return {"bytes": 8 * (tables + vol + io + outs), "flops": flops}


# ------------------------------------------------------- double precision
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    a = torch.as_tensor(np.asarray(a)).to(_dev())
    return a.to(torch.complex128) if a.is_complex() else a.double()


def _centred(x, dims, inverse=False):
    x = torch.fft.ifftshift(x, dim=dims)
    x = (torch.fft.ifftn if inverse else torch.fft.fftn)(x, dim=dims)
    return torch.fft.fftshift(x, dim=dims)


def _coor(n):
    return (torch.arange(n, dtype=torch.float64, device=_dev()) - n // 2) / (RES * n)


K0N, KMAX = N_BG / WAVELENGTH, NA / WAVELENGTH


def _pupil(nx, ny):
    """(|k_xy|, k_z, inside the aperture) on the centred field spectrum."""
    kxy = torch.sqrt(_coor(nx)[:, None] ** 2 + _coor(ny)[None, :] ** 2)
    return kxy, torch.sqrt(torch.clamp(K0N ** 2 - kxy ** 2, min=0)), kxy < KMAX


_ZEROS = []


def _bessel_zeros(n):
    """First n positive zeros of J0 (McMahon's estimate and Newton steps)."""
    if not _ZEROS:
        b = (torch.arange(1, n + 1, dtype=torch.float64, device=_dev()) - 0.25) * math.pi
        r = b + 1 / (8 * b) - 31 / (384 * b ** 3)
        for _ in range(5):
            r = r + torch.special.bessel_j0(r) / torch.special.bessel_j1(r)
        _ZEROS.append(r)
    return _ZEROS[0]


def _truncated_green(out, refocus):
    """Free-space Green's function (or refocusing kernel) truncated in x-y,
    Fourier in all axes, on an `out` grid: a band-limited radial profile from
    a discrete Hankel transform, interpolated onto an oversized grid that is
    cropped in space."""
    s = [v * 1.1 * math.sqrt(2) + 10 for v in out[:2]] + [out[2] + 10]
    side = math.ceil(max(s[0] * RES, s[1] * RES) / RES)
    big = [side, side, s[2]]
    nz = big[2]
    roots = _bessel_zeros(40001)
    top, c = roots[-1], roots[:-1]
    samples = len(c)
    cropping = math.hypot(side, side) * 2 / (2 * samples)
    pos = int(torch.argmin(torch.abs(c - c[-1] * cropping))) + 1
    j1 = torch.abs(torch.special.bessel_j1(c))
    kern, rad, scale = 2 * math.pi / top * j1, j1, math.sqrt(2 / top) / j1
    kxy = _pupil(side, side)[0]
    h = c / c[-1] * (kxy.max() * 2)
    hz = torch.sqrt(torch.clamp(K0N ** 2 - h ** 2, min=0))
    inside = h < KMAX
    ratio = (nz - 5) / nz
    g = torch.sinc((hz[:, None] - _coor(nz)[None, :]) * (RES * nz) * ratio) * ratio * inside[:, None]
    g = g.to(torch.complex128)
    if not refocus:
        g = g / (hz + (~inside).double())[:, None] / (4j * math.pi)
    nk = c[:pos] / c[pos - 1]
    band = (nk < 0.9).double() + ((nk < 1) & (nk > 0.9)).double() * (1 - nk) * 10
    m = scale[:pos, None] * scale[None, :] * torch.special.bessel_j0(c[:pos, None] / top * c[None, :])
    m = m.to(torch.complex128)
    img = (m @ (g / rad[:, None])) * kern[:pos, None]
    g = (m.T @ (img * band[:, None] / kern[:pos, None])) * rad[:, None]
    near = torch.clamp(torch.searchsorted(h, kxy.reshape(-1)), min=1)
    near2 = torch.clamp(torch.where(h[near - 1] < kxy.reshape(-1), near + 1, near), max=samples)
    w = (kxy.reshape(-1) - h[near - 1]) / (h[near2 - 1] - h[near - 1])
    w = torch.where(near2 == near, torch.ones_like(w), w)
    res = torch.empty((out[0], out[1], nz), dtype=torch.complex128, device=_dev())
    o = [side // 2 - out[0] // 2, side // 2 - out[1] // 2, nz // 2 - out[2] // 2]
    for z in range(nz):
        p = g[near - 1, z] * w + g[near2 - 1, z] * (1 - w)
        p = _centred(p.reshape(side, side) * (nz / RES ** 2), (0, 1), True)
        res[:, :, z] = _centred(p[o[0]:o[0] + out[0], o[1]:o[1] + out[1]], (0, 1))
    res = _centred(res, (2,), True)[:, :, o[2]:o[2] + out[2]]
    return _centred(res, (2,))


class _Born:
    """The convergent Born solver in double precision: the series of
    FORWARD_SOLVER_CONVERGENT_BORN.m term by term."""

    def __init__(self, c):
        self.c = c
        self.vec = c["kind"] == "vector"
        nx, ny, nz = self.size = [c["nx"], c["ny"], c["nz"]]
        conv = [2 * nx, 2 * ny, nz]
        self.refocus = _centred(_centred(_truncated_green(conv, True), (0, 1, 2), True), (0, 1)) * RES ** 2
        k = _centred(_truncated_green(conv, False), (0, 1, 2), True)
        self.k_trans, self.k_ref = _centred(k.conj(), (0, 1)), _centred(k, (0, 1))
        self.kxy, kz, self.inside = _pupil(nx, ny)
        cos = kz / K0N
        one = torch.ones_like(cos)
        self.p_in = self.inside / torch.sqrt(torch.where(self.inside, cos, one))
        self.p_out = self.inside * torch.sqrt(cos)
        px = _edge_px(c["edge"])
        self.pad = _padded(c)
        self.roi = tuple(slice(px, px + n) for n in self.size)
        mask, ramp = 1, 1
        self.q = []
        for j, n in enumerate(self.pad):
            shp = [1, 1, 1]
            shp[j] = n
            i = torch.arange(1, n + 1, dtype=torch.float64, device=_dev())
            x = torch.roll(torch.abs(i - (n // 2 + 1) + 0.5) - 0.5, -(n // 2)) / (px - 0.5)
            mask = mask * torch.clamp(x, max=1).reshape(shp)
            x = torch.exp(-0.5j * math.pi * (i - 1) / n)
            ramp = ramp * (x / x[n // 2]).reshape(shp)
            self.q.append(torch.fft.ifftshift(_coor(n) + 0.25 / (RES * n)).reshape(shp))
        self.mask, self.ramp = mask, ramp
        if self.vec:
            self._polarisation(nx)

    def _polarisation(self, n):
        k = _coor(n) / K0N
        kx, ky = torch.broadcast_tensors(k[:, None], k[None, :])
        kz = torch.sqrt(torch.clamp(1 - kx ** 2 - ky ** 2, min=0))
        rho = torch.sqrt(kx ** 2 + ky ** 2)
        ok = rho > 0
        ux = torch.where(ok, kx / torch.where(ok, rho, 1.0), 1.0)
        uy = torch.where(ok, ky / torch.where(ok, rho, 1.0), 0.0)
        nrm = torch.sqrt(rho ** 2 + kz ** 2)
        s = torch.stack([kx, ky, kz]) / nrm
        rad = torch.stack([ux, uy])
        t = -(s[:2] * rad).sum(0) * s
        t[:2] += rad
        live = kz > 0
        t = t / torch.where(live, torch.sqrt((t ** 2).sum(0)), 1.0)
        self.rad, self.perp, self.tan, self.live = rad, torch.stack([uy, -ux]), t, live

    def set_ri(self, ri):
        k2 = (2 * math.pi * K0N) ** 2
        self.pot = k2 * (ri ** 2 / N_BG ** 2 - 1)
        eps = self.eps = 1.01 * float(self.pot.abs().max())
        v = torch.zeros(self.pad, dtype=torch.complex128, device=_dev())
        v[self.roi] = self.pot
        self.v = v - 1j * eps
        step = 2 * (2 * math.pi * K0N) / eps
        diag = math.sqrt(sum((n * RES) ** 2 for n in self.pad))
        self.iters = 2 * math.ceil(diag / step / 2 + 1)
        self.greens = []
        for odd in (False, True):
            q = [self._flip(x) if odd else x for x in self.q]
            g = 1 / (4 * math.pi ** 2 * (q[0] ** 2 + q[1] ** 2 + q[2] ** 2) - k2 - 1j * eps)
            self.greens.append((g, [x / K0N for x in q]))
        self.absorb = k2 / (k2 + 1j * eps)

    @staticmethod
    def _flip(x):
        """x(-k) on an FFT-ordered axis (the one longer than 1)."""
        d = max(range(3), key=lambda i: x.shape[i])
        return torch.roll(torch.flip(x, (d,)), 1, d)

    def _propagate(self, psi, it):
        odd = it % 2 == 1
        g, rad = self.greens[odd]
        ramp = self.ramp.conj() if odd else self.ramp
        f = torch.fft.fftn(psi * ramp, dim=(-3, -2, -1))
        if self.vec:
            dot = rad[0] * f[0] + rad[1] * f[1] + rad[2] * f[2]
            f = torch.stack([f[i] - self.absorb * rad[i] * dot for i in range(3)])
        return torch.fft.ifftn(g * f, dim=(-3, -2, -1)) * ramp.conj()

    def volume(self, spec):
        """Total field of one input spectrum [(3,) nx, ny] in the RI grid."""
        nx, ny, _ = self.size
        a, b = nx - nx // 2, ny - ny // 2
        lead = spec.shape[:-2]
        s = torch.zeros(lead + (2 * nx, 2 * ny), dtype=torch.complex128, device=_dev())
        s[..., a:a + nx, b:b + ny] = _centred(spec, (-2, -1), True)
        s = _centred(s, (-2, -1))
        inc = _centred(s[..., None] * self.refocus, (-3, -2), True)[..., a:a + nx, b:b + ny, :]
        c = 1j / self.eps
        at = (Ellipsis,) + self.roi
        src = torch.zeros(lead + tuple(self.pad), dtype=torch.complex128, device=_dev())
        src[at] = 0.5 * c * self.pot * inc
        total = last = held = None
        for it in range(1, self.iters + 1):
            if it <= 2:
                last = self.v * self._propagate(src, it) * self.mask
                total, held = (last, last) if it == 1 else (total + last, held)
                continue
            psi = c * last * self.v
            last = (last - psi + self.v * self._propagate(psi, it)) * self.mask
            total = total + last
            if it == 3:
                last = last + held
        return total[at] + inc

    def spectrum(self, wave):
        """Input spectrum of one wave [pols, nx, ny] with the pupil applied."""
        f = _centred(wave, (-2, -1)) * self.p_in
        if not self.vec:
            return f[0]
        f = f * self.live
        out = (f * self.rad).sum(0) * self.tan
        out[:2] += (f * self.perp).sum(0) * self.perp
        return out

    def project(self, vol, spec, reflected=False):
        """Transmitted (with the input spectrum) or reflected field [pols, nx, ny]."""
        nx, ny, nz = self.size
        a, b = nx - nx // 2, ny - ny // 2
        e = torch.zeros(vol.shape[:-3] + (2 * nx, 2 * ny, nz), dtype=torch.complex128, device=_dev())
        e[..., a:a + nx, b:b + ny, :] = vol * self.pot * RES ** 3
        e = (_centred(e, (-3, -2)) * (self.k_ref if reflected else self.k_trans)).sum(-1)
        f = _centred(_centred(e, (-2, -1), True)[..., a:a + nx, b:b + ny], (-2, -1))
        f = (f if reflected else f + spec) * self.p_out
        if not self.vec:
            return _centred(f, (-2, -1), True)[None]
        tan = self.tan.clone()
        tan[2] *= -1 if reflected else 1
        f = f * self.live
        f = (f * tan).sum(0) * self.rad + (f[:2] * self.perp).sum(0) * self.perp
        return _centred(f, (-2, -1), True)

    def gradient(self, ri, waves, meas):
        """Mean gradient [nx, ny, nz] and misfit; waves, meas [n, nx, ny]."""
        self.set_ri(ri)
        vols, diffs = [], []
        for w, m in zip(waves, meas):
            s = self.spectrum(w[None])
            vols.append(self.volume(s))
            diffs.append(self.project(vols[-1], s)[0] - m)
        self.set_ri(torch.flip(ri, (2,)).conj())
        grad = 0
        for v, d in zip(vols, diffs):
            adj = self.volume(self.spectrum(d.conj()[None]))
            grad = grad + v.conj() * torch.flip(adj.conj(), (2,))
        return -1j * grad / len(vols), float(sum((d.abs() ** 2).sum() for d in diffs))


def _tv_prox(x, lam, lo, hi):
    """TV proximal step of a real volume by dual FISTA, clipped to [lo, hi]."""
    def div(p):
        return sum(p[k] - torch.roll(p[k], 1, k) for k in range(3))

    def primal(r):
        return torch.clamp(x - lam * div(r), lo, hi)

    p = [torch.zeros_like(x) for _ in range(3)]
    r, t = p, 1.0
    for _ in range(INNER):
        old, u = p, primal(r)
        p = [r[k] + (u - torch.roll(u, -1, k)) / (12 * lam) for k in range(3)]
        a = torch.sqrt(torch.clamp(p[0] ** 2 + p[1] ** 2 + p[2] ** 2, min=1))
        p = [v / a for v in p]
        t_new = (1 + math.sqrt(1 + 4 * t ** 2)) / 2
        r = [p[k] + (t - 1) / t_new * (p[k] - old[k]) for k in range(3)]
        t = t_new
    return primal(p)


def _exact_fista(c, ri, waves, meas):
    b = _Born(c)
    n2 = N_BG ** 2
    ri = 0.5 * (ri + np.float32(N_BG)).astype(np.float64)
    ri = _t(ri.astype(np.float32)).to(torch.complex128)
    u = x = ri ** 2 / n2 - 1
    t = 1.0
    for _ in range(3):
        grad, _ = b.gradient(ri, waves, meas)
        s = _tv_prox((u - STEP * grad).real, TV * STEP, 0.0, 1.5 ** 2 / n2 - 1)
        t_new = (1 + math.sqrt(1 + 4 * t ** 2)) / 2
        u = s + (t - 1) / t_new * (s - x)
        x, t = s, t_new
        ri = N_BG * torch.sqrt(u.to(torch.complex128) + 1)
    return ri


def _exact_bpm(c, ri, waves):
    """[waves, ny, nx], as solve_device lays it out."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    _, kz, inside = _pupil(nx, ny)
    screen = 2j * math.pi / WAVELENGTH * (ri - N_BG) * RES
    step = torch.fft.ifftshift(torch.exp(2j * math.pi * kz * RES) * inside)
    out = []
    for w in waves:
        f = _centred(w, (0, 1))
        # the peak of a plane wave's spectrum, in column-major order
        cos = (kz / K0N).T.reshape(-1)[int(torch.argmax(f.abs().T.reshape(-1)))]
        f = torch.fft.fft2(_centred(f * torch.exp(2j * math.pi * kz * RES * (-(nz // 2) - 1)), (0, 1), True))
        for z in range(nz):
            f = torch.fft.fft2(torch.fft.ifft2(f * step) * torch.exp(screen[:, :, z] / cos))
        f = _centred(torch.fft.ifft2(f), (0, 1)) * torch.exp(2j * math.pi * kz * RES * (-(nz - nz // 2 - 1)))
        out.append(_centred(f, (0, 1), True).T)
    return torch.stack(out)


def exact(case, seed):
    c, kind = case, case["kind"]
    ri = _phantom(c, seed)
    host = _waves(c, seed, 2 if kind == "vector" else 1)
    waves = _t(host).permute(3, 2, 0, 1).contiguous()           # [n, pols, nx, ny]
    if kind == "bpm":
        return _exact_bpm(c, _t(ri), waves[:, 0])
    if kind in ("gradient", "fista"):
        meas = _t(_measured(c, seed, host)).permute(3, 2, 0, 1)[:, 0]
        if kind == "fista":
            return _exact_fista(c, ri, waves[:, 0], meas)
        start = _t((0.5 * (ri + np.float32(N_BG))).astype(np.float32)).to(torch.complex128)
        grad, err = _Born(c).gradient(start, waves[:, 0], meas)
        return grad.permute(2, 1, 0), err
    b = _Born(c)
    b.set_ri(_t(ri))
    trans, ref, vol = [], [], []
    for w in waves:
        s = b.spectrum(w)
        v = b.volume(s)
        trans.append(b.project(v, s))
        if c["volume"]:
            ref.append(b.project(v, s, True))
            vol.append(v if b.vec else v[None])
    # device arrays [n, pols, ny, nx], host arrays [nx, ny, pols, n]
    trans, ref, vol = (torch.stack(v) if v else None for v in (trans, ref, vol))
    if c["host"]:
        flip = lambda v, axes: v if v is None else v.permute(*axes)  # noqa: E731
        return flip(trans, (2, 3, 1, 0)), flip(ref, (2, 3, 1, 0)), flip(vol, (2, 3, 4, 1, 0))
    return trans.transpose(2, 3), None if ref is None else ref.transpose(2, 3), \
        None if vol is None else vol.permute(0, 1, 4, 3, 2)
