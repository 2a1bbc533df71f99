"""The two fused passes per slice of the beam-propagation solver (every plane
without the 3D output except 128 x 128) on samples with contrast and
absorption that differ in every slice.

Against the oracle and against the separate launches (ODT_KERNELS=generic) of
the same call within rel-L2 1e-5, the bound of the other beam-propagation
tests: sides of a few points, of one radix (29, 31, 8), odd ones, ones with the
large radices 23 and 29, above 512 and above 1280 points (8 and 4 pencils per
tile), line and column counts that are no multiple of the tiles.

Rounding, against a double-precision march on the solver's own
single-precision tables: what constants and scales rounded to float add up
over the slices is about half as much in the fused passes (split constants,
exact scales), and it is half of the separate launches' error or more, so over
several sizes (on a single one either side's contributions may happen to
cancel) the error is below 0.8 of theirs in the geometric mean."""
import numpy as np
import pytest
import scipy.fft as sfft

import cases
from oracle import bpm, cbs

pytestmark = pytest.mark.gpu


def _solver(size, cos_correction=True, absorbing=True):
    from inverse_solver_b200 import FORWARD_SOLVER_BPM

    p = bpm.bpm_default_parameters(dict(size=list(size), wavelength=cases.LAM, NA=1.2, RI_bg=cases.NM,
                                        resolution=[0.1] * 3, vector_simulation=False, cos_correction=cos_correction))
    rng = np.random.default_rng(sum(size))
    ri = cases.NM + 0.1 * rng.random(size)
    if absorbing:
        ri = ri + 0.01j * rng.random(size)
    ri = ri.astype(np.complex64 if absorbing else np.float32)
    s = FORWARD_SOLVER_BPM(p)
    s.set_RI(ri)
    return s, p, ri


def _waves(size, n):
    """Plane waves of the field's k-grid, normal incidence first, inside the aperture."""
    x, y = np.arange(size[0])[:, None] / size[0], np.arange(size[1])[None, :] / size[1]
    out = np.empty((size[0], size[1], 1, n), np.complex64)
    for k in range(n):
        i1, i2 = round(0.08 * k * size[0]), round(-0.05 * k * size[1])
        out[:, :, 0, k] = np.exp(2j * np.pi * (i1 * x + i2 * y))
    return out


def worst(a, b):
    return max(cbs.rel_l2(a[..., k], b[..., k]) for k in range(a.shape[-1]))


@pytest.mark.parametrize("cos_correction", [True, False])
@pytest.mark.parametrize("size", [[8, 6, 5], [32, 28, 6], [29, 31, 5], [45, 50, 8], [58, 46, 6], [192, 96, 6], [640, 36, 4],
                                  [36, 640, 4], [1296, 24, 3], [24, 1296, 3], [50, 44, 1]])
def test_fused_passes_match_oracle_and_separate_launches(size, cos_correction, monkeypatch):
    s, p, ri = _solver(size, cos_correction)
    f = _waves(size, 3)
    t, _, _ = s.solve(f)
    monkeypatch.setenv("ODT_KERNELS", "generic")
    tg, _, _ = s.solve(f)
    monkeypatch.delenv("ODT_KERNELS")
    o = bpm.ForwardSolverBPM(p, single=True)
    o.set_RI(ri)
    ot, _, _ = o.solve(f)
    assert worst(t, tg) < 1e-5
    assert worst(t, ot) < 1e-5


def _double(s, f):
    c, axes = np.complex128, (0, 1)
    pre, post = (a.astype(c)[:, :, None] for a in s._phases())
    x = cbs.fftc2(f[:, :, 0].astype(c))
    ct = np.asarray(s.utility.cos_theta, np.float32).ravel(order="F").astype(float)
    ic = 1 / ct[np.abs(x).reshape(-1, x.shape[2], order="F").argmax(0)]
    x = sfft.fft2(cbs.fftc2(x * pre, inverse=True), axes=axes)
    rk, fm = s.refocus_kernel.astype(c)[:, :, None], s.field_multiplier.astype(c)
    for z in range(fm.shape[2]):
        x = sfft.ifft2(x * rk, axes=axes) * np.exp(fm[:, :, z, None] * ic)
        x = sfft.fft2(x, axes=axes)
    return cbs.fftc2(cbs.fftc2(sfft.ifft2(x, axes=axes)) * post, inverse=True)[:, :, None]


def test_fused_passes_round_better_than_separate_launches(monkeypatch):
    ratio = []
    for size in ([64, 64, 64], [192, 192, 96], [100, 90, 64], [128, 120, 96], [160, 160, 96], [108, 81, 64]):
        s, p, _ = _solver(size, absorbing=False)
        s.set_RI(cases.sphere_phantom(size, [0.1] * 3, cases.NM, seed=1, n_spheres=4, radius_um=(0.5, 1.2)))
        f = cases.circle_fields(p, 3)
        ref = _double(s, f)
        t, _, _ = s.solve(f)
        monkeypatch.setenv("ODT_KERNELS", "generic")
        tg, _, _ = s.solve(f)
        monkeypatch.delenv("ODT_KERNELS")
        ratio.append(cbs.rel_l2(t, ref) / cbs.rel_l2(tg, ref))
    print("fused / separate:", ["%.2f" % r for r in ratio])
    assert np.exp(np.mean(np.log(ratio))) < 0.8
