"""GPU parity of the pipelined z-pass (csrc/z_pass.cu) at the edges of its
range: z lengths n = A R for the smallest and largest A and R, A = R, the
largest box (256 rows), A = 8 (kernels of their own) and an A above 10; planes
of an odd number of columns (8-byte copies instead of tiled ones) and planes
that are no multiple of the 16-column tile.  Against the generic tile kernels
(ODT_KERNELS=generic), whose transforms are the same up to the order of the
arithmetic: relative L2 5e-6, the bound the other pairs of passes have."""
import os

import numpy as np
import pytest

import cases
from oracle import cbs

pytestmark = pytest.mark.gpu


def _solve(p, RI, fields, generic):
    from inverse_solver_b200 import FORWARD_SOLVER_CONVERGENT_BORN

    old = os.environ.pop("ODT_KERNELS", None)
    if generic:
        os.environ["ODT_KERNELS"] = "generic"
    try:
        s = FORWARD_SOLVER_CONVERGENT_BORN(p)
        s.set_RI(RI)
        out = s.solve(fields)
        sim = s.sim_size
        s.delete()
    finally:
        os.environ.pop("ODT_KERNELS", None)
        if old is not None:
            os.environ["ODT_KERNELS"] = old
    return out, sim


# (x, y) padded 44 x 40 (even, 110 tiles), 45 x 39 (odd, a partial tile);
# z padded: 46 = 2*23, 49 = 7*7, 57 = 3*19, 62 = 2*31, 64 = 8*8, 85 = 5*17,
# 121 = 11*11, 145 = 5*29, 153 = 9*17, 248 = 8*31, 256 = 8*32 -> 16*16
@pytest.mark.parametrize("nz", [46, 49, 57, 62, 64, 85, 121, 145, 153, 248, 256])
@pytest.mark.parametrize("nx,ny", [(44, 40), (45, 39)])
def test_z_pass_matches_generic(nx, ny, nz):
    size = [nx - 24, ny - 24, nz - 24]
    p = cases.params(size, [6, 6, 6], return_3D=True, iterations_number=6)
    RI = cases.sphere_phantom(size, [0.1] * 3, cases.NM, seed=nz, n_spheres=2, radius_um=(0.3, 0.7))
    fields = cases.circle_fields(p, 3)
    (t1, _, f1), sim = _solve(p, RI, fields, False)
    (t2, _, f2), _ = _solve(p, RI, fields, True)
    assert sim == [nx, ny, nz]
    for k in range(3):
        assert cbs.rel_l2(t1[..., k], t2[..., k]) < 5e-6
        assert cbs.rel_l2(f1[..., k], f2[..., k]) < 5e-6
    assert np.isfinite(f1).all()
