"""GPU parity of the pipelined y-FFTs of any length (csrc/y_pass.cu) on
rectangular planes: y lengths n = A R with A = 2 and 3 (tiles of 32 columns),
A = R, A = 8 (kernels of their own), A above 10 and the largest box; planes of
an even and an odd number of columns (tiled and 8-byte copies) that are no
multiple of a tile.  Against the generic tile kernels: relative L2 5e-6, the
bound of the other pairs of passes; dyadic solves take the same passes."""
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


@pytest.mark.parametrize("ny", [46, 49, 57, 64, 96, 108, 121, 145, 155, 248, 256])
@pytest.mark.parametrize("nx", [50, 45])
def test_y_pass_matches_generic(nx, ny):
    size = [nx - 24, ny - 24, 16]
    p = cases.params(size, [6, 6, 6], return_3D=True, iterations_number=6)
    RI = cases.sphere_phantom(size, [0.1] * 3, cases.NM, seed=ny, n_spheres=2, radius_um=(0.3, 0.7))
    fields = cases.circle_fields(p, 3)
    (t1, _, f1), sim = _solve(p, RI, fields, False)
    (t2, _, f2), _ = _solve(p, RI, fields, True)
    assert sim == [nx, ny, 40] and np.isfinite(f1).all()
    for k in range(3):
        assert cbs.rel_l2(t1[..., k], t2[..., k]) < 5e-6
        assert cbs.rel_l2(f1[..., k], f2[..., k]) < 5e-6
