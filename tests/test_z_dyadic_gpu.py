"""GPU parity of the dyadic z-pass of any length (csrc/z_dyadic.cu) at the edges
of its range: z lengths n = A R with the smallest and largest A and R, A = R, A
above 10 and the largest number of rows, behind planes of an even number of
columns (16-byte copies; square ones in the fused xy-pass's order), of an odd
number (8-byte copies) and of a partial last tile.  Against the generic tile
kernels: relative L2 5e-6, the bound of the other pairs of passes."""
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


@pytest.mark.parametrize("n,nz", [(40, 46), (40, 49), (45, 57), (45, 121), (50, 62), (88, 88), (50, 85), (42, 155),
                                  (45, 152), (40, 256)])
def test_z_dyadic_matches_generic(n, nz):
    size = [n - 24, n - 24, nz - 24]
    p = cases.params(size, [6, 6, 6], return_reflection=True, return_3D=True, iterations_number=6)
    p["vector_simulation"] = True
    RI = cases.sphere_phantom(size, [0.1] * 3, cases.NM, seed=nz, n_spheres=2, radius_um=(0.3, 0.7))
    fields = cases.circle_fields(p, 2)
    fields = np.concatenate([fields, 0.5j * fields], axis=2)
    (t1, r1, f1), sim = _solve(p, RI, fields, False)
    (t2, r2, f2), _ = _solve(p, RI, fields, True)
    assert sim == [n, n, nz] and np.isfinite(f1).all()
    for k in range(2):
        assert cbs.rel_l2(t1[..., k], t2[..., k]) < 5e-6
        assert cbs.rel_l2(f1[..., k], f2[..., k]) < 5e-6
