"""GPU parity of the direct-product transforms of lengths q p with a prime p
above 31 (csrc/prime_pass.cu): the smallest (37) and a large prime (251), both
tile widths, q = 1, 2, 3 and larger q, on the x-, y- and z-axis of the Born
loop (z as one pass, also behind the fused xy-pass) and in the centred 2D
transforms of odd fields, against the Bluestein path (ODT_KERNELS=generic).
Each transform carries single-precision rounding of a few units (2e-7 to 5e-7,
either way), six of them per iteration and the input / output stages: 1e-5
relative L2, the bound the suite has for Bluestein grids against its oracle
halved."""
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


@pytest.mark.parametrize("pad", [[37, 40, 44], [44, 37, 40], [44, 40, 37], [88, 88, 89], [41, 74, 111], [127, 40, 251],
                                 [185, 36, 41], [40, 202, 61], [48, 45, 254], [45, 37, 222]])
@pytest.mark.parametrize("acyclic", [True, False])
def test_prime_axes_match_bluestein(pad, acyclic):
    size = [n - 24 for n in pad]
    if not acyclic and max(pad) > 130:
        pytest.skip("one setting of the phase ramp is enough on the large grids")
    p = cases.params(size, [6, 6, 6], return_reflection=True, return_3D=True, iterations_number=6, acyclic=acyclic)
    RI = cases.sphere_phantom(size, [0.1] * 3, cases.NM, seed=sum(pad), n_spheres=2, radius_um=(0.3, 0.6))
    fields = cases.circle_fields(p, 3)
    (t1, r1, f1), sim = _solve(p, RI, fields, False)
    (t2, r2, f2), _ = _solve(p, RI, fields, True)
    assert sim == pad and np.isfinite(f1).all()
    for k in range(3):
        assert cbs.rel_l2(f1[..., k], f2[..., k]) < 1e-5
        assert cbs.rel_l2(t1[..., k], t2[..., k]) < 1e-5
        assert cbs.rel_l2(r1[..., k], r2[..., k]) < 3e-5
