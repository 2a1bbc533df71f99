"""GPU parity of the fused xy-pass (csrc/born_xy.cu) on the planes that
tests/test_xy_gpu.py does not reach: the smallest (40 points, R = 5), planes
of several CTAs per SM (56, 64, 72, 80 points) and the two-CTA clusters of 168
to 224 points (even and odd R, the largest), for scalar and dyadic solves,
against the separate passes (ODT_XY=0): relative L2 5e-6, the bound between
these passes on the benchmark's grid; and a series of 2 iterations, whose last
pass adds X(1) (see BornArgs in csrc/cbs_kernels.cuh)."""
import os

import numpy as np
import pytest

import cases
from oracle import cbs

pytestmark = pytest.mark.gpu


def _solve(p, RI, fields, xy):
    from inverse_solver_b200 import FORWARD_SOLVER_CONVERGENT_BORN

    old = os.environ.get("ODT_XY")
    os.environ["ODT_XY"] = "1" if xy else "0"
    try:
        s = FORWARD_SOLVER_CONVERGENT_BORN(p)
        s.set_RI(RI)
        s.set_profiling(True)
        out = s.solve(fields)
        used = {k for k, (ms, n) in s.kernel_times().items() if n > 0}
        s.delete()
    finally:
        os.environ.pop("ODT_XY", None)
        if old is not None:
            os.environ["ODT_XY"] = old
    assert ("born_xy_edge" in used) == xy
    return out


@pytest.mark.parametrize("n,iters,vector", [(40, 6, False), (56, 6, False), (64, 6, False), (72, 6, False),
                                            (80, 6, False), (168, 5, False), (184, 4, False), (216, 6, False),
                                            (224, 6, False), (224, 2, False), (88, 6, True), (168, 4, True)])
def test_fused_planes_match_separate_passes(n, iters, vector):
    size = [n - 24, n - 24, 12]
    p = cases.params(size, [6, 6, 2], return_3D=True, iterations_number=iters)
    p["vector_simulation"] = vector
    RI = cases.sphere_phantom(size, [0.1] * 3, cases.NM, seed=n, n_spheres=2, radius_um=(0.2, 0.5))
    fields = cases.circle_fields(p, 3)
    if vector:
        fields = np.concatenate([fields, 0.5j * fields], axis=2)
    t1, _, f1 = _solve(p, RI, fields, True)
    t2, _, f2 = _solve(p, RI, fields, False)
    assert np.isfinite(f1).all()
    for k in range(3):
        assert cbs.rel_l2(t1[..., k], t2[..., k]) < 5e-6
        assert cbs.rel_l2(f1[..., k], f2[..., k]) < 5e-6
