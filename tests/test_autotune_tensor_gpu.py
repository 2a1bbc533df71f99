"""Autotuned plans of RI tensors and of scalar potentials on one dyadic grid are
chosen apart: a tensor has no fused xy-pass (odt_autotune)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor_first", [True, False])
def test_tensor_and_scalar_potentials_are_tuned_apart(tensor_first):
    from inverse_solver_b200 import FORWARD_SOLVER_CONVERGENT_BORN

    n = 40 if tensor_first else 48   # the cache lives as long as the process
    p = cases.params([n, n, 24], [6, 6, 6], vector_simulation=True, iterations_number=4)
    RI = cases.sphere_phantom([n, n, 24], [0.1] * 3, cases.NM, seed=3, n_spheres=2, radius_um=(0.4, 0.8))
    tensor = np.zeros(RI.shape + (3, 3), np.float32)
    for j in range(3):
        tensor[..., j, j] = RI
    got = {}
    for kind in ([True, False] if tensor_first else [False, True]):
        s = FORWARD_SOLVER_CONVERGENT_BORN(p)
        s.set_RI(tensor if kind else RI)
        got[kind] = s.autotune(2)
        s.delete()
    assert not got[True]["cached"] and not got[False]["cached"]
    assert "fused_xy" in got[False]["ms"] and "fused_xy" not in got[True]["ms"]
