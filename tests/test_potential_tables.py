"""The tables that a solver keeps between potentials stay its own: what a
caller does to the attributes of one potential (utility_border, the 1D
tables) does not reach the next."""
import numpy as np

import cases
from inverse_solver_b200.forward import CBSHostSetup


def _state(h):
    pp, keep = h.prepare_potential(cases.small_RI())
    u = h.utility_border
    return ([float(pp.green_scale), float(pp.green_offset), float(pp.dV), int(pp.bornmax), list(pp.absorb), float(u.k0_nm)],
            [a.copy() for a in keep] + [u.k3.copy(), u.NA_circle.copy(), u.fourier_coor[0].copy()])


def test_attributes_of_one_potential_do_not_reach_the_next():
    h = CBSHostSetup(cases.small_params())
    scalars, arrays = _state(h)
    u = h.utility_border
    u.k0_nm *= 2
    u.dV = -1.0
    u.k3 += 1
    u.NA_circle[:] = False
    u.fourier_coor[0] *= 3
    for a in h.attenuation_mask1d + h.ramp1d + h.kq2 + h.rads1d:
        a *= 5
    again, arrays2 = _state(h)
    assert again == scalars
    assert all(np.array_equal(a, b) for a, b in zip(arrays, arrays2))
