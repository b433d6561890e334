"""The shared-memory Jacobi eigensolver at the edges of its sets of four indices.

Orders 1 to 8 (one set, two sets, padded by one to three rows), 109 to 112 (the largest), cold in the
first iteration and warm in the others, as the density solver of a single point, against the default
solver. Both converge the SCF to 1e-10 eV and 1e-9 in the density; the energy's error is of second order in the density's, the
levels' of first: 1e-7 eV per atom and 1e-5 eV.
"""
import numpy as np
import pytest

from pm7b200 import api
from pm7b200 import geometry as G

pytestmark = pytest.mark.gpu

A0 = 0.529177210903
SMALL = {  # order -> (z, xyz in Angstrom)
    1: ([1], [[0, 0, 0]]),
    2: ([1, 1], [[0, 0, 0], [0, 0, 0.74]]),
    4: ([10], [[0, 0, 0]]),
    5: ([9, 1], [[0, 0, 0], [0, 0, 0.95]]),
    6: ([8, 1, 1], [[0, 0, 0], [0.96, 0, 0], [-0.24, 0.93, 0]]),
    7: ([7, 1, 1, 1], [[0, 0, 0.1], [0.94, 0, -0.25], [-0.47, 0.81, -0.25], [-0.47, -0.81, -0.25]]),
    8: ([6, 1, 1, 1, 1], [[0, 0, 0], [0.63, 0.63, 0.63], [-0.63, -0.63, 0.63], [-0.63, 0.63, -0.63], [0.63, -0.63, -0.63]]),
}


def _molecule(order):
    if order in SMALL:
        z, x = SMALL[order]
        return np.array(z), np.array(x, float) / A0
    z, x = G.alkane(17, seed=3)  # 104 orbitals, and a small molecule beside it
    zs, xs = _molecule(order - 104)
    return np.concatenate([z, zs]), np.concatenate([x, xs + x.max(axis=0) + 8.0])


@pytest.mark.parametrize("order", sorted(SMALL) + [109, 110, 111, 112])
def test_single_point_by_jacobi(order, monkeypatch):
    z, x = _molecule(order)
    mult = 2 if order == 1 else 1
    ref = api.run_pm7(z, x, multiplicity=mult, p_tol=1.0e-9, e_tol=1.0e-10)
    monkeypatch.setenv("PM7_DENSITY_SOLVER", "jacobi")
    got = api.run_pm7(z, x, multiplicity=mult, p_tol=1.0e-9, e_tol=1.0e-10)
    assert len(got["mo_energies"]) == order
    assert abs(got["total_ev"] - ref["total_ev"]) < 1e-7 * len(z)
    np.testing.assert_allclose(got["mo_energies"], ref["mo_energies"], rtol=0, atol=1e-5)
