"""The whole-GPU tridiagonalisation behind the plain path's levels, at its edges.

Orders where its shapes change: one CTA's registers (4 rows), a CTA more, the 512-column
boundaries of a thread's columns, the first orders with rows in shared memory, and the last one
below the library solver. The levels of `run_pm7` without matrices (this path) are compared with
those of the same run with matrices (cuSOLVER's eigenvectors): the two take the same matrix, both
are backward stable, so they differ by a few n eps |F| < 2000 * 2e-16 * 100 eV = 4e-11; 1e-9 leaves
a factor of 25.
"""
import numpy as np
import pytest

from pm7b200 import api, geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters", [1, 19, 20, 85, 86, 171, 173, 247, 341])
def test_levels_match_the_library_eigensolver(waters):
    z, x = geometry.water_cluster(waters, seed=waters)
    lean = api.run_pm7(z, x, want_matrices=0)
    full = api.run_pm7(z, x, want_matrices=1)
    assert lean["nao"] == 6 * waters
    np.testing.assert_allclose(lean["mo_energies"], full["mo_energies"], rtol=0, atol=1e-9)


@pytest.mark.parametrize("carbons", [3, 22, 60])
def test_levels_of_two_spins(carbons):
    z, x = geometry.alkane(carbons, seed=carbons)
    lean = api.run_pm7(z[:-1], x[:-1], multiplicity=2, want_matrices=0)
    full = api.run_pm7(z[:-1], x[:-1], multiplicity=2, want_matrices=1)
    for k in ("mo_energies", "mo_energies_beta"):
        np.testing.assert_allclose(lean[k], full[k], rtol=0, atol=1e-9)


@pytest.mark.parametrize("scale", [1e-180, 1e-30, 1.0, 1e30, 1e120])
def test_values_at_the_ends_of_the_exponent_range(scale):
    # the minors' recurrence (norm within 1e+-100) and the pivots' recurrence beyond it; the bound of
    # the random matrices of test_gpu_eigvals, relative to the largest level
    rng = np.random.default_rng(5)
    mats = []
    for n in (1, 9, 40, 161):
        a = rng.standard_normal((n, n))
        mats.append(0.5 * (a + a.T) * scale)
    mats.append(np.diag(np.repeat([1.0, 2.0], 30)) * scale)  # exact multiplicities, no couplings
    for a, w in zip(mats, api.eigenvalues(mats)):
        ref = np.linalg.eigvalsh(a / scale)
        assert np.max(np.abs(w / scale - ref)) < 1e-12 * max(1.0, np.sqrt(len(a))) * max(1.0, np.abs(ref).max())
