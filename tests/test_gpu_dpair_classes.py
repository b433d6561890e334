"""The MNDO/d-frame kernels' classes of pairs (two d atoms, one, none), against the CPU oracle.

Each class is a launch of its own over all near pairs, four pairs (or stencil points) to a block:
molecules with pairs of one class only, with every class, and with pair counts that do not fill a
block. The Fock matrix takes the tolerance of the integrals times the ten sums of an element, the
gradient that of a fixed density (1e-6 eV/Bohr).
"""
import numpy as np
import pytest

from oracle import harness
from pm7b200 import api

pytestmark = pytest.mark.gpu

CASES = {
    "one_two_d_pair": [17, 17],
    "two_d_only": [16, 17, 35],
    "one_d_pair": [17, 1],
    "one_d_and_none": [16, 1, 6, 1, 8],
    "every_class": [17, 6, 16, 1, 26, 8, 1],
}


def _molecule(name):
    z = np.array(CASES[name])
    rng = np.random.default_rng(len(z))
    k = np.arange(len(z))
    x = np.stack([3.9 * np.cos(1.3 * k) * (1 + 0.2 * k), 3.9 * np.sin(1.3 * k) * (1 + 0.2 * k), 1.1 * k], axis=1)
    nao = int(sum(1 if v == 1 else (9 if v in (16, 17, 26, 35) else 4) for v in z))
    a = rng.normal(size=(nao, nao)) * 0.1
    p = a @ a.T / nao
    np.fill_diagonal(p, np.abs(np.diag(p)) + 0.5)
    return z, x + 0.1 * rng.normal(size=x.shape), p


@pytest.mark.parametrize("name", sorted(CASES))
def test_fock_and_gradient_by_pair_classes(name):
    z, x, p = _molecule(name)
    np.testing.assert_allclose(api.fock(z, x, p, 0.5 * p), harness.fock(z, x, p, 0.5 * p), rtol=0, atol=1.0e-9)
    got = api.fixed_density_gradient(z, x, p, None)
    ref = harness.fixed_density_gradient(z, x, p, None)
    assert np.max(np.abs(got - ref)) < 1.0e-6
