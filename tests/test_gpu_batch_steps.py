"""Two steps of the batched SCF whose kernels change with the molecule or share a warp, against the
single-point path: the Lanczos bounds at the order where a cluster takes over from one block (320
orbitals), and A-DIIS weights, a warp per molecule, with molecules of different history lengths side by
side. Both paths converge to 1e-10 eV; the energies agree to 1e-7 eV per atom.
"""
import pytest

from pm7b200 import api
from pm7b200 import geometry as G

pytestmark = pytest.mark.gpu


def _check(mols, **kw):
    got = api.run_batch(mols, e_tol=1.0e-10, p_tol=1.0e-9, **kw)
    for (z, x), r in zip(mols, got):
        ref = api.run_pm7(z, x, e_tol=1.0e-10, p_tol=1.0e-9, **kw)
        assert abs(r["total_ev"] - ref["total_ev"]) < 1e-7 * len(z)


@pytest.mark.parametrize("waters", [(53,), (54,), (53, 54, 130)])
def test_lanczos_bounds_by_one_block_and_by_clusters(waters):
    _check([G.water_cluster(n, seed=n) for n in waters])


@pytest.mark.parametrize("switch", [0.1, 1.0e-3])
def test_adiis_weights_by_a_warp(switch):
    mols = [G.alkane(n, seed=n) for n in (1, 2, 3, 5, 8, 13, 21)] + [G.water_cluster(n, seed=n) for n in (1, 4, 9)]
    _check(mols, adiis_switch=switch)
