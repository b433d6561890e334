"""The one-launch SP2 purification against the eigensolver, where its tiling can go wrong.

Sizes: fewer orbitals than a tile, one tile exactly, a tile plus one, odd orders, orders that
are no multiple of the 8-deep K step, the first order with two waves of tiles (17 blocks of 32
and up), and the last below the integer tensor-core path. Both solvers converge the same SCF
to p_tol 1e-9 (rms), so a density element differs by the two convergence errors only; with
~n^2 elements at an rms of 1e-9 each 1e-7 leaves a factor of 50 for the largest one.
"""
import os

import numpy as np
import pytest

from pm7b200 import api, geometry

pytestmark = pytest.mark.gpu

MOLECULES = {
    2: lambda: (np.array([1, 1], dtype=np.uint8), np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]])),
    8: lambda: geometry.alkane(1, seed=1),
    32: lambda: geometry.alkane(5, seed=2),
    38: lambda: geometry.alkane(6, seed=3),
    114: lambda: geometry.water_cluster(19, seed=4),
    128: lambda: geometry.alkane(21, seed=5),
    242: lambda: geometry.alkane(40, seed=6),
    516: lambda: geometry.water_cluster(86, seed=7),
    546: lambda: geometry.water_cluster(91, seed=8),
    762: lambda: geometry.water_cluster(127, seed=9),
}


def _solve(solver, z, x, **kw):
    old = os.environ.get("PM7_DENSITY_SOLVER")
    os.environ["PM7_DENSITY_SOLVER"] = solver
    try:
        return api.run_pm7(z, x, p_tol=1.0e-9, e_tol=1.0e-10, **kw)
    finally:
        if old is None:
            del os.environ["PM7_DENSITY_SOLVER"]
        else:
            os.environ["PM7_DENSITY_SOLVER"] = old


@pytest.mark.parametrize("nao", sorted(MOLECULES))
def test_purification_matches_eigensolver(nao):
    z, x = MOLECULES[nao]()
    a = _solve("sp2", z, x)
    b = _solve("syevd", z, x)
    assert a["nao"] == b["nao"]
    assert np.abs(a["density"] - a["density"].T).max() == 0.0
    assert np.abs(a["density"] - b["density"]).max() < 1.0e-7
    assert abs(a["total_ev"] - b["total_ev"]) < 1.0e-9 * abs(b["total_ev"])


@pytest.mark.parametrize("carbons", [5, 20, 43])
def test_purification_of_two_spins(carbons):
    z, x = geometry.alkane(carbons, seed=carbons)
    a = _solve("sp2", z[:-1], x[:-1], multiplicity=2)
    b = _solve("syevd", z[:-1], x[:-1], multiplicity=2)
    assert np.abs(a["density"] - b["density"]).max() < 1.0e-7
    assert np.abs(a["spin_density"] - b["spin_density"]).max() < 1.0e-7


def test_the_same_bits_twice_and_from_two_threads():
    # cooperative launches of two host threads on two contexts share the device
    import threading

    z, x = geometry.water_cluster(45, seed=3)
    first = api.run_pm7(z, x)
    out = [None, None]

    def work(k):
        out[k] = api.run_pm7(z, x)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in out:
        assert r["total_ev"] == first["total_ev"] and (r["density"] == first["density"]).all()
