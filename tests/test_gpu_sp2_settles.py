"""That SP2 itself gives the densities which other tests compare, and not the eigensolver behind it.

A purification that does not settle is repeated on the Gershgorin interval and then replaced by an
eigensolve, so a result alone cannot show a kernel that never settles at some size, or a narrowed
interval that misses part of the spectrum. Here the counts of both are zero: over the sizes where
the one-launch purification changes its tiling, for two spins, and for batches on both sides of the
order where a cluster finds the bounds (320) and with molecules of all kinds side by side.

The purification alone, on matrices with a known spectrum (occupied levels in [-40, -5], the others
in [0, 10]): its projector, and the interval against the extreme levels. Lanczos steps give a Ritz
interval inside the spectrum's range R, widened by 2% and 4% of itself and a pad of 1e-3 of that
(+1e-6) at each end, so it may not be longer than 1.064 R + 3e-6. The projector is off by the
stopping rule, 1e-13 n_occ, and by the roundings of up to 40 squarings, n eps of the interval each,
seen through the gap (interval / gap < 11): 40 n 1.1e-16 11; twice both for w = 2.

A-DIIS weights by a warp: a batch takes the iterations of the single-molecule path, which computes
them on the host, give or take the one that a last rounding may decide.
"""
import contextlib
import os

import numpy as np
import pytest

from pm7b200 import api
from pm7b200 import geometry as G

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _env(**kw):
    old = {k: os.environ.get(k) for k in kw}
    os.environ.update(kw)
    try:
        yield
    finally:
        for k, v in old.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v


def _counted(call):
    before = api.sp2_counts()
    r = call()
    after = api.sp2_counts()
    return r, {k: after[k] - before[k] for k in after}


MOLECULES = {
    2: lambda: (np.array([1, 1], dtype=np.uint8), np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]])),
    8: lambda: G.alkane(1, seed=1),
    32: lambda: G.alkane(5, seed=2),
    38: lambda: G.alkane(6, seed=3),
    114: lambda: G.water_cluster(19, seed=4),
    128: lambda: G.alkane(21, seed=5),
    242: lambda: G.alkane(40, seed=6),
    516: lambda: G.water_cluster(86, seed=7),
    546: lambda: G.water_cluster(91, seed=8),
    762: lambda: G.water_cluster(127, seed=9),
    780: lambda: G.water_cluster(130, seed=10),
    1410: lambda: G.water_cluster(235, seed=11),
}


@pytest.mark.parametrize("nao", sorted(MOLECULES))
def test_every_purification_of_a_solve_settles_at_once(nao):
    z, x = MOLECULES[nao]()
    with _env(PM7_DENSITY_SOLVER="sp2"):
        r, n = _counted(lambda: api.run_pm7(z, x, want_matrices=0))
    assert r["nao"] == nao and n["asked"] == r["iterations"]
    assert n["retried"] == 0 and n["unsettled"] == 0


@pytest.mark.parametrize("carbons", [5, 20, 43])
def test_every_purification_of_two_spins_settles_at_once(carbons):
    z, x = G.alkane(carbons, seed=carbons)
    with _env(PM7_DENSITY_SOLVER="sp2"):
        r, n = _counted(lambda: api.run_pm7(z[:-1], x[:-1], multiplicity=2, want_matrices=0))
    assert n["asked"] == 2 * r["iterations"]
    assert n["retried"] == 0 and n["unsettled"] == 0


@pytest.mark.parametrize("gemm", ["dmma", "i8"])
@pytest.mark.parametrize("n", [33, 121, 318, 324, 512, 513, 767, 1000, 1409])
def test_projector_and_interval_of_a_known_spectrum(n, gemm):
    rng = np.random.default_rng(n)
    occ = 2 * n // 3
    levels = np.concatenate([np.linspace(-40.0, -5.0, occ), np.linspace(0.0, 10.0, n - occ)])
    q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    f = (q * levels) @ q.T
    f = 0.5 * (f + f.T)
    with _env(PM7_SP2_GEMM=gemm):
        p, info = api.sp2(f, occ)
    assert info["settled"] and info["retries"] == 0 and info["i8"] == (gemm == "i8")
    assert info["lo"] <= levels[0] and info["hi"] >= levels[-1]
    assert info["hi"] - info["lo"] <= 1.064 * 50.0 + 3.0e-6
    ref = 2.0 * q[:, :occ] @ q[:, :occ].T
    assert np.abs(p - ref).max() <= 2.0 * (1.0e-13 * occ + 40 * n * 1.1e-16 * 11.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("waters", [(53,), (54,), (53, 54, 130), (130, 1, 54, 16, 53, 20, 2)])
def test_every_purification_of_a_batch_settles(waters, precision):
    mols = [G.water_cluster(n, seed=n) for n in waters]
    res, n = _counted(lambda: api.run_batch(mols, precision=precision, want_matrices=0))
    assert not any(isinstance(r, Exception) for r in res)
    assert n["batch_asked"] >= max(r["iterations"] for r in res) and n["batch_unsettled"] == 0


@pytest.mark.parametrize("switch", [0.1, 1.0e-3])
def test_adiis_weights_by_a_warp_take_the_iterations_of_the_host(switch):
    mols = [G.alkane(n, seed=n) for n in (1, 2, 3, 5, 8, 13, 21)] + [G.water_cluster(n, seed=n) for n in (1, 4, 9)]
    for (z, x), r in zip(mols, api.run_batch(mols, adiis_switch=switch, want_matrices=0)):
        ref = api.run_pm7(z, x, adiis_switch=switch, want_matrices=0)
        assert abs(r["iterations"] - ref["iterations"]) <= 1
