"""The timed work of the engine: what a program that uses it has it do, over the real range.

Molecules come from the package's own seeded generators (`pm7b200.geometry`): water clusters
(the sp frame, three-dimensional), alkanes and alkyl radicals, and S/Cl-substituted chains (the
MNDO/d frame). The engine takes host arrays and returns host arrays, so a pass is the whole
call. `listed` holds fixed sizes, `draw` more of the same kinds over their ranges.
"""
import math
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "pm7-rs_b200"))

from pm7b200 import api, geometry  # noqa: E402

# Results that are compared: everything a caller reads that has one right value. Eigenvectors
# (free in sign and within degenerate levels), iteration counts and timings are left out.
SCALARS = ("total_ev", "heat_of_formation_kcal", "electronic_ev", "core_ev", "correction_kcal")


def listed():
    return [
        # one small molecule (11 atoms, 20 orbitals): an interactive call, all latency
        dict(name="propane", kind="point", molecule="alkane", size=3, precision="fp64", matrices=False),
        # an organic radical (61 atoms, 121 orbitals), UHF: two spin densities per cycle
        dict(name="radical20", kind="point", molecule="radical", size=20, precision="fp64", matrices=False),
        # 34 waters (102 atoms, 204 orbitals) with the default options, density returned
        dict(name="water34", kind="point", molecule="water", size=34, precision="fp64", matrices=True),
        # one force call of an optimiser or an MD step: SCF and gradient, d frame
        dict(name="chain41_force", kind="gradient", molecule="chain", size=41, precision="fp64"),
        # a force call on a mid-sized cluster (333 atoms, 666 orbitals)
        dict(name="water111_force", kind="gradient", molecule="water", size=111, precision="fp64"),
        # the benchmark's single point: 1,002 atoms, 2,004 orbitals
        dict(name="water334", kind="point", molecule="water", size=334, precision="fp64", matrices=False),
        # the largest: 3,000 atoms, 6,000 orbitals, early cycles in fp32
        dict(name="water1000_mixed", kind="point", molecule="water", size=1000, precision="mixed", matrices=False),
        # a screening batch: alkanes up to C40 and water clusters up to 64, one call
        dict(name="batch512", kind="batch", molecule="batch", size=512, precision="fp64"),
        # forces of many molecules at once (a training-set run), 3 to 500 atoms, sp and d
        dict(name="batch64_force_mixed", kind="batch_gradient", molecule="stream", size=64, precision="mixed"),
        # a serving process: requests of 3 to 500 atoms handed to a running engine, all collected
        dict(name="served128", kind="served", molecule="stream", size=128, precision="fp64"),
        # a long chain by divide and conquer with its gradient (482 atoms)
        dict(name="dandc160", kind="dandc", size=160),
        # orbital levels of given Fock matrices, orders 30 to 700
        dict(name="levels16", kind="levels", size=16, order=700),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("point", "point", "point", "gradient", "gradient", "batch", "batch_gradient", "served",
                       "dandc", "levels"))
    precision = rng.choice(("fp64", "fp64", "mixed"))
    if kind == "point":
        molecule = rng.choice(("water", "water", "alkane", "chain", "radical"))
        hi = {"water": 1000 if precision == "mixed" else 600, "alkane": 240, "chain": 160, "radical": 60}[molecule]
        lo = 200 if molecule == "water" and precision == "mixed" else 2
        return dict(kind=kind, molecule=molecule, size=_log(rng, lo, hi),
                    precision="fp64" if molecule == "radical" else precision,
                    matrices=molecule != "water" and rng.random() < 0.3)
    if kind == "gradient":
        molecule = rng.choice(("water", "chain", "alkane"))
        return dict(kind=kind, molecule=molecule, size=_log(rng, 2, 333 if molecule == "water" else 120),
                    precision=precision)
    if kind == "batch":
        return dict(kind=kind, molecule=rng.choice(("batch", "stream")), size=_log(rng, 12, 600), precision=precision)
    if kind == "batch_gradient":
        return dict(kind=kind, molecule=rng.choice(("batch", "stream")), size=_log(rng, 8, 128), precision=precision)
    if kind == "served":
        return dict(kind=kind, molecule="stream", size=_log(rng, 8, 192), precision=precision)
    if kind == "dandc":
        return dict(kind=kind, size=_log(rng, 24, 320))
    return dict(kind=kind, size=_log(rng, 2, 32), order=_log(rng, 40, 1200))


def _one(molecule, size):
    """The molecule of a kind and size (the radical: an alkane without its last hydrogen)."""
    if molecule == "water":
        return geometry.water_cluster(size, seed=size)
    if molecule == "chain":
        return geometry.substituted_chain(size, np.random.default_rng(size))
    z, xyz = geometry.alkane(size, seed=size)
    return (z[:-1], xyz[:-1]) if molecule == "radical" else (z, xyz)


def _many(case):
    """The molecules of a batch or a burst of requests."""
    return getattr(geometry, case["molecule"])(case["size"], seed=case["size"])


def _moved(molecule, rng):
    """Another geometry of the same molecule: every coordinate off by up to 0.03 Bohr."""
    z, xyz = molecule
    return z, xyz + rng.uniform(-0.03, 0.03, size=xyz.shape)


def _fock_like(n, rng):
    """A symmetric matrix with the look of a Fock matrix: levels of -40 to 10 eV on the diagonal,
    couplings that fall off with the distance of the orbitals, a last bit of noise everywhere."""
    i = np.arange(n)
    a = rng.normal(size=(n, n)) * (6.0 * np.exp(-np.abs(i[:, None] - i[None, :]) / 6.0) + 0.02)
    a = 0.5 * (a + a.T)
    a[i, i] += rng.uniform(-40.0, 10.0, size=n)
    return a


def _matrices(case, seed):
    """Orders spread over 30 .. `order` (log-uniform, the largest always there)."""
    rng = np.random.default_rng(seed)
    lo = min(30, case["order"])
    at = np.random.default_rng(case["order"]).uniform(math.log(lo), math.log(case["order"] + 0.5), size=case["size"])
    orders = np.exp(at).astype(int)
    orders[0] = case["order"]
    return [_fock_like(int(n), rng) for n in orders]


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = dict(case)
    if kind in ("point", "gradient"):
        s["z"], s["xyz"] = _moved(_one(case["molecule"], case["size"]), rng)
        s["options"] = dict(precision=case["precision"], want_matrices=int(case.get("matrices", False)))
        if case["molecule"] == "radical":
            s["options"]["multiplicity"] = 2
    elif kind in ("batch", "batch_gradient", "served"):
        s["molecules"] = [_moved(m, rng) for m in _many(case)]
        s["options"] = dict(precision=case["precision"], want_matrices=0)
        if kind == "served":
            s["engine"] = api.Engine()
    elif kind == "dandc":
        s["z"], s["xyz"] = _moved(geometry.flat_alkane(case["size"]), rng)
    else:
        s["matrices"] = _matrices(case, seed)
    return s


def _outputs(r):
    out = {k: r[k] for k in SCALARS}
    for k in ("charges", "mo_energies", "mo_energies_beta", "dipole_debye", "density", "spin_density", "gradient"):
        if r.get(k) is not None:
            out[k] = r[k]
    return out


def _joined(results):
    """One array per quantity over all molecules, in input order."""
    rows = []
    for r in results:
        if isinstance(r, Exception):
            raise r
        rows.append(_outputs(dict(r["scf"], gradient=r["gradient"]) if "scf" in r else r))
    return {k: np.concatenate([np.asarray(row[k], dtype=np.float64).reshape(-1) for row in rows]) for k in rows[0]}


def run(s):
    kind = s["kind"]
    if kind == "point":
        return _outputs(api.run_pm7(s["z"], s["xyz"], **s["options"]))
    if kind == "gradient":
        r = api.closed_form_gradient(s["z"], s["xyz"], **s["options"])
        return _outputs(dict(r["scf"], gradient=r["gradient"]))
    if kind == "batch":
        return _joined(api.run_batch(s["molecules"], **s["options"]))
    if kind == "batch_gradient":
        return _joined(api.run_batch_gradient(s["molecules"], **s["options"]))
    if kind == "served":
        tickets = [s["engine"].submit(z, x, **s["options"]) for z, x in s["molecules"]]
        return _joined([s["engine"].poll(t, wait=True)[1] for t in tickets])
    if kind == "dandc":
        r = api.run_dandc(s["z"], s["xyz"], dandc=dict(core_size=8, p_tol=1.0e-7), gradient=True, want_matrices=0)
        return {k: r[k] for k in ("energy_ev", "electronic_ev", "core_core_ev", "correction_ev", "fermi_ev",
                                  "charges", "gradient")}
    return {"levels": np.concatenate(api.eigenvalues(s["matrices"]))}


def exact(case, seed):
    """Eigenvalues by numpy; a self-consistent field has no closed reference of seconds."""
    if case["kind"] != "levels" or case["size"] * case["order"] ** 3 > 4e10:
        return None
    return {"levels": np.concatenate([np.linalg.eigvalsh(m) for m in _matrices(case, seed)])}


CYCLES = 15  # SCF cycles of an ordinary molecule at the default tolerances


def _solve_work(z, gradient=False):
    """Per cycle: the commutator (2 n^3), a density from an n x n Fock matrix (an eigensolve's
    4/3 n^3 and the occupied product) and one pass over H, F and P; the last levels once."""
    n = int(sum(1 if int(v) == 1 else (9 if int(v) > 10 else 4) for v in z))
    flops = CYCLES * (2.0 + 4.0 / 3.0 + 0.6) * n ** 3 + 4.0 / 3.0 * n ** 3
    byts = CYCLES * 3 * 8.0 * n * n + 40.0 * len(z)
    if gradient:
        flops += 100.0 * 12 * len(z) ** 2 / 2
        byts += 24.0 * len(z)
    return flops, byts


def work(case):
    kind = case["kind"]
    if kind == "levels":
        orders = [len(m) for m in _matrices(case, 1)]
        return {"flops": sum(4.0 / 3.0 * n ** 3 for n in orders), "bytes": sum(8.0 * n * (n + 1) for n in orders)}
    if kind in ("point", "gradient"):
        molecules = [_one(case["molecule"], case["size"])]
    elif kind == "dandc":  # subsystems of about 48 atoms and 110 orbitals, 50 cycles, two products each
        subs = case["size"] * 3 / 8
        return {"flops": subs * 50 * 6.0 * 110 ** 3, "bytes": subs * 50 * 3 * 8.0 * 110 ** 2}
    else:
        molecules = _many(case)
    total = [_solve_work(z, "gradient" in kind) for z, _ in molecules]
    return {"flops": sum(t[0] for t in total), "bytes": sum(t[1] for t in total)}
