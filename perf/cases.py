"""The work that users of this library have it do, as cases that a harness can time.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare`` what a
program holds before the call, ``run`` one pass through the public entry points of ``am1gpu.native``,
``work`` the bytes and operations of a pass that no method can leave out, and ``exact`` the results in
64 bits from plain numpy where plain numpy has them.

The library is called with host arrays and answers in host arrays, so a pass is the whole call.
"""

from __future__ import annotations

import math
import pathlib
import sys

import numpy as np

_PACKAGE = str(pathlib.Path("am1-rs_b200").resolve())
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from am1gpu import _abi, native, workloads  # noqa: E402

SCF_ITERATIONS = 11  # what a molecule of these generators takes from the SAD guess


def listed() -> list[dict]:
    return [
        # The smallest call: one molecule of a few atoms from a script.  Launches and latency only.
        {"name": "single_methane", "path": "single", "kind": "alkane", "size": 1},
        # The plain one-molecule call at an ordinary size: the 32-water cluster (192 orbitals).
        {"name": "single_water32", "path": "single", "kind": "water", "size": 32},
        # One step of a geometry optimisation or of molecular dynamics: energy and gradient of one
        # open-shell chain of odd size (C13H27, 79 orbitals, both spin channels).
        {"name": "gradient_radical13", "path": "gradient", "kind": "radical", "size": 13},
        # Screening: the benchmark's batch, 4096 alkanes of 1..40 carbons and water clusters of 1..64
        # monomers, FP64, host buffers that the program keeps between calls.
        {"name": "batch_4096", "path": "batch", "count": 4096, "radicals": 0, "precision": "fp64"},
        # The same kind of screening on the mixed-precision path with one radical in nine.
        {"name": "batch_mixed_1152", "path": "batch", "count": 1024, "radicals": 128, "precision": "mixed"},
        # What a serving loop collects while a batch runs: sizes log-uniform on 3..600 atoms, one
        # request in ten open shell; a fifth of them are above 448 orbitals.
        {"name": "serving_64", "path": "serving", "count": 64},
        # One large molecule: 512 waters, 3072 orbitals.
        {"name": "large_water512", "path": "single", "kind": "water", "size": 512},
        # Forces of a batch: 192 alkanes and water clusters of the benchmark's sizes.
        {"name": "gradient_batch_192", "path": "gradient_batch", "count": 192},
        # Right-hand sides of one response iteration: 3N trial densities of the 32-water cluster.
        {"name": "response_water32", "path": "response", "kind": "water", "size": 32, "nrhs": 288},
        # Divide and conquer: the subsystem eigenproblems of one SCF iteration, 24..320 rows, ragged.
        {"name": "eigen_batch_96", "path": "eigen_batch", "count": 96, "low": 24, "high": 320},
        # A dense symmetric eigenproblem of odd size with its vectors, above the on-chip sizes.
        {"name": "eigen_1501", "path": "eigen", "n": 1501},
        # The density step of one SCF iteration on its own, at the largest orbital count that
        # the screening batch has.
        {"name": "purify_384", "path": "purify", "n": 384, "precision": "fp64"},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng) -> dict:
    path = rng.choice(["single", "single", "gradient", "batch", "batch", "serving", "gradient_batch", "response",
                       "eigen_batch", "eigen", "purify"])
    kind = rng.choice(["alkane", "water", "radical"])
    # 1..200 waters or 1..132 carbons: 6..1200 and 8..794 orbitals
    size = _log_int(rng, 1, 200 if kind == "water" else 132)
    if path == "single":
        return {"path": path, "kind": kind, "size": size}
    if path == "gradient":
        return {"path": path, "kind": kind, "size": min(size, 64)}
    if path == "batch":
        count = _log_int(rng, 16, 2048)
        return {"path": path, "count": count, "radicals": rng.choice([0, count // 8, count // 3]),
                "precision": rng.choice(["fp64", "mixed"])}
    if path == "serving":
        return {"path": path, "count": _log_int(rng, 4, 96)}
    if path == "gradient_batch":
        return {"path": path, "count": _log_int(rng, 4, 384)}
    if path == "response":
        kind = rng.choice(["alkane", "water"])
        size = _log_int(rng, 2, 40)
        return {"path": path, "kind": kind, "size": size, "nrhs": _log_int(rng, 1, 9 * size)}
    if path == "eigen_batch":
        low = _log_int(rng, 5, 100)
        return {"path": path, "count": _log_int(rng, 2, 192), "low": low, "high": rng.randint(low, 400)}
    if path == "eigen":
        return {"path": path, "n": _log_int(rng, 16, 2400)}
    return {"path": path, "n": _log_int(rng, 12, 448), "precision": rng.choice(["fp64", "fp64", "tf32"])}


# ---------------------------------------------------------------------------------------
# Sizes are a case's own; coordinates and matrix elements come from the seed.
# ---------------------------------------------------------------------------------------
def _nao(kind: str, size: int) -> int:
    return {"water": 6 * size, "alkane": 6 * size + 2, "radical": 6 * size + 1}[kind]


def _natoms(kind: str, size: int) -> int:
    return {"water": 3 * size, "alkane": 3 * size + 2, "radical": 3 * size + 1}[kind]


def _members(case: dict) -> list[tuple[str, int]]:
    """(kind, size) of every molecule of a case."""
    path = case["path"]
    if path in ("batch", "gradient_batch"):
        out = [("alkane", 1 + (7 * (i // 2)) % 40) if i % 2 == 0 else ("water", 1 + (11 * (i // 2)) % 64) for i in range(case["count"])]
        return out + [("radical", 1 + (7 * i) % 40) for i in range(case.get("radicals", 0))]
    if path == "serving":
        out = []
        for i in range(case["count"]):
            # the i-th of evenly spread quantiles of the log-uniform law, in a scattered order
            q = ((i * 0.6180339887498949) % 1.0 + 0.5 / case["count"]) % 1.0
            atoms = 3.0 * 200.0 ** q
            if i % 10 == 9:
                out.append(("radical", max(1, round((atoms - 1) / 3))))
            elif i % 2 == 0:
                out.append(("alkane", max(1, round((atoms - 2) / 3))))
            else:
                out.append(("water", max(1, round(atoms / 3))))
        return out
    return [(case["kind"], case["size"])]


def _eigen_sizes(case: dict) -> list[int]:
    if case["path"] == "eigen":
        return [case["n"]]
    return [case["low"] + (case["high"] - case["low"]) * ((i * 37) % case["count"]) // max(1, case["count"] - 1)
            for i in range(case["count"])]


def _molecule(kind: str, size: int, rng: np.random.Generator) -> workloads.Mol:
    if kind == "water":
        return workloads.water_cluster(size, rng)
    return workloads.alkane(size, rng, radical=kind == "radical")


def _symmetric(n: int, rng: np.random.Generator) -> np.ndarray:
    """Symmetric, with diagonal elements spread as a Fock matrix's (-40 to 10 eV)."""
    a = rng.standard_normal((n, n)) * (4.0 / math.sqrt(n))
    a = 0.5 * (a + a.T)
    a[np.diag_indices(n)] += rng.uniform(-40.0, 10.0, n)
    return a


def _gapped(n: int, rng: np.random.Generator) -> tuple[np.ndarray, int]:
    """A dense matrix with an AM1 spectrum (occupied -40 to -12 eV, virtual 1 to 10 eV) and its occupation."""
    occ = max(1, (2 * n) // 3)
    eps = np.concatenate([rng.uniform(-40.0, -12.0, occ), rng.uniform(1.0, 10.0, n - occ)])
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    f = (q * eps) @ q.T
    return 0.5 * (f + f.T), occ


def prepare(case: dict, seed: int):
    rng = np.random.default_rng([seed, 17])
    path = case["path"]
    if path in ("eigen", "eigen_batch"):
        return case, [_symmetric(n, rng) for n in _eigen_sizes(case)]
    if path == "purify":
        return case, _gapped(case["n"], rng)
    mols = [_molecule(kind, size, rng) for kind, size in _members(case)]
    if path in ("single", "gradient"):
        return case, mols[0]
    triples = [(m.numbers, _abi.angstrom_to_bohr(m.xyz), m.charge, m.multiplicity) for m in mols]
    if path == "response":
        n = _nao(case["kind"], case["size"])
        d = rng.standard_normal((case["nrhs"], n, n)) * 0.05
        return case, triples[0], d + d.transpose(0, 2, 1)
    if path == "gradient_batch":
        return case, triples
    return case, native.Batch(triples)


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def _record(r: dict) -> dict:
    """The numbers of a result dictionary, its lists as arrays."""
    out = {}
    for k, v in r.items():
        if v is None or isinstance(v, str):
            continue
        out[k] = np.asarray(v) if isinstance(v, (list, np.ndarray)) else v
    return out


def _batch_outputs(b: native.Batch) -> dict:
    scalars = np.array([(r.total_ev, r.electronic_ev, r.core_ev, r.heat_of_formation_kcal, r.dipole_magnitude) for r in b.res])
    return {
        "total_ev": scalars[:, 0], "electronic_ev": scalars[:, 1], "core_ev": scalars[:, 2],
        "heat_of_formation_kcal": scalars[:, 3], "dipole_magnitude": scalars[:, 4],
        "charges": np.concatenate([rb.charges for rb in b.rbs]),
        "mo_energies": np.concatenate([rb.mo_energies for rb in b.rbs]),
        "status": np.array(b.status),
    }


def run(state):
    case = state[0]
    path = case["path"]
    if path == "single":
        return _record(native.single_point(state[1].numbers, state[1].xyz, state[1].charge, state[1].multiplicity))
    if path == "gradient":
        return _record(native.gradient(state[1].numbers, state[1].xyz, state[1].charge, state[1].multiplicity))
    if path == "batch":
        state[1].run(precision=case["precision"])
        return _batch_outputs(state[1])
    if path == "serving":
        state[1].run()
        return _batch_outputs(state[1])
    if path == "gradient_batch":
        status, res = native.gradient_batch(state[1])
        return {"status": np.array(status), "gradient": np.concatenate([r["gradient"] for r in res]),
                "charges": np.concatenate([r["charges"] for r in res]), "energy_ev": np.array([r["energy_ev"] for r in res])}
    if path == "response":
        return native.g_matrix_batch(state[1][0], state[1][1], state[2])
    if path == "eigen_batch":
        status, pairs = native.eigh_batch(state[1])
        return {"status": np.array(status), "w": np.concatenate([w for w, _ in pairs]),
                "v": np.concatenate([v.reshape(-1) for _, v in pairs])}
    if path == "eigen":
        w, v = native.eigh(state[1][0])
        return {"w": w, "v": v}
    p, _ = native.density_purify(state[1][0], state[1][1], 2.0, case["precision"])
    return p


def work(case: dict) -> dict:
    """Inputs read once and outputs written once.  Operations: an SCF iteration needs a density of each
    channel's Fock matrix and the commutator of the two (2 n^3; a density by the cheapest route known here, eight
    symmetric products, 8 n^3); an eigendecomposition with vectors 4/3 n^3 for the reduction and 2 n^3 for the
    back-transformation; G(P) 2 operations per two-electron integral and exchange or Coulomb element."""
    path = case["path"]
    if path in ("eigen", "eigen_batch"):
        ns = _eigen_sizes(case)
        return {"bytes": sum(16.0 * n * n + 8.0 * n for n in ns), "flops": sum(10.0 / 3.0 * n ** 3 for n in ns)}
    if path == "purify":
        return {"bytes": 16.0 * case["n"] ** 2, "flops": 8.0 * case["n"] ** 3}
    if path == "response":
        n, heavy = _nao(case["kind"], case["size"]), case["size"]
        light = _natoms(case["kind"], case["size"]) - heavy
        integrals = 100 * heavy * (heavy - 1) / 2 + 10 * heavy * light + light * (light - 1) / 2
        return {"bytes": 16.0 * case["nrhs"] * n * n, "flops": case["nrhs"] * 8.0 * integrals}
    flops = nbytes = 0.0
    for kind, size in _members(case):
        n, channels = _nao(kind, size), 2 if kind == "radical" else 1
        flops += SCF_ITERATIONS * channels * 10.0 * n ** 3
        nbytes += 28.0 * _natoms(kind, size) + 8.0 * _natoms(kind, size) + 8.0 * n * channels + 128.0
        if path in ("gradient", "gradient_batch"):
            nbytes += 24.0 * _natoms(kind, size)
    return {"bytes": nbytes, "flops": flops}


def exact(case: dict, seed: int):
    """Eigenvalues and projectors from numpy's LAPACK.  An eigenvector's sign is free, and an SCF's results
    are those of its own stopping test over this method's integrals, which plain numpy does not have: no value."""
    path = case["path"]
    if path in ("eigen", "eigen_batch"):
        mats = prepare(case, seed)[1]
        w = np.concatenate([np.linalg.eigvalsh(a) for a in mats])
        return {"w": w, "v": None} if path == "eigen" else {"status": None, "w": w, "v": None}
    if path == "purify":
        f, occ = prepare(case, seed)[1]
        _, v = np.linalg.eigh(f)
        return 2.0 * v[:, :occ] @ v[:, :occ].T
    return None
