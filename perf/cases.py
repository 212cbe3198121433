"""Performance cases: the work that a user of this framework gives it.

Every case goes through the public Python binding (``tblite_b200``) with host
buffers in and out, as the C ABI has it: single molecules, batches of uneven
structures, a geometry step with its gradient, the request loop, the batched
generalized eigensolver and the integral stage.  Structures come from the
repository's own generators (n-alkanes, water clusters); a case fixes the
sizes, the seed the coordinates.

``run`` returns energies, iteration counts, statuses, charges, moments and,
where asked for, gradients, orbital energies and densities.  Left out are
``scf_error`` (the last change, noise by construction) and ``e_ts`` on its
own (with a gap at the Fermi level it only reflects where inside the gap the
level search stopped; it is part of ``e_elec``).
"""
import math
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "tblite-cuda_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from tblite_b200 import capi, geometry  # noqa: E402

PARAMS = {"hco": os.path.join(PKG, "params", "synthetic_hco.tbp"),
          "hco_d4": os.path.join(PKG, "params", "synthetic_hco_d4.tbp")}

# nominal SCF iterations, for the work estimate only
ITERATIONS = 8

_calculators = {}


def calculator(name):
    """One calculator per parameter file for the whole process, as a program keeps it."""
    if name not in _calculators:
        _calculators[name] = capi.Calculator(PARAMS[name])
    return _calculators[name]


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # one small organic molecule per call: launches and latency
        {"name": "octane_one", "kind": "singlepoint", "molecules": "alkane", "count": 1, "smallest": 8, "largest": 8,
         "graphs": True},
        # one ordinary solvent cluster per call (138 AOs)
        {"name": "cluster_one", "kind": "singlepoint", "molecules": "water", "count": 1, "smallest": 23,
         "largest": 23, "graphs": False},
        # one large cluster per call, the largest of the batch workload (384 AOs)
        {"name": "cluster_64_one", "kind": "singlepoint", "molecules": "water", "count": 1, "smallest": 64,
         "largest": 64, "graphs": False},
        # one long chain per call (722 AOs), where dense linear algebra dominates
        {"name": "chain_120_one", "kind": "singlepoint", "molecules": "alkane", "count": 1, "smallest": 120,
         "largest": 120, "graphs": False},
        # screening: many small molecules at once (6..60 AOs)
        {"name": "screen_small_400", "kind": "singlepoint", "molecules": "both", "count": 400, "smallest": 1,
         "largest": 10, "graphs": True},
        # an uneven batch of solvent clusters, the batch workload (48..384 AOs)
        {"name": "clusters_1024", "kind": "singlepoint", "molecules": "water", "count": 1024, "smallest": 8,
         "largest": 64, "graphs": True},
        # a batch of long chains (122..1196 AOs)
        {"name": "chains_48", "kind": "singlepoint", "molecules": "alkane", "count": 48, "smallest": 20,
         "largest": 199, "graphs": False},
        # one geometry step of a few molecules: dispersion, gradient, orbital energies and densities
        {"name": "gradient_16", "kind": "gradient", "molecules": "both", "count": 16, "smallest": 6, "largest": 40},
        # the mixed-precision form, converged tightly
        {"name": "mixed_clusters_64", "kind": "mixed", "molecules": "water", "count": 64, "smallest": 8,
         "largest": 64},
        # generalized eigenproblems from another code's matrices
        {"name": "sygvd_24", "kind": "sygvd", "count": 24, "smallest": 30, "largest": 420},
        # a burst of requests of mixed sizes through the serving loop
        {"name": "serving_96", "kind": "serving", "molecules": "both", "count": 96, "smallest": 3, "largest": 62},
        # overlap, core Hamiltonian and moment integrals of one structure for another code (498 AOs)
        {"name": "integrals_83", "kind": "integrals", "molecules": "water", "count": 1, "smallest": 83,
         "largest": 83},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "one", "screen", "batch", "chains", "gradient", "mixed", "sygvd", "serving",
                       "integrals"])
    if kind == "one":
        mol = rng.choice(["water", "alkane"])
        n = _log_int(rng, 1, 64 if mol == "water" else 120)
        return {"kind": "singlepoint", "molecules": mol, "count": 1, "smallest": n, "largest": n,
                "graphs": rng.random() < 0.5}
    if kind == "screen":
        return {"kind": "singlepoint", "molecules": "both", "count": _log_int(rng, 40, 400),
                "smallest": rng.randint(1, 3), "largest": rng.randint(4, 10), "graphs": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": "singlepoint", "molecules": "water", "count": _log_int(rng, 12, 900),
                "smallest": rng.randint(4, 12), "largest": rng.randint(20, 64), "graphs": rng.random() < 0.5}
    if kind == "chains":
        return {"kind": "singlepoint", "molecules": "alkane", "count": _log_int(rng, 4, 40),
                "smallest": rng.randint(10, 40), "largest": rng.randint(60, 190), "graphs": False}
    if kind == "gradient":
        return {"kind": "gradient", "molecules": "both", "count": _log_int(rng, 2, 16),
                "smallest": rng.randint(2, 8), "largest": rng.randint(10, 40)}
    if kind == "mixed":
        return {"kind": "mixed", "molecules": "water", "count": _log_int(rng, 4, 64),
                "smallest": rng.randint(6, 12), "largest": rng.randint(16, 64)}
    if kind == "sygvd":
        return {"kind": "sygvd", "count": _log_int(rng, 1, 24), "smallest": _log_int(rng, 12, 60),
                "largest": _log_int(rng, 80, 420)}
    if kind == "serving":
        return {"kind": "serving", "molecules": "both", "count": _log_int(rng, 16, 96),
                "smallest": rng.randint(3, 6), "largest": rng.randint(20, 62)}
    n = _log_int(rng, 10, 100)
    return {"kind": "integrals", "molecules": "water", "count": 1, "smallest": n, "largest": n}


# --------------------------------------------------------------------------- inputs
def _sizes(case):
    """`count` sizes from smallest to largest, evenly spread, in a fixed shuffled order."""
    n = case["count"]
    s = np.rint(np.linspace(case["smallest"], case["largest"], n)).astype(int) if n > 1 else \
        np.array([case["largest"]])
    return [int(x) for x in np.random.default_rng(7).permutation(s)]


def _kinds(case):
    """(kind, size) of each molecule; 'both' alternates water clusters and alkanes."""
    both = case["molecules"] == "both"
    return [(("water", "alkane")[i & 1] if both else case["molecules"], s) for i, s in enumerate(_sizes(case))]


def _nat_nao(kind, size):
    return (3 * size, 6 * size) if kind == "water" else (3 * size + 2, 6 * size + 2)


def _molecules(case, seed):
    rng = np.random.default_rng(seed)
    return [geometry.water_cluster(s, rng) if kind == "water" else geometry.alkane(s, rng)
            for kind, s in _kinds(case)]


def _pair(n, rng):
    """A symmetric-definite pair like a tight-binding one: a banded Hamiltonian with a
    spread of on-site levels and an overlap close to the identity."""
    decay = np.exp(-np.abs(np.subtract.outer(np.arange(n), np.arange(n))) / 6.0)
    a = rng.standard_normal((n, n)) * decay * 0.2
    h = (a + a.T) * 0.5 + np.diag(rng.uniform(-1.0, 1.0, n))
    b = rng.standard_normal((n, n)) * decay
    s = np.eye(n) + 0.05 * (b @ b.T) / 6.0
    return h, 0.5 * (s + s.T)


def _pairs(case, seed):
    rng = np.random.default_rng(seed)
    return [_pair(n, rng) for n in _sizes(case)]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "sygvd":
        calculator("hco")
        p = _pairs(case, seed)
        state["H"], state["S"] = [x[0] for x in p], [x[1] for x in p]
        return state
    state["calc"] = calculator("hco_d4" if kind == "gradient" else "hco")
    state["mols"] = _molecules(case, seed)
    if kind == "serving":
        state["server"] = capi.Server(state["calc"], 16 << 30, max_batch=64)
    return state


# --------------------------------------------------------------------------- one pass
_SCALARS = ("energy", "e_rep", "e_elec", "e_band", "e_es2", "e_aes2", "e_es3", "e_disp")
_COUNTS = ("iterations", "status", "nsh", "nao")
_ARRAYS = ("dipole", "qat", "qsh", "dpat", "qpat")


def _collect(results, counts=_COUNTS):
    out = {k: np.array([r[k] for r in results]) for k in _SCALARS}
    out.update({k: np.array([r[k] for r in results], np.int64) for k in counts})
    out.update({k: np.concatenate([r[k] for r in results]) for k in _ARRAYS})
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "singlepoint":
        return _collect(state["calc"].singlepoint_batch(state["mols"], use_graphs=int(case["graphs"])))
    if kind == "gradient":
        res = state["calc"].singlepoint_batch(state["mols"], gradient=True, wavefunction=True)
        out = _collect(res)
        out["gradient"] = np.concatenate([r["gradient"] for r in res])
        out["sigma"] = np.array([r["sigma"] for r in res])
        out["emo"] = np.concatenate([r["wfn"]["emo"] for r in res])
        out["density"] = np.concatenate([r["wfn"]["density"].ravel() for r in res])
        return out
    if kind == "mixed":
        # which iteration the mixed phase ends at depends on FP32 noise: the
        # converged values are returned, not the iteration count
        res = state["calc"].singlepoint_batch(state["mols"], precision=1, accuracy=1e-5)
        return _collect(res, ("status", "nsh", "nao"))
    if kind == "serving":
        server, got = state["server"], {}
        for m in state["mols"]:
            server.submit(m)
        while len(got) < len(state["mols"]):
            server.step()
            got.update(server.poll())
        return _collect([got[t] for t in sorted(got)])
    if kind == "sygvd":
        status, pairs = capi.sygvd_batch(state["H"], state["S"])
        # an eigenvector's sign is arbitrary: a program that compares or
        # stores vectors fixes it; here by the sum with alternating weights
        vectors = []
        for w, c in pairs:
            t = np.cos(np.arange(len(w)) * 1.7) @ c
            vectors.append((c * np.where(t < 0.0, -1.0, 1.0)).ravel())
        return {"status": status, "values": np.concatenate([w for w, _ in pairs]), "vectors": np.concatenate(vectors)}
    S, H0, D, Q = capi.get_hamiltonian(state["calc"], state["mols"][0])
    return {"S": S, "H0": H0, "D": D, "Q": Q}


# --------------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass that the path cannot do without.

    Per SCF iteration and structure of N AOs: the eigensolve 4 N^3, the
    transforms and the density 6 N^3 + 2 N^2 n_occ (n_occ ~ 2N/3 or N/2), and
    S, H0, the nine moment planes and P read once (96 N^2 bytes); for a
    single structure that fits on the chip the planes still count once."""
    kind = case["kind"]
    if kind == "sygvd":
        n = np.array(_sizes(case), float)
        return {"bytes": float((8 * (3 * n * n + n)).sum()), "flops": float((9.0 * n ** 3).sum())}
    nn = np.array([_nat_nao(k, s) for k, s in _kinds(case)], float)
    nat, nao = nn[:, 0], nn[:, 1]
    io = 28 * nat + 8 * (12 * nat + 14 * nat)
    if kind == "integrals":
        return {"bytes": float((8 * 11 * nao ** 2 + 28 * nat).sum()), "flops": float((400.0 * nao ** 2).sum())}
    flops = ITERATIONS * (4.0 + 6.0 + 1.2) * nao ** 3 + nao ** 3
    bytes_ = ITERATIONS * 96.0 * nao ** 2 + io
    if kind == "gradient":
        flops = flops + 2.0 * nao ** 3
        bytes_ = bytes_ + 8.0 * nao ** 2 + 8 * (nao + 3 * nat)
    return {"bytes": float(bytes_.sum()), "flops": float(flops.sum())}


# --------------------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """Eigenpairs from numpy's LAPACK (the singlepoints have no value outside this repository)."""
    if case["kind"] != "sygvd":
        return None
    values, vectors = [], []
    for h, s in _pairs(case, seed):
        li = np.linalg.inv(np.linalg.cholesky(s))
        w, z = np.linalg.eigh(li @ h @ li.T)
        c = li.T @ z
        t = np.cos(np.arange(len(w)) * 1.7) @ c
        values.append(w)
        vectors.append((c * np.where(t < 0.0, -1.0, 1.0)).ravel())
    return {"status": None, "values": np.concatenate(values), "vectors": np.concatenate(vectors)}
