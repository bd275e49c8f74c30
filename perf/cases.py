"""The calls this framework is used for, from one water molecule to a water cluster of a thousand basis functions.

Every case goes through the public Python entry points (`native.run`, `native.batch`, `native.optimize_batch`,
`native.numerical_hessian_batch`), which take host arrays and return host arrays, so a pass includes the copies. All
arithmetic is FP64 with the reference's default options unless the case says otherwise.

The organics are the benchmark's (C/H/N/O/S trees, `workloads.organic`): a pool of grown molecules evenly over the case's
range of sizes. A seed turns each one at random and displaces its atoms by up to 0.02 A, as the frames of a trajectory or the
conformers of a search are.
"""
import functools
import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pm3-rs_b200"))

from pm3_rs import native, workloads  # noqa: E402

POOL = 48  # grown molecules per range of sizes


def listed():
    return [
        # one tiny molecule at a time: a script's or a calculator's call, where latency is all
        {"name": "water", "kind": "water", "count": 1, "gradient": False},
        # one molecule with forces: a step of molecular dynamics or of an external optimiser
        {"name": "single-24", "kind": "organic", "count": 1, "lo": 24, "hi": 24, "gradient": True, "method": "pm3"},
        # one drug-sized molecule, energy and charges only
        {"name": "single-61", "kind": "organic", "count": 1, "lo": 61, "hi": 61, "gradient": False, "method": "pm3"},
        # a small ensemble with forces: conformers of small molecules, fewer than the GPU has SMs
        {"name": "batch-64", "kind": "organic", "count": 64, "lo": 5, "hi": 17, "gradient": True, "method": "pm3"},
        # screening, an ordinary batch: two molecules per SM or so
        {"name": "batch-300", "kind": "organic", "count": 300, "lo": 5, "hi": 60, "gradient": False, "method": "pm3"},
        # screening, the benchmark's molecules in a large batch
        {"name": "batch-4096", "kind": "organic", "count": 4096, "lo": 5, "hi": 60, "gradient": False, "method": "pm3"},
        # training data for a force field: corrected energies and forces of many mid-sized molecules
        {"name": "d3h4-1000", "kind": "organic", "count": 1000, "lo": 10, "hi": 35, "gradient": True, "method": "pm3-d3h4"},
        # open shells: doublets through the unrestricted loop, with forces
        {"name": "radicals-24", "kind": "radical", "count": 24, "lo": 8, "hi": 22, "gradient": True, "method": "pm3"},
        # harmonic analysis: 6N tightly converged SCFs with gradients per molecule
        {"name": "hessian-3", "kind": "hessian", "count": 3, "lo": 8, "hi": 14},
        # the first steps of a batched relaxation: many dependent small batches
        {"name": "optimize-40", "kind": "optimize", "count": 40, "lo": 6, "hi": 20, "steps": 6},
        # a solvent box as one system, forces included: the 34-water cluster (n = 204) on the whole GPU
        {"name": "cluster-34", "kind": "cluster", "count": 34, "gradient": True},
        # a larger box (n = 966): dense linear algebra on the whole GPU
        {"name": "cluster-161", "kind": "cluster", "count": 161, "gradient": False},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "batch", "batch", "batch", "radical", "hessian", "optimize", "cluster", "cluster"])
    grad = rng.random() < 0.5
    if kind == "single":
        n = _spread(rng, 5, 65)
        method = rng.choice(["pm3", "pm3", "pm3-d3h4"])
        return {"kind": "organic", "count": 1, "lo": n, "hi": n, "gradient": grad, "method": method}
    if kind == "batch":
        lo = rng.randint(5, 20)
        hi = rng.randint(lo + 5, 60)
        count = _spread(rng, 2, 4000)
        method = rng.choice(["pm3", "pm3", "pm3-d3h4"])
        return {"kind": "organic", "count": count, "lo": lo, "hi": hi, "gradient": grad, "method": method}
    if kind == "radical":
        lo = rng.randint(6, 10)
        return {"kind": "radical", "count": _spread(rng, 1, 40), "lo": lo, "hi": rng.randint(lo + 2, 22), "gradient": grad,
                "method": "pm3"}
    if kind == "hessian":
        lo = rng.randint(5, 9)
        return {"kind": "hessian", "count": rng.randint(1, 4), "lo": lo, "hi": rng.randint(lo + 2, 14)}
    if kind == "optimize":
        lo = rng.randint(5, 12)
        return {"kind": "optimize", "count": _spread(rng, 1, 60), "lo": lo, "hi": rng.randint(lo + 3, 24),
                "steps": rng.randint(2, 6)}
    return {"kind": "cluster", "count": _spread(rng, 33, 161), "gradient": grad}


@functools.lru_cache(maxsize=None)
def _pool(radical, lo, hi):
    """Grown molecules with sizes evenly spread over [lo, hi], the same for every seed."""
    k = POOL if hi > lo else 4
    grow = workloads.radical if radical else workloads.organic
    return [grow(int(round(lo + (hi - lo) * i / (k - 1))), 7001 + 31 * i) for i in range(k)]


def _picks(case, rng):
    pool = _pool(case["kind"] == "radical", case["lo"], case["hi"])
    # the molecules belong to the case, their geometries to the seed
    order = np.random.default_rng(case["count"]).permutation(case["count"])
    mols = []
    for i in order:
        z, x = pool[i * len(pool) // case["count"] if case["count"] < len(pool) else i % len(pool)]
        q, r = np.linalg.qr(rng.normal(size=(3, 3)))
        q = q * np.sign(np.diag(r))
        if np.linalg.det(q) < 0.0:
            q[:, 0] = -q[:, 0]
        mols.append((z, x @ q.T + rng.uniform(-0.02, 0.02, x.shape)))
    return workloads.pack(mols)


def _cluster(count, seed):
    """`count` waters on the first sites of the smallest near-cubic grid that holds them."""
    g = [1, 1, 1]
    while g[0] * g[1] * g[2] < count:
        g[g.index(min(g))] += 1
    return workloads.water_cluster(count, grid=tuple(g), seed=seed)


def _inputs(case, seed):
    """(offsets, atomic numbers, coordinates in Angstrom) of a case's molecules."""
    if case["kind"] == "water":
        z, x = workloads.water_cluster(1, grid=(1, 1, 1), seed=seed)
        x = x + np.random.default_rng(seed).uniform(-0.02, 0.02, x.shape)
        return np.array([0, 3], np.int32), z, x
    if case["kind"] == "cluster":
        z, x = _cluster(case["count"], seed)
        return np.array([0, len(z)], np.int32), z, x
    return _picks(case, np.random.default_rng(seed))


def prepare(case, seed):
    offsets, z, x = _inputs(case, seed)
    options = native.options(multiplicity=2 if case["kind"] == "radical" else 1)
    if case.get("method") == "pm3-d3h4":
        options.variant = 2
    return {"case": case, "offsets": offsets, "z": z, "x": x * native.ANGSTROM_TO_BOHR, "options": options}


def run(state):
    c, offs, z, x, o = state["case"], state["offsets"], state["z"], state["x"], state["options"]
    if c["kind"] == "hessian":
        r = native.numerical_hessian_batch(offs, z, x, o)
        return {"hessians": r["hessians"], "status": r["status"]}
    if c["kind"] == "optimize":
        r = native.optimize_batch(offs, z, x, o, max_iter=c["steps"], want_gradient=True)
        return {k: r[k] for k in ("positions_bohr", "gradients", "energy_ev", "heat_of_formation_kcal", "converged")}
    if c["count"] == 1 or c["kind"] == "cluster":
        r = native.run(z, x, o, want_gradient=c["gradient"])
        out = {k: r[k] for k in ("total_ev", "electronic_ev", "core_ev", "heat_of_formation_kcal", "homo_ev", "lumo_ev",
                                 "converged", "charges")}
        out["dipole_debye"] = np.array(r["dipole_debye"])
        if c["gradient"]:
            out["gradient"] = r["gradient"]
        return out
    r = native.batch(offs, z, x, o, want_gradient=c["gradient"])
    out = {k: getattr(r, k) for k in ("total_ev", "electronic_ev", "core_ev", "heat_of_formation_kcal", "homo_ev", "lumo_ev",
                                      "converged", "charges", "dipole_debye")}
    if c["gradient"]:
        out["gradients"] = r.gradients
    return out


def work(case):
    """The inputs and results once; the FP64 operations of one eigensolve, commutator, Fock build and density per SCF
    iteration, at the numbers of iterations that such molecules take."""
    iterations, solves = 12.0, 1.0
    if case["kind"] == "water":
        sizes = [(3.0, 6.0)]
    elif case["kind"] == "cluster":
        sizes = [(3.0 * case["count"], 6.0 * case["count"])]
    else:  # 2.55 basis functions per atom; three sizes stand for the even spread over [lo, hi]
        at = [case["lo"], 0.5 * (case["lo"] + case["hi"]), case["hi"]]
        sizes = [(a, 2.55 * a) for a in at]
    atoms = flops = 0.0
    for a, n in sizes:
        if case["kind"] == "hessian":
            iterations, solves = 20.0, 6.0 * a
        elif case["kind"] == "optimize":
            solves = case["steps"] + 1.0
        elif case["kind"] == "radical":
            iterations = 120.0
        occ = 0.5 * n
        atoms += a / len(sizes)
        flops += solves * iterations * (4.0 / 3.0 * n**3 + 2.0 * n**3 + 2.0 * n * n * occ + 2.0 * n * n * occ) / len(sizes)
    count = 1 if case["kind"] in ("water", "cluster") else case["count"]
    nbytes = 28.0 * atoms + 8.0 * atoms + 72.0 + (24.0 * atoms if case.get("gradient") else 0.0)
    if case["kind"] == "hessian":
        nbytes = 28.0 * atoms + 72.0 * atoms * atoms
    elif case["kind"] == "optimize":
        nbytes = 28.0 * atoms + 48.0 * atoms + 20.0
    return {"bytes": count * nbytes, "flops": count * flops}


# PM3's published core-repulsion parameters: core charge, G_ss (eV), alpha (1/A), and the two Gaussians (K, L in 1/A^2, M in A)
_CORE = {
    1: (1.0, 14.7942080, 3.3563860, ((1.1287500, 5.0962820, 1.5374650), (-1.0603290, 6.0037880, 1.5701890))),
    6: (4.0, 11.2007080, 2.7078070, ((0.0501070, 6.0031650, 1.6422140), (0.0507330, 6.0029790, 0.8924880))),
    7: (5.0, 11.9047870, 2.8305450, ((1.5016740, 5.9011480, 1.7107400), (-1.5057720, 6.0046580, 1.7161490))),
    8: (6.0, 15.7557600, 3.2171020, ((-1.1311280, 6.0024770, 1.6073110), (1.1378910, 5.9505120, 1.5983950))),
    16: (6.0, 8.9646670, 2.2697060, ((-0.3991910, 6.0006690, 0.9621230), (-0.0548990, 6.0018450, 1.5799440))),
}


def _core_repulsion(z, x):
    """PM3's core-core energy (eV) of one molecule at positions in Angstrom."""
    i, j = np.triu_indices(len(z), 1)
    if not len(i):
        return 0.0
    zc, gss, alpha, gauss = (np.array([_CORE[int(e)][k] for e in z]) for k in range(4))
    r = np.sqrt(((x[i] - x[j]) ** 2).sum(-1))
    ev, a0 = 27.211386245988, 0.529177210903  # CODATA 2018
    rho = 0.5 * ev / gss
    ss = ev / np.sqrt((r / a0) ** 2 + (rho[i] + rho[j]) ** 2)
    zz = zc[i] * zc[j]
    # an N or O with an H: the heavy atom's exponential is scaled by the distance
    scale = lambda a, b: np.where(np.isin(z[a], (7, 8)) & (z[b] == 1), r, 1.0)  # noqa: E731
    e = zz * ss * (1.0 + scale(i, j) * np.exp(-alpha[i] * r) + scale(j, i) * np.exp(-alpha[j] * r))
    for a in (i, j):
        for k in range(2):
            kk, ll, mm = gauss[a, k, 0], gauss[a, k, 1], gauss[a, k, 2]
            e = e + zz / r * kk * np.exp(-ll * (r - mm) ** 2)
    return float(e.sum())


def exact(case, seed):
    """The core-core energies, the one output with a closed form. The others are a self-consistent state, which both
    sides know to the tolerance at which the iteration stops: there the two runs are compared with each other."""
    if case["kind"] in ("hessian", "optimize"):
        return None
    offsets, z, x = _inputs(case, seed)
    e = [_core_repulsion(z[a:b], x[a:b]) for a, b in zip(offsets[:-1], offsets[1:])]
    single = case["count"] == 1 or case["kind"] == "cluster"
    return {"core_ev": e[0] if single else np.array(e)}
