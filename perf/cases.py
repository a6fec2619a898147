"""Performance cases of the xTB engine: what a program that uses it asks for, through its
public entry points (``Calculator.singlepoint``, ``batch_singlepoint``, the autograd bridge and
the two device-pointer extensions).

Sizes follow the repository's benchmark workloads (water clusters, linear alkanes, the mixed
ensemble) and its tests.  Every geometry is thermally displaced from the seed, so no two seeds
share one.  Energies, gradients and charges of a single point come out of a self-consistent
iteration that stops at a convergence threshold (1e-6 Eh at the default accuracy), so they have
no exact value to compare with; the matrix entry points do.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tblite_gb300 import autograd, library, workloads
from tblite_gb300.interface import Calculator, batch_singlepoint

# orbitals per element and occupied pairs of the two systems
_AO = {"GFN2-xTB": {1: 1, 6: 4, 8: 4}, "GFN1-xTB": {1: 2, 6: 4, 8: 4}, "IPEA1-xTB": {1: 2, 6: 4, 8: 4}}


def _single(system, size, **more):
    case = {"kind": "single", "system": system, "size": size, "method": "GFN2-xTB", "charge": 0,
            "solver": "diagonalization", "solvation": False, "population": False}
    case.update(more)
    return case


def listed():
    return [
        # latency: one step of a molecular dynamics run on a water dimer (the smoke molecule)
        dict(_single("water", 2), name="water_dimer"),
        # ionisation potentials: the radical cation of a small molecule, open shell, GFN1
        dict(_single("alkane", 8, method="GFN1-xTB", charge=1), name="alkane8_cation_gfn1"),
        # an ordinary single point, the 32-water benchmark cluster
        dict(_single("water", 32), name="water32"),
        # the largest molecule of the drop-in path (C200H402) with population analysis: density
        # matrix and bond orders
        dict(_single("alkane", 200, population=True), name="c200h402"),
        # a solvated cluster through the spectral projection: half of the 1000-water benchmark
        dict(_single("water", 500, solver="purification", solvation=True), name="water500_alpb"),
        # a small batch: conformers and small fragments, where launches count
        {"kind": "batch", "name": "batch48_small", "count": 48, "waters": 8, "carbons": 8,
         "method": "GFN2-xTB"},
        # the mixed ensemble of the benchmark (3-192 atoms) at a quarter of its size
        {"kind": "batch", "name": "ensemble1024", "count": 1024, "waters": 64, "carbons": 60,
         "method": "GFN2-xTB"},
        # the same ensemble with GFN1
        {"kind": "batch", "name": "ensemble384_gfn1", "count": 384, "waters": 64, "carbons": 60,
         "method": "GFN1-xTB"},
        # parameter fitting: energies, forces and parameter gradients of the alkane batch
        {"kind": "train", "name": "fit128", "count": 128, "carbons": 40},
        # FP64-accurate products on device matrices: ragged, and a large symmetric one
        {"kind": "gemm", "name": "gemm_ragged", "m": 1202, "n": 601, "k": 777, "sym": False},
        {"kind": "gemm", "name": "gemm_sym3072", "m": 3072, "n": 3072, "k": 3072, "sym": True},
        # density matrix without device allocation inside a latency-bound loop
        {"kind": "density", "name": "density384", "n": 384, "k": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "batch", "batch", "train", "gemm", "density"])
    if kind == "single":
        form = rng.choice(["water", "alkane", "cation", "projected"])
        method = rng.choice(["GFN2-xTB", "GFN2-xTB", "GFN1-xTB", "IPEA1-xTB"])
        if form == "cation":
            return _single("alkane", _log_int(rng, 2, 13), method=method, charge=1,
                           population=rng.random() < 0.5)
        if form == "projected":
            return _single("water", _log_int(rng, 24, 420), solver="purification",
                           solvation=rng.random() < 0.5)
        size = _log_int(rng, 1, 64) if form == "water" else _log_int(rng, 2, 160)
        return _single(form, size, method=method, population=rng.random() < 0.3,
                       solvation=method == "GFN2-xTB" and rng.random() < 0.3)
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 4, 700), "waters": _log_int(rng, 4, 64),
                "carbons": _log_int(rng, 4, 60), "method": rng.choice(["GFN2-xTB", "GFN1-xTB"])}
    if kind == "train":
        return {"kind": "train", "count": _log_int(rng, 4, 128), "carbons": _log_int(rng, 5, 40)}
    if kind == "gemm":
        m, n, k = (_log_int(rng, 100, 3000) for _ in range(3))
        sym = rng.random() < 0.5
        return {"kind": "gemm", "m": m, "n": m if sym else n, "k": m if sym else k, "sym": sym}
    n = _log_int(rng, 12, 720)
    return {"kind": "density", "n": n, "k": max(1, int(n * rng.uniform(0.3, 0.95)))}


def _molecule(system, size, rng):
    """Numbers and thermally displaced positions (Bohr) of a water cluster or an alkane."""
    make = workloads.water_cluster_k if system == "water" else workloads.alkane
    numbers, positions = make(size, seed=int(rng.integers(1 << 31)))
    return numbers, positions + rng.normal(scale=0.02, size=positions.shape)


def _sizes(case):
    """The molecules of a batch: a property of the case, the same for every seed."""
    rng = np.random.default_rng([case["count"], case["carbons"]])
    if case["kind"] == "train":
        return [("alkane", int(c)) for c in rng.integers(4, case["carbons"] + 1, case["count"])]
    out = []
    for i in range(case["count"]):
        system, top = (("water", case["waters"]), ("alkane", case["carbons"]))[i % 2]
        out.append((system, min(top, int(math.exp(rng.uniform(0.0, math.log(top + 1)))))))
    return out


def _device_matrix(rng, rows, cols):
    return torch.from_numpy(rng.standard_normal((rows, cols))).cuda()


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "single":
        numbers, positions = _molecule(case["system"], case["size"], rng)
        start = positions + rng.normal(scale=0.02, size=positions.shape)
        calc = Calculator(case["method"], numbers, start, charge=float(case["charge"]),
                          uhf=case["charge"])
        if case["solvation"]:
            calc.add("alpb-solvation", "water")
        if case["solver"] != "diagonalization":
            calc.set("density-solver", case["solver"])
        return {"case": case, "calc": calc, "positions": positions}
    if kind in ("batch", "train"):
        mols = [_molecule(system, size, rng) for system, size in _sizes(case)]
        calcs = [Calculator(case.get("method", "GFN2-xTB"), z, x) for z, x in mols]
        if kind == "batch":
            return {"case": case, "calcs": calcs, "positions": [x for _, x in mols]}
        inputs = []
        for c, (_, x) in zip(calcs, mols):
            values = autograd.shell_parameters(c)
            inputs.append((torch.tensor(x, dtype=torch.float64, requires_grad=True),
                           {k: torch.tensor(values[k] * (1.0 + 1e-3 * rng.standard_normal(values[k].size)),
                                            dtype=torch.float64, requires_grad=True)
                            for k in autograd.PARAMETERS}))
        return {"case": case, "calcs": calcs, "inputs": inputs}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        # column-major operands; a symmetric product is A A^T
        a = _device_matrix(rng, k, m)
        b = a.t().contiguous() if case["sym"] else _device_matrix(rng, n, k)
        return {"case": case, "a": a, "b": b}
    n, k = case["n"], case["k"]
    f = torch.from_numpy(np.where(np.arange(k) < 0.9 * k, 2.0, rng.uniform(0.0, 2.0, k))).cuda()
    return {"case": case, "c": _device_matrix(rng, k, n) / math.sqrt(n), "f": f,
            "p": torch.empty((n, n), dtype=torch.float64, device="cuda")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "single":
        calc = state["calc"]
        calc.update(state["positions"])
        res = calc.singlepoint()
        out = {"energy": res.get("energy")}
        for key in ("gradient", "virial", "charges", "dipole"):
            out[key] = res.get(key)
        if case["solver"] == "diagonalization":
            out["orbital-energies"] = res.get("orbital-energies")
        if case["population"]:
            out["bond-orders"] = res.get("bond-orders")
            out["density-matrix"] = res.get("density-matrix")
        return out
    if kind == "batch":
        for calc, x in zip(state["calcs"], state["positions"]):
            calc.update(x)
        results = batch_singlepoint(state["calcs"])
        return {"energy": np.array([r.get("energy") for r in results]),
                "gradient": np.concatenate([r.get("gradient") for r in results]),
                "charges": np.concatenate([r.get("charges") for r in results])}
    if kind == "train":
        leaves = [[x, *prm.values()] for x, prm in state["inputs"]]
        for leaf in leaves:
            for t in leaf:
                t.grad = None
        energy = autograd.gfn2_energies_batch(state["calcs"], [x for x, _ in state["inputs"]],
                                              [prm for _, prm in state["inputs"]])
        energy.sum().backward()
        out = {"energy": energy.detach()}
        for i, key in enumerate(("positions", *autograd.PARAMETERS)):
            out["d_" + key] = torch.cat([leaf[i].grad.reshape(-1) for leaf in leaves])
        return out
    lib = library.load()
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "gemm":
        c = torch.empty((case["n"], case["m"]), dtype=torch.float64, device="cuda")
        rc = lib.tblite_gb300_split_gemm(case["m"], case["n"], case["k"], state["a"].data_ptr(),
                                         state["b"].data_ptr(), c.data_ptr(), int(case["sym"]),
                                         stream)
        if rc != 0:
            raise RuntimeError(f"split GEMM returned {rc}")
        return c
    rc = lib.tblite_gb300_density_matrix_noalloc(case["n"], case["k"], state["c"].data_ptr(),
                                                 state["f"].data_ptr(), state["p"].data_ptr(),
                                                 stream)
    if rc != 0:
        raise RuntimeError(f"density matrix returned {rc}")
    return state["p"]


def exact(case, seed):
    if case["kind"] == "gemm":
        state = prepare(case, seed)
        return state["b"] @ state["a"]
    if case["kind"] == "density":
        state = prepare(case, seed)
        return (state["c"] * state["f"][:, None]).t() @ state["c"]
    return None


def _molecule_work(system, size, method):
    ao = _AO[method]
    if system == "water":
        nat, n, occ = 3 * size, (ao[8] + 2 * ao[1]) * size, 4 * size
    else:
        nat, n, occ = 3 * size + 2, ao[6] * size + ao[1] * (2 * size + 2), 3 * size + 1
    # one overlap factorisation and inverse, then per SCF iteration (about 8 of them) the
    # reduction, the eigenvalues, the occupied vectors and the density
    flops = n ** 3 + 8 * (16 / 3 * n ** 3 + 2 * n * n * occ)
    # positions and numbers in; energy, gradient, charges, virial, dipole out
    return flops, nat * (4 + 8 * 3) + 8 * (4 * nat + 13), nat, n


def work(case):
    kind = case["kind"]
    if kind == "single":
        flops, nbytes, nat, n = _molecule_work(case["system"], case["size"], case["method"])
        if case["solver"] == "diagonalization":
            nbytes += 8 * n
        if case["population"]:
            nbytes += 8 * (nat * nat + n * n)
        return {"bytes": nbytes, "flops": flops}
    if kind in ("batch", "train"):
        parts = [_molecule_work(s, k, case.get("method", "GFN2-xTB")) for s, k in _sizes(case)]
        return {"bytes": sum(p[1] for p in parts), "flops": sum(p[0] for p in parts)}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        flops = n * (n + 1) * k if case["sym"] else 2 * m * n * k
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": flops}
    n, k = case["n"], case["k"]
    return {"bytes": 8 * (n * k + k + n * n), "flops": n * (n + 1) * k}
