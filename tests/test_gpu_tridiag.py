"""Fixed-point tridiagonalisation at the orders where its launch or its layout changes.

Molecules of waters, ammonias and hydrogens are put together to a given number of orbitals: one
CTA, 8-CTA cluster (64 .. 256), cooperative grid (257 .. 512; one molecule of more orbitals takes
the FP64 kernel), the tensor-core products (from 128 on, above 512 by another kernel), and in a
batch the one-CTA, cluster and 16-CTA cluster forms (up to 162, up to about 430, above).
The orbital energies are compared with LAPACK's of the oracle's converged Fock matrix; an SCF
converged to 1e-9 Eh fixes them to well below the 1e-7 Eh used here.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORBITALS = [2, 6, 7, 32, 33, 63, 64, 65, 127, 128, 161, 162, 163, 256, 257]
LARGE = [433, 512, 513]


def _molecule(nao):
    """nao orbitals: ammonias (7) until the rest is even, waters (6), H2 (2); 3.2 A lattice."""
    from tblite_gb300 import workloads

    rng = np.random.default_rng(nao)
    water = np.array([[0.0, 0.0, 0.0], [0.759, 0.0, 0.588], [-0.759, 0.0, 0.588]])
    ammonia = np.array([[0.0, 0.0, 0.0], [0.94, 0.0, 0.38], [-0.47, 0.814, 0.38],
                        [-0.47, -0.814, 0.38]])
    h2 = np.array([[0.0, 0.0, 0.0], [0.74, 0.0, 0.0]])
    parts, left = [], nao
    if left % 2:
        parts.append(([7, 1, 1, 1], ammonia))
        left -= 7
    while left >= 6:
        parts.append(([8, 1, 1], water))
        left -= 6
    while left:
        parts.append(([1, 1], h2))
        left -= 2
    side = int(np.ceil(len(parts) ** (1 / 3)))
    z, x = [], []
    for k, (num, pos) in enumerate(parts):
        site = np.array([k % side, (k // side) % side, k // side ** 2], dtype=float) * 3.2
        z += num
        x.append(pos + site + rng.uniform(-0.1, 0.1, size=3))
    return np.array(z), np.vstack(x) * workloads.AA2BOHR


def _oracle(z, x):
    from oracle import gfn2

    return gfn2.singlepoint(gfn2.new_calc(gfn2.Molecule(z, x), accuracy=1e-3))


def _check(res, ref):
    assert abs(res.get("energy") - ref.energy) < 1e-7
    assert np.max(np.abs(res.get("gradient") - ref.gradient)) < 1e-6
    assert np.max(np.abs(res.get("charges") - ref.qat)) < 1e-6
    assert np.max(np.abs(res.get("orbital-energies") - np.asarray(ref.emo))) < 1e-7


def _calculator(z, x):
    from tblite_gb300.interface import Calculator

    calc = Calculator("GFN2-xTB", z, x)
    calc.set("accuracy", 1e-3)
    return calc


@pytest.mark.parametrize("nao", ORBITALS + LARGE)
def test_one_molecule(nao):
    z, x = _molecule(nao)
    res = _calculator(z, x).singlepoint()
    assert res.get("norbitals") == nao
    _check(res, _oracle(z, x))
    c = res.get("orbital-coefficients")
    assert np.all(np.isfinite(c))


@pytest.mark.parametrize("sizes", [ORBITALS, [33] * 80 + [64, 65, 162, 163], LARGE])
def test_batch(sizes):
    """Diagonalised batches: few molecules (clusters wider than needed) and many."""
    from tblite_gb300 import library
    from tblite_gb300.interface import batch_fallbacks, batch_singlepoint

    mols = {nao: _molecule(nao) for nao in set(sizes)}
    refs = {nao: _oracle(*mols[nao]) for nao in mols}
    library.set_batch_density_solver("diagonalization")
    try:
        results = batch_singlepoint([_calculator(*mols[nao]) for nao in sizes])
        assert batch_fallbacks() == 0
    finally:
        library.set_batch_density_solver("purification")
    for nao, res in zip(sizes, results):
        _check(res, refs[nao])
