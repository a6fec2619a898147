"""Orbitals of a one-molecule single point: orthonormal, and solutions of the last Fock matrix.

The SCF computes the occupied levels and a few empty ones; the other vectors follow once it has
converged.  In symmetric molecules the boundary between the two falls inside a degenerate set of
empty levels (benzene: 21 of 30 orbitals, ethane 13 of 14, neopentane 22 of 32), whose vectors
have to come out orthogonal all the same.

Bounds.  Vectors of levels closer than 1e-5 of |T| are orthogonalised against one another, others
come from inverse iteration by themselves: their overlap is a few units of 2.2e-16 / 1e-5, hence
1e-10.  The orbital equations hold to what the Fock matrix of an SCF converged to 2e-8 in its charges
is off from the oracle's (hardness below 1, a few atoms each): 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AA = 1.8897261246257702


def _ring(n, radius, start=0.0):
    a = start + 2.0 * np.pi * np.arange(n) / n
    return np.stack([radius * np.cos(a), radius * np.sin(a), np.zeros(n)], axis=1)


def benzene():
    return np.array([6] * 6 + [1] * 6), np.vstack([_ring(6, 1.39), _ring(6, 2.48)]) * AA


def ethane():
    shift = np.array([0.0, 0.0, 1.16])
    x = np.vstack([[[0.0, 0.0, 0.765], [0.0, 0.0, -0.765]], _ring(3, 1.02) + shift,
                   _ring(3, 1.02, np.pi) - shift])
    return np.array([6, 6] + [1] * 6), x * AA


def neopentane():
    axes = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]]) / np.sqrt(3.0)
    z, x = [6], [np.zeros(3)]
    for u in axes:
        z += [6, 1, 1, 1]
        x.append(1.53 * u)
        for o in axes:
            if o @ u < 0.9:
                v = o - (o @ u) * u
                v /= np.linalg.norm(v)
                x.append(1.53 * u + 1.09 * (u / 3.0 - v * np.sqrt(8.0) / 3.0))
    return np.array(z), np.array(x) * AA


def water_ring(n):
    water = np.array([[0.0, 0.0, 0.0], [0.759, 0.0, 0.588], [-0.759, 0.0, 0.588]])
    z, x = [], []
    for c in _ring(n, 0.5 + 3.2 * n / 6):
        u = c / np.linalg.norm(c)
        turn = np.array([[u[0], -u[1], 0.0], [u[1], u[0], 0.0], [0.0, 0.0, 1.0]])
        z += [8, 1, 1]
        x.append(water @ turn.T + c)
    return np.array(z), np.vstack(x) * AA


def chain(carbons):
    """An alkane in zigzag along x: 2.4 Bohr per carbon."""
    z, x = [], []
    for k in range(carbons):
        up = 1.0 if k % 2 else -1.0
        c = np.array([1.27 * k, 0.43 * up, 0.0])
        z += [6, 1, 1]
        x += [c, c + [0.0, 0.63 * up, 0.89], c + [0.0, 0.63 * up, -0.89]]
        if k in (0, carbons - 1):
            z.append(1)
            x.append(c + [-0.89 if k == 0 else 0.89, -0.63 * up, 0.0])
    return np.array(z), np.array(x) * AA


MOLECULES = {"benzene": benzene, "ethane": ethane, "neopentane": neopentane,
             "water_ring4": lambda: water_ring(4), "water_ring5": lambda: water_ring(5),
             "chain16": lambda: chain(16)}


@pytest.mark.parametrize("name", list(MOLECULES))
def test_orbitals(name):
    z, x = MOLECULES[name]()
    if name == "chain16":
        assert np.ptp(x, axis=0).max() > 34.0
    _check(z, x)


# one CTA, cluster, grid, the FP64 kernels above; products on FP64 tiles and the tensor cores
@pytest.mark.parametrize("nao", [2, 7, 33, 63, 64, 65, 127, 128, 163, 256, 257, 512, 513])
def test_orbitals_by_size(nao):
    from test_gpu_tridiag import _molecule

    _check(*_molecule(nao))


def _check(z, x):
    from oracle import gfn2
    from oracle.d4 import D4
    from tblite_gb300.interface import Calculator

    calc = Calculator("GFN2-xTB", z, x)
    calc.set("accuracy", 1e-3)
    calc.set("save-integrals", True)
    res = calc.singlepoint()
    c, s = res.get("orbital-coefficients").T, res.get("overlap-matrix")  # orbitals in columns
    assert np.abs(c.T @ s @ c - np.eye(len(s))).max() < 1e-10
    ocalc = gfn2.new_calc(gfn2.Molecule(z, x), accuracy=1e-3)
    ref = gfn2.singlepoint(ocalc)
    st = gfn2.setup(ocalc)
    v = gfn2.potentials(ocalc, st, ref.qsh, ref.qat, ref.dpat, ref.qpat, D4(ocalc, st))
    f = gfn2.fock(ocalc, st, *v)[0]
    assert np.abs(f @ c - s @ c * res.get("orbital-energies")).max() < 1e-6
