"""Kernels at the sizes where their launch, their layout or their range changes (needs a GPU).

* Fixed-point Cholesky inverse: overlaps whose smallest pivot lies just inside and just outside the
  fixed-point range (outside, the FP64 kernels take the matrix), alone and in a batch.  Its orders
  (one CTA, cluster, none) are those of the tridiagonalisation test.
* Three-body dispersion: partner lists and queues of just under and just over 32 and 64 atoms,
  and partners beyond the cutoff.
* Pipelined split GEMM: inner dimensions around a k chunk (32) and a drain window (192) with
  operands whose digits are all of one size and sign, the largest sums the accumulators can meet.

References: the CPU oracle, and for the products exact integers.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _oracle(z, x):
    from oracle import gfn2

    return gfn2.singlepoint(gfn2.new_calc(gfn2.Molecule(z, x), accuracy=1e-3))


def _calculator(z, x):
    from tblite_gb300.interface import Calculator

    calc = Calculator("GFN2-xTB", z, x)
    calc.set("accuracy", 1e-3)
    return calc


def _check(res, ref):
    """An SCF converged to 1e-9 Eh: 1e-7 Eh, 1e-6 of the charges; forces relative to the largest."""
    scale = max(1.0, np.max(np.abs(ref.gradient)))
    assert abs(res.get("energy") - ref.energy) < 1e-7 * max(1.0, abs(ref.energy))
    assert np.max(np.abs(res.get("gradient") - ref.gradient)) < 1e-6 * scale
    assert np.max(np.abs(res.get("charges") - ref.qat)) < 1e-6


def _close_pair(d):
    """Two protons d Bohr apart (overlap about 1 - d^2 / 4) and a water."""
    z = np.array([1, 1, 8, 1, 1])
    x = np.array([[0.0, 0.0, 0.0], [0.0, 0.0, d], [0.0, 0.0, 6.0], [1.4, 0.0, 7.1],
                  [-1.4, 0.0, 7.1]])
    return z, x


@pytest.mark.parametrize("d", [0.015, 0.03, 0.06])
def test_nearly_dependent_overlap(d):
    z, x = _close_pair(d)
    _check(_calculator(z, x).singlepoint(), _oracle(z, x))


def test_nearly_dependent_overlap_in_a_batch():
    from tblite_gb300 import library
    from tblite_gb300.interface import batch_fallbacks, batch_singlepoint

    ds = [0.015, 0.03, 0.06, 1.4]
    library.set_batch_density_solver("diagonalization")
    try:
        results = batch_singlepoint([_calculator(*_close_pair(d)) for d in ds])
        assert batch_fallbacks() == 0
    finally:
        library.set_batch_density_solver("purification")
    for d, res in zip(ds, results):
        _check(res, _oracle(*_close_pair(d)))


def _cluster(waters, hydrogens, far=0):
    """waters and H2 molecules on a lattice of 3.1 A, far more waters 40 Bohr away."""
    from tblite_gb300 import workloads

    rng = np.random.default_rng(waters + 7 * hydrogens + 49 * far)
    water = np.array([[0.0, 0.0, 0.0], [0.759, 0.0, 0.588], [-0.759, 0.0, 0.588]])
    h2 = np.array([[0.0, 0.0, 0.0], [0.74, 0.0, 0.0]])
    count = waters + hydrogens
    side = int(np.ceil(count ** (1 / 3)))
    z, x = [], []
    for k in range(count + far):
        kk = k if k < count else k - count
        site = np.array([kk % side, (kk // side) % side, kk // side ** 2], dtype=float) * 3.1
        if k >= count:
            site[2] += 21.2
        is_h2 = waters <= k < count
        z += [1, 1] if is_h2 else [8, 1, 1]
        x.append((h2 if is_h2 else water) + site + rng.uniform(-0.1, 0.1, size=3))
    return np.array(z), np.vstack(x) * workloads.AA2BOHR


# 3, 31, 32, 33, 64, 65 and 66 atoms, and partners beyond the cutoff of 25 Bohr
@pytest.mark.parametrize("waters,hydrogens,far", [(1, 0, 0), (9, 2, 0), (10, 1, 0), (11, 0, 0),
                                                  (20, 2, 0), (21, 1, 0), (22, 0, 0), (11, 0, 3),
                                                  (26, 1, 1)])
def test_three_body_partners(waters, hydrogens, far):
    z, x = _cluster(waters, hydrogens, far)
    _check(_calculator(z, x).singlepoint(), _oracle(z, x))


# 28, 30, 33, 35 and 64 Bohr long: from 34 Bohr on the one-molecule path keeps the FP64 kernels' sums
@pytest.mark.parametrize("carbons", [11, 12, 13, 14, 26])
def test_elongated_molecules(carbons):
    from tblite_gb300 import workloads

    z, x = workloads.alkane(carbons, seed=carbons)
    _check(_calculator(z, x).singlepoint(), _oracle(z, x))


def _product(lib, a, b, sym):
    import torch

    m, k = a.shape
    n = b.shape[1]
    ta = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    tb = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
    tc = torch.full((n, m), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = lib.tblite_gb300_split_gemm(m, n, k, ctypes.c_void_p(ta.data_ptr()),
                                     ctypes.c_void_p(tb.data_ptr()),
                                     ctypes.c_void_p(tc.data_ptr()), 1 if sym else 0, None)
    assert rc == 0
    return tc.cpu().numpy().T


@pytest.mark.parametrize("k", [1, 31, 32, 33, 191, 192, 193, 385])
@pytest.mark.parametrize("sym", [False, True])
def test_split_product_windows(k, sym):
    """Elements +-(1 - 2^-30) and +-(128 + 2^-22) / 256: exact products, so the error is the split's.

    55 fractional bits hold every element exactly; what is dropped are the products of digits p + q > 6
    (at most 21 of them per k, below 2^14 2^(-14 - 56) of the operands' scale): 2^-51 per k.
    """
    from tblite_gb300 import _build, library

    _build.build()
    lib = library.load()
    rng = np.random.default_rng(k)
    values = np.array([1.0 - 2.0 ** -30, (128.0 + 2.0 ** -22) / 256.0])
    m, n = (192, 192) if sym else (130, 66)
    a = values[rng.integers(0, 2, size=(m, k))] * np.where(rng.random((m, 1)) < 0.5, -1.0, 1.0)
    a[0] = values[0]
    a[1] = -values[1]
    b = np.ascontiguousarray(a.T) if sym else values[rng.integers(0, 2, size=(k, n))]
    c = _product(lib, a, b, sym)
    ia, ib = (a * 2.0 ** 30).astype(np.int64), (b * 2.0 ** 30).astype(np.int64)
    hi = (ia >> 15) @ ib  # exact: below 2^15 2^30 k
    lo = (ia & 32767) @ ib
    ref = hi.astype(np.longdouble) * 32768 + lo.astype(np.longdouble)
    err = np.abs(c.astype(np.longdouble) * np.longdouble(2.0 ** 60) - ref) / np.longdouble(2.0 ** 60)
    # the drop, and half a unit in the last place of the FP64 result
    assert float(np.max(err)) <= k * 2.0 ** -51 + 2.0 ** -53 * k
