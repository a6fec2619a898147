"""Chains on both sides of the length from which a single point keeps the FP64 kernels (needs a GPU).

Up to 512 orbitals a molecule whose box is longer than 34 Bohr along an axis takes the FP64
reduction, overlap factor and sums of the molecules above 512 orbitals.  Zigzag alkanes just below
and just above, a longer one, and the longer one turned onto the diagonal of its box, which brings
it below again: all of them against the oracle.

Both SCFs stop at 2e-10 (root mean square over the charges and moments); ten times that and the
square root of their number (about 700) bound a charge by 5e-8 (levels and forces, with hardnesses and
their derivatives below 1 Eh, alike), and 50 charges at up to 20 Bohr the dipole by 1e-6 if their errors
do not all add up.  The dipoles are about 0.05.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AA = 1.8897261246257702
LIMIT = 34.0


def _chain(carbons):
    """Zigzag along x, 2.4 Bohr per carbon, thermally displaced."""
    z, x = [], []
    for k in range(carbons):
        up = 1.0 if k % 2 else -1.0
        c = np.array([1.27 * k, 0.43 * up, 0.0])
        z += [6, 1, 1]
        x += [c, c + [0.0, 0.63 * up, 0.89], c + [0.0, 0.63 * up, -0.89]]
        if k in (0, carbons - 1):
            z.append(1)
            x.append(c + [-0.89 if k == 0 else 0.89, -0.63 * up, 0.0])
    x = np.array(x) * AA
    return np.array(z), x + np.random.default_rng(carbons).normal(scale=0.02, size=x.shape)


def _turned(x):
    """The x axis onto (1, 1, 1)."""
    u = np.array([[1.0, 1.0, 1.0], [1.0, -1.0, 0.0], [1.0, 1.0, -2.0]])
    return x @ (u / np.linalg.norm(u, axis=1)[:, None])


@pytest.mark.parametrize("carbons,turned,above", [(13, False, False), (14, False, True),
                                                  (20, False, True), (20, True, False)])
def test_chain(carbons, turned, above):
    from oracle import gfn2
    from tblite_gb300.interface import Calculator

    z, x = _chain(carbons)
    if turned:
        x = _turned(x)
    assert (np.ptp(x, axis=0).max() > LIMIT) == above
    calc = Calculator("GFN2-xTB", z, x)
    calc.set("accuracy", 1e-5)
    res = calc.singlepoint()
    ref = gfn2.singlepoint(gfn2.new_calc(gfn2.Molecule(z, x), accuracy=1e-5))
    assert abs(res.get("energy") - ref.energy) < 1e-9
    assert np.max(np.abs(res.get("charges") - ref.qat)) < 5e-8
    assert np.max(np.abs(res.get("orbital-energies") - ref.emo)) < 5e-8
    assert np.max(np.abs(res.get("gradient") - ref.gradient)) < 5e-8
    dipole = (x * ref.qat[:, None]).sum(0) + ref.dpat.sum(0)
    assert np.max(np.abs(res.get("dipole") - dipole)) < 1e-6
