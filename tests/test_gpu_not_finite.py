"""A Fock matrix that is not finite ends in an error, and the next call is right (needs a GPU).

The fixed-point tridiagonalisation cannot hold an infinity or a NaN: it writes NaN levels, as the
FP64 kernels would have found, for one CTA (6 orbitals) and for a cluster (66).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [float("nan"), float("inf")])
@pytest.mark.parametrize("waters", [1, 11])
def test_field(waters, field):
    from tblite_gb300 import workloads
    from tblite_gb300.exceptions import TBLiteRuntimeError
    from tblite_gb300.interface import Calculator

    z, x = workloads.water_cluster_k(waters, seed=9)
    calc = Calculator("GFN2-xTB", z, x)
    calc.set("max-iter", 4)
    calc.add("electric-field", [field, 0.0, 0.0])
    with pytest.raises(TBLiteRuntimeError):
        calc.singlepoint()
    good = Calculator("GFN2-xTB", z, x)
    first, second = good.singlepoint(), good.singlepoint()
    assert np.isfinite(first.get("energy"))
    assert abs(first.get("energy") - second.get("energy")) < 1e-10
