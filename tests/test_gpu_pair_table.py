"""Single points with and without the pair table of the electrostatics (needs a GPU).

The table (up to 1 GiB) is optional: where the device has no memory for it the pairs are evaluated in
place, one launch less.  Both forms converge to 2e-8 in the charges: the same iterations, 1e-9 Eh,
1e-7 of the charges and forces.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters,solver", [(1, "diagonalization"), (5, "diagonalization"),
                                           (33, "diagonalization"), (33, "purification")])
def test_without_memory_for_the_table(waters, solver):
    from tblite_gb300 import library, workloads
    from tblite_gb300.interface import Calculator

    z, x = workloads.water_cluster_k(waters, seed=5)
    lib = library.load()
    results, launches = [], []
    for fault in (0, 2):
        calc = Calculator("GFN2-xTB", z, x)
        calc.set("accuracy", 1e-3)
        calc.set("density-solver", solver)
        lib.tblite_gb300_set_calculator_fault(calc._ctx, calc._calc, fault)
        library.context_check(calc._ctx)
        before = lib.tblite_gb300_get_launch_count()
        results.append(calc.singlepoint())
        launches.append(lib.tblite_gb300_get_launch_count() - before)
    with_table, without = results
    assert launches[1] == launches[0] - 1
    assert abs(with_table.get("energy") - without.get("energy")) < 1e-9
    for key in ("charges", "gradient"):
        assert np.max(np.abs(with_table.get(key) - without.get(key))) < 1e-7
