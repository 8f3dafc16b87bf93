"""The count scans by one block per array (up to four tiles of 4,096 counts) and by three kernels (more).

A batch of n equal molecules has n times the lists of one; its scans hold 3 n + 1 counts, so n is chosen on both
sides of one tile and of the line between the two forms.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1364, 1365, 1366, 5460, 5461, 5462])
def test_lists_of_a_batch_of_equal_molecules(n):
    from xreac_gb300 import Calculator, ForceField
    from xreac_gb300.workloads import MOLECULES

    symbols, x = MOLECULES["H2O"]()
    calc = Calculator(ForceField.bundled("ffield.reax.HO.2015"))
    one = calc.evaluate(symbols, x)
    sizes = calc.list_sizes()
    many = calc.evaluate_many([dict(symbols=symbols, positions=x)] * n)
    assert calc.list_sizes() == tuple(n * v for v in sizes)
    assert [r.energy for r in many] == [many[0].energy] * n
    assert many[-1].energy == pytest.approx(one.energy, rel=1e-12)
