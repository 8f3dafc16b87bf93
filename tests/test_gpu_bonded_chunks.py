"""Angles and torsions, whose warps take between one and eight centres or middles by how many a call has.

A call's molecules must get the energies and forces that one of them gets alone, whatever the number of atoms makes
the chunks: eight atoms a warp (up to 32 atoms), one (up to 1,216), sizes on both sides of the next lines, and eight again.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [2, 3, 4, 135, 136, 270, 271, 405, 406, 945, 1100])  # 9 atoms each
def test_energies_and_forces_do_not_depend_on_the_chunks(copies):
    from xreac_gb300 import Calculator, ForceField

    x = np.array([[0.0, 0.0, 0.0], [1.52, 0.0, 0.0], [2.05, 1.32, 0.05], [-0.38, 1.02, 0.1], [-0.4, -0.5, 0.9],
                  [-0.38, -0.55, -0.88], [1.9, -0.52, 0.89], [1.88, -0.55, -0.87], [3.0, 1.28, 0.12]])
    symbols = ["C", "C", "O", "H", "H", "H", "H", "H", "H"]
    calc = Calculator(ForceField.bundled("ffield.reax.CHO.2008"))
    want = calc.evaluate(symbols, x)
    got = calc.evaluate_many([dict(symbols=symbols, positions=x)] * copies)
    for g in got:
        # sums of some tens of terms of up to 1e3 kcal/mol (per A) in another order, charges equal within 1e-12
        assert abs(g.energy - want.energy) < 1e-9
        for name, value in want.components.items():
            assert abs(g.components[name] - value) < 1e-9, name
        np.testing.assert_allclose(g.forces, want.forces, atol=1e-8, rtol=0)
