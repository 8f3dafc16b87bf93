"""Single systems' grid teams on both sides of the lines of their block counts (152 multiprocessors): a block for every
12 rows up to two thirds of the chip (1,212 atoms), that many up to 48 rows a block (4,848), then one for every 48 rows
until the chip is full (7,296). Charges must solve the QEq equations, as in the test of larger boxes."""

import pytest
from test_gpu_qeq_rows import test_charges_of_large_boxes_solve_the_qeq_equations as check_charges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mol", [203, 204, 404, 405, 1616, 1617, 2432, 2433])
def test_charges_at_the_lines_of_the_team_sizes(n_mol):
    check_charges(n_mol)


@pytest.mark.parametrize("n_mol,graph", [(202, "replayed"), (203, "direct"), (213, "direct")])
def test_a_single_system_past_the_direct_solvers_gets_a_team(n_mol, graph):
    """Teams are launched cooperatively, which is not recorded; a cluster's launches are, and replayed at the third call."""
    from test_gpu_qeq_rows import lattice_water
    from xreac_gb300 import Calculator, ForceField

    calc = Calculator(ForceField.bundled("ffield.reax.HO.2015"))
    symbols, x, cell = lattice_water(n_mol, seed=n_mol)
    for _ in range(3):
        calc.evaluate(symbols, x, cell=cell, pbc=True)
    assert calc.last_graph == graph
