"""Single systems' grid teams on both sides of the lines of their block counts (152 multiprocessors): a block for every
12 rows up to two thirds of the chip (1,212 atoms), that many up to 48 rows a block (4,848), then one for every 48 rows
until the chip is full (7,296). Charges must solve the QEq equations, as in the test of larger boxes."""

import pytest
from test_gpu_qeq_rows import test_charges_of_large_boxes_solve_the_qeq_equations as check_charges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mol", [203, 204, 404, 405, 1616, 1617, 2432, 2433])
def test_charges_at_the_lines_of_the_team_sizes(n_mol):
    check_charges(n_mol)
