"""Grid-team QEq: rows and scalars exchanged by tagged packets (blocks of at most 64 rows) or plain rows (more).

Systems of a batch that start at odd and even atoms, of sizes that leave a block one row and several, must get
the charges they get alone, and a wait that runs out inside an exchange must end the call with an error and
leave the context usable.
"""

import numpy as np
import pytest
from test_gpu_qeq_rows import lattice_water

pytestmark = pytest.mark.gpu


def calculator():
    from xreac_gb300 import Calculator, ForceField

    return Calculator(ForceField.bundled("ffield.reax.HO.2015"))


def system(n_mol):
    symbols, x, cell = lattice_water(n_mol, seed=n_mol)
    return dict(symbols=symbols, positions=x, cell=cell, pbc=True)


# after 0, 1, 2 and 3 molecules (0, 3, 6, 9 atoms): 1,029, 1,101 and 2,049 atoms in teams of one batch
@pytest.mark.parametrize("before", [0, 1, 2, 3])
def test_teams_of_a_batch_give_the_charges_of_single_calls(before):
    calc = calculator()
    teams = [system(n) for n in (343, 367, 683)]
    small = [system(before)] if before else []
    got = calc.evaluate_many(small + teams)[len(small):]
    for s, g in zip(teams, got):
        want = calc.evaluate(**s)
        # both solve to 1e-13 of the start's norm (about 0.5 sqrt(n)), and the error of the charges is that residual
        # over the smallest eigenvalue of H (above 1): 1e-13 * 0.5 * sqrt(2049) * sqrt(14) = 9e-12
        np.testing.assert_allclose(g.charges, want.charges, atol=2e-11, rtol=0)


# a wait of the setup, of the first exchange's neighbourhood and of an iteration, with packets (2,049 atoms) and
# with plain rows (12,003 atoms)
@pytest.mark.parametrize("n_mol", [683, 4001])
@pytest.mark.parametrize("fail_at", [5, 6, 7, 11])
def test_exchange_that_runs_out_raises_and_the_context_recovers(n_mol, fail_at):
    calc = calculator()
    s = system(n_mol)
    want = calc.evaluate(**s)
    calc.set_wait_test(polls=2000, fail_at=fail_at)
    with pytest.raises(RuntimeError, match="gave up"):
        calc.evaluate(**s)
    calc.set_wait_test()
    got = calc.evaluate(**s)
    assert got.energy == want.energy
    np.testing.assert_array_equal(got.charges, want.charges)


# two teams of 1,024-thread blocks (9,003 and 9,000 atoms, about 120 rows a block), whose plain rows lie side by side
def test_teams_with_plain_rows_do_not_touch_each_other():
    calc = calculator()
    boxes = [system(n) for n in (3001, 3000)]
    got = calc.evaluate_many(boxes)
    for s, g in zip(boxes, got):
        want = calc.evaluate(**s)
        # the bound above at 9,003 atoms: 1e-13 * 0.5 * sqrt(9003) * sqrt(14) = 1.8e-11 for each of the two
        np.testing.assert_allclose(g.charges, want.charges, atol=4e-11, rtol=0)
    for _ in range(3):
        for g, again in zip(got, calc.evaluate_many(boxes)):
            np.testing.assert_array_equal(again.charges, g.charges)


def test_every_wait_has_its_own_number():
    """Whatever wait of a solve a test makes run out, barrier, sum or packet exchange, the call raises; past the last one
    it does not. A solve has more waits than iterations."""
    calc = calculator()
    s = system(343)
    calc.evaluate(**s)
    iterations = calc.qeq_work()[0]
    raised = []
    for k in range(1, 4 * iterations):
        calc.set_wait_test(polls=2000, fail_at=k)
        try:
            calc.evaluate(**s)
            raised.append(False)
        except RuntimeError:
            raised.append(True)
    assert raised.index(False) > iterations
    assert not any(raised[raised.index(False):])
