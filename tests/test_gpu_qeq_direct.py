"""The direct QEq solvers (one block up to 288 atoms, a cluster of blocks up to 608) against the oracle's dense KKT solve of src/xreac/energy.py:89-103.

Sizes lie on both sides of their 32-row tiles, of their launch classes (32, 96, 288, 608 atoms) and of their end; the
next size takes the CG solver. Cells so small that an atom sees its own images, net charges, warm starts, adjoint solves
and batches go through it too. Charges agree to 1e-10 e, the limit of the reference's backend comparison
(scripts/validate.py:122-146), whatever the solver.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FF = "ffield.reax.HO.2015"


def _calc():
    from xreac_gb300 import Calculator, ForceField

    return Calculator(ForceField.bundled(FF))


def _cg(calc):
    calc.set_qeq(max_iterations=399)  # a bounded iteration count selects the CG solver
    return calc


def _cluster(n, seed=3):
    """The first n atoms of a water cluster at liquid density (the last molecule may be cut)."""
    from xreac_gb300.workloads import water_cluster

    m = (n + 2) // 3
    s = water_cluster(n_mol=m, box=max(4.0, (30.0 * m) ** (1 / 3)), min_oo=2.4, seed=seed, jitter=0.05)
    return list(s.symbols[:n]), np.ascontiguousarray(s.positions[:n])


def _dense(symbols, x, cell=None, charge=0.0):
    from oracle import reaxff_oracle as oracle
    from xreac_gb300 import ForceField

    ff = ForceField.bundled(FF)
    i, j, s = oracle.neighbor_list(x, float(ff.general[12]), cell, None if cell is None else True)
    m = None if cell is None else np.asarray(cell, dtype=float)
    edges = oracle.Edges.from_sorted(i, j, s, len(x), m)
    v = x[edges.j] - x[edges.i] + edges.offsets
    return oracle.qeq_charges(oracle._Model(ff, symbols, edges), np.sqrt((v * v).sum(axis=1)), charge)


SIZES = [1, 2, 3, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 129, 160, 191, 192, 193, 224, 225, 256, 257, 287, 288, 289,
         320, 321, 415, 416, 417, 512, 513, 607, 608, 609, 641, 704, 735, 736, 737]


@pytest.mark.parametrize("n", SIZES)
def test_cluster_charges(n):
    symbols, x = _cluster(n)
    calc = _calc()
    r = calc.evaluate(symbols, x, total_charge=1.0 if n % 2 else 0.0)
    np.testing.assert_allclose(r.charges, _dense(symbols, x, charge=1.0 if n % 2 else 0.0), atol=1e-10, rtol=0)
    steps = calc.qeq_work()[0]
    assert steps <= 8 if n <= 608 else steps > 8  # refinement steps, or CG iterations
    warm = calc.evaluate(symbols, x + 1e-3, total_charge=1.0 if n % 2 else 0.0, initial_charges=r.charges + 0.01)
    np.testing.assert_allclose(warm.charges, r.charges, atol=1e-10, rtol=0)


@pytest.mark.parametrize("n_mol,side", [(1, 4.0), (8, 6.5), (27, 9.4), (60, 12.3), (110, 15.0), (205, 18.4)])
def test_small_cells_with_self_images(n_mol, side):
    from xreac_gb300 import Calculator, ForceField
    from xreac_gb300.workloads import water_box

    s = water_box(n_mol=n_mol, box=side, min_oo=2.4, seed=6)
    calc = Calculator(ForceField.bundled(FF), max_expanded_atoms=100000)
    r = calc.evaluate(s.symbols, s.positions, cell=s.cell, pbc=True)
    assert calc.qeq_work()[0] <= 8 or 3 * n_mol > 608  # (larger systems take the CG solver)
    np.testing.assert_allclose(r.charges, _dense(s.symbols, s.positions, s.cell), atol=1e-10, rtol=0)


def test_batch_equals_cg_with_charge_response():
    items = [dict(symbols=s, positions=x) for s, x in (_cluster(n, seed=n) for n in (3, 30, 96, 99, 180, 288, 300, 420, 608, 650))]
    direct, cg = _calc(), _cg(_calc())
    for full in (False, True):
        a, b = direct.evaluate_many(items, full_derivative=full), cg.evaluate_many(items, full_derivative=full)
        for p, q in zip(a, b):
            np.testing.assert_allclose(p.charges, q.charges, atol=1e-10, rtol=0)
            # the forces differ by the charges' 1e-13 e times some 1e4 kcal/mol/A/e of Coulomb gradient
            np.testing.assert_allclose(p.forces, q.forces, atol=2e-8, rtol=0)
    again = direct.evaluate_many(items, full_derivative=True)
    for p, q in zip(a, again):
        assert p.energy == q.energy
        np.testing.assert_array_equal(p.charges, q.charges)


def test_a_system_the_elimination_cannot_solve_goes_to_cg():
    """Close-packed atoms give the matrix a negative eigenvalue; whether the elimination without pivoting
    copes or not, the charges are the dense solve's (the reference accepts such a system)."""
    symbols, x = _cluster(60, seed=9)
    for scale in (1.0, 0.6, 0.45):
        y = x * scale
        r = _calc().evaluate(symbols, y)
        want = _dense(symbols, y)
        np.testing.assert_allclose(r.charges, want, atol=1e-9 * max(1.0, np.abs(want).max()), rtol=0)
