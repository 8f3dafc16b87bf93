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


def _matrix(ff, symbols, x, cell=None):
    """H (with the hardness on its diagonal) and chi of the QEq equations, in numpy float64."""
    import torch

    from oracle import reaxff_oracle as oracle

    i, j, s = oracle.neighbor_list(x, float(ff.general[12]), cell, None if cell is None else True)
    edges = oracle.Edges.from_sorted(i, j, s, len(x), None if cell is None else np.asarray(cell, dtype=float))
    model = oracle._Model(ff, symbols, edges)
    v = x[edges.j] - x[edges.i] + edges.offsets
    _, shield = oracle._shield_taper(model, torch.as_tensor(np.sqrt((v * v).sum(axis=1))))
    n = len(x)
    h = np.bincount(edges.i * n + edges.j, weights=14.4 * shield.numpy(), minlength=n * n).reshape(n, n)
    h[np.diag_indices(n)] += model.a["eta"]
    return h, np.asarray(model.a["chi"], dtype=float)


def _residual(h, chi, q):
    """The projected residual's norm over that of the uniform start, in the solver's norm <D^-1 r, r>^(1/2)."""
    di = 1.0 / np.diag(h)

    def norm(g):
        g = g - (di * g).sum() / di.sum()
        return np.sqrt((di * g * g).sum())

    return norm(h @ q + chi) / norm(h @ np.full(len(q), q.sum() / len(q)) + chi)


# the last correction is made without a gradient after it: whatever it was predicted to do, the charges meet the tolerance
@pytest.mark.parametrize("n", [2, 3, 5, 6, 9, 33, 96, 97, 192, 193, 288, 289, 400, 607, 608])
def test_the_charges_meet_the_tolerance(n):
    from xreac_gb300 import ForceField

    ff, calc = ForceField.bundled(FF), _calc()
    for seed in range(20 if n < 10 else 2):
        symbols, x = _cluster(n, seed=seed)
        h, chi = _matrix(ff, symbols, x)
        for charge in (0.0, 1.0):
            r = calc.evaluate(symbols, x, total_charge=charge)
            assert calc.qeq_work()[0] <= 8
            assert _residual(h, chi, r.charges) <= 1e-13
            near = r.charges + np.random.default_rng(seed).normal(0.0, 1e-4, n)
            assert _residual(h, chi, calc.evaluate(symbols, x, total_charge=charge, initial_charges=near).charges) <= 1e-13


@pytest.mark.parametrize("n_mol,side", [(8, 6.5), (27, 9.4), (60, 12.3), (110, 15.0)])
def test_the_charges_of_small_cells_meet_the_tolerance(n_mol, side):
    from xreac_gb300 import Calculator, ForceField
    from xreac_gb300.workloads import water_box

    ff = ForceField.bundled(FF)
    s = water_box(n_mol=n_mol, box=side, min_oo=2.4, seed=6)
    calc = Calculator(ff, max_expanded_atoms=100000)
    r = calc.evaluate(s.symbols, s.positions, cell=s.cell, pbc=True)
    h, chi = _matrix(ff, list(s.symbols), np.array(s.positions), s.cell)
    assert _residual(h, chi, r.charges) <= 1e-13


def _nearly_singular(n, smallest=1e-5):
    """A cluster and a force field whose hardnesses are lowered until the smallest eigenvalue of H on sum q = 0 is
    ``smallest``: the FP32 factorization (relative error some 1e-6 of the largest, about 100) no longer solves it."""
    from xreac_gb300 import ForceField

    symbols, x = _cluster(n, seed=9)
    ff = ForceField.bundled(FF)
    h, chi = _matrix(ff, symbols, x)
    z = np.linalg.svd(np.ones((1, n)))[2][1:].T
    shift = np.linalg.eigvalsh(z.T @ h @ z)[0] - smallest
    for a in {id(a): a for a in ff.atoms.values()}.values():
        a["eta"] -= shift
    k = np.ones((n + 1, n + 1))
    k[:n, :n] = h - shift * np.eye(n)
    k[n, n] = 0.0
    return ff, dict(symbols=symbols, positions=x), np.linalg.solve(k, np.append(-chi, 0.0))[:n]


# Both solves' residuals, and the matrices' rounding, are some 1e-15 of the largest entries, about 100, against a
# smallest eigenvalue of 1e-5, which nearly all of the charges (1e5 e) lie along: relative errors below 1e-6. 1e-3 tells
# right from wrong.
@pytest.mark.parametrize("n", [60, 180, 400])
def test_what_the_direct_solver_leaves_is_solved_by_cg(n):
    from xreac_gb300 import Calculator

    ff, s, want = _nearly_singular(n)
    calc, cg = Calculator(ff), Calculator(ff)
    cg.set_wait_test(polls=1 << 22)  # the CG solver, without a limit on its iterations
    for full in (False, True):
        r, c = calc.evaluate(**s, full_derivative=full), cg.evaluate(**s, full_derivative=full)
        assert calc.qeq_work()[0] > 16  # (8 refinement steps at most for the charges and as many for the adjoint)
        np.testing.assert_allclose(r.charges, want, atol=1e-3 * np.abs(want).max(), rtol=0)
        np.testing.assert_allclose(r.forces, c.forces, atol=1e-3 * np.abs(c.forces).max(), rtol=0)


def test_a_batch_of_which_some_are_left_to_cg():
    from xreac_gb300 import ForceField

    hard = {n: _nearly_singular(n) for n in (60, 180, 400)}
    easy = {n: _cluster(n, seed=n) for n in (3, 60, 99, 300, 350)}
    order = [3, -180, 60, -400, 99, -60, 300, -400, 350, -180]
    items = [hard[-n][1] if n < 0 else dict(symbols=easy[n][0], positions=easy[n][1]) for n in order]
    sets = [1 + list(hard).index(-n) if n < 0 else 0 for n in order]
    calc = _calc()
    calc.load_parameter_sets([hard[n][0] for n in hard])
    alone = _calc()
    for full in (False, True):
        got = calc.evaluate_many(items, full_derivative=full, parameter_sets=sets)
        assert calc.qeq_work()[0] > 8 * 2 * len(order)
        for n, item, g in zip(order, items, got):
            if n < 0:
                want = hard[-n][2]
                np.testing.assert_allclose(g.charges, want, atol=1e-3 * np.abs(want).max(), rtol=0)
            else:
                one = alone.evaluate(**item, full_derivative=full)
                np.testing.assert_allclose(g.charges, one.charges, atol=1e-10, rtol=0)
                np.testing.assert_allclose(g.forces, one.forces, atol=2e-8, rtol=0)
