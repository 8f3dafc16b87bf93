"""QEq of large single systems: the row solver whose rows lie in shared memory or stream from the L2 cache.

The charges of a periodic water box must solve the QEq equations of src/xreac/energy.py:89-103, whatever the
number of atoms does to the solver's layout: whole tiles of 32 rows or equal shares per block (the line lies at
64 rows), rows in shared memory or streamed (from about 11,000 atoms), with or without room for the FP64 stage
(26,624 atoms). The residual H q + chi is formed in numpy float64 from the oracle's shields over the exported
neighbour list; it is the same multiplier for every atom.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice_water(n_mol, seed):
    """Water on jittered lattice sites at about 1 g/cm^3 in a periodic cube (quick at any size)."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n_mol ** (1 / 3) - 1e-9))
    side = max((n_mol * 29.9) ** (1 / 3), 2.95 * m)
    pick = np.sort(rng.choice(m**3, n_mol, replace=False))
    o = np.stack((pick // m**2, pick // m % m, pick % m), axis=1) * (side / m)
    half = np.deg2rad(52.25)
    a = rng.normal(size=(n_mol, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(n_mol, 3)))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    h1, h2 = (o + 0.97 * (np.cos(half) * a + s * np.sin(half) * b) for s in (1, -1))
    x = np.stack((o, h1, h2), axis=1).reshape(-1, 3)
    return ["O", "H", "H"] * n_mol, x + rng.normal(0.0, 0.05, x.shape), np.diag([side] * 3)


# 9,726 and 9,732 atoms: 64 and 65 rows a block on 152 blocks; 11,700 and 12,003: the rows no longer fit; 27,003:
# more than 8 bytes an atom leave room for
@pytest.mark.parametrize("n_mol", [3242, 3244, 3900, 4001, 9001])
def test_charges_of_large_boxes_solve_the_qeq_equations(n_mol):
    from oracle import reaxff_oracle as oracle
    from xreac_gb300 import Calculator, ForceField

    import torch

    ff = ForceField.bundled("ffield.reax.HO.2015")
    symbols, x, cell = lattice_water(n_mol, seed=n_mol)
    calc = Calculator(ff)
    r = calc.evaluate(symbols, x, cell=cell, pbc=True)
    i, j, s = calc.neighbor_list()
    edges = oracle.Edges.__new__(oracle.Edges)
    edges.i, edges.j, edges.n = i.astype(np.int64), j.astype(np.int64), len(x)
    model = oracle._Model(ff, symbols, edges)
    v = x[j] - x[i] + s @ cell
    _, shield = oracle._shield_taper(model, torch.as_tensor(np.sqrt((v * v).sum(axis=1))))
    residual = np.bincount(i, weights=14.4 * shield.numpy() * r.charges[j], minlength=len(x))
    residual += model.a["eta"] * r.charges + model.a["chi"]
    # the solver stops at 1e-13 of the start's norm, which is about 0.5 sqrt(n) in units of sqrt(D) (D about 14): even
    # all of it in one atom is below 1e-13 * 0.5 * sqrt(n) * sqrt(14) = 3e-11 for these sizes
    assert np.abs(residual - residual.mean()).max() < 1e-10
    assert abs(r.charges.sum()) < 1e-10
