"""Pair forces, which a lane of a warp adds up over its pairs of one atom: forces at the edges of the warps' chunks.

A warp takes 128 pairs of the list, so the chunks of these clusters end within an atom's pairs, at their end, and
hold atoms with few pairs (the last ones of an open system) next to atoms with many; in the periodic cells
pairs join an atom and its images (shifts of one and two cells), which must not push themselves.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(symbols, x, cell=None):
    from oracle import reaxff_oracle as oracle
    from xreac_gb300 import Calculator, ForceField

    ff = ForceField.bundled("ffield.reax.HO.2015")
    r = Calculator(ff).evaluate(symbols, x, cell=cell, pbc=cell is not None)
    o = oracle.evaluate(ff, symbols, x, cell=cell, pbc=cell is not None)
    # forces are sums of at most some hundred terms of up to 1e3 kcal/mol/A from both sides, charges equal within
    # 1e-10 (a Coulomb term of 332 kcal/mol/A follows them): the bound of the other comparisons with the oracle
    np.testing.assert_allclose(r.forces, o["forces"], atol=2e-8, rtol=0)


def _water(n_mol, box, seed):
    from xreac_gb300.workloads import water_cluster

    s = water_cluster(n_mol=n_mol, box=box, min_oo=2.4, seed=seed, jitter=0.05)
    return list(s.symbols), np.array(s.positions)


# within 10 A of each other: 120, 136, 253, 276, 496 and 528 pairs
@pytest.mark.parametrize("n", [2, 16, 17, 23, 24, 32, 33])
def test_open_clusters(n):
    symbols, x = _water((n + 2) // 3, 6.0, seed=n)
    _compare(symbols[:n], np.ascontiguousarray(x[:n]))


@pytest.mark.parametrize("side,n_mol", [(5.2, 1), (5.2, 2), (9.0, 5), (12.0, 9)])
def test_small_cells(side, n_mol):
    symbols, x = _water(n_mol, min(side, 7.0), seed=n_mol)
    _compare(symbols, x, np.array([[side, 0, 0], [0.2 * side, side, 0], [-0.1 * side, 0.1 * side, side]]))
