"""The exported bonds come in bond order, whole, whatever their number per atom and per 128-bond tile.

Up to four bonds per atom arrive with the call's other results, any further ones in a second copy; compressed
clusters have more. Each atom's exported orders add up to its total bond order (src/xreac/energy.py:167-178), which
comes from another kernel: the same sums in another order, a few ulps of at most some 20 terms.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,many", [(1.0, False), (0.62, True), (0.55, True)])
@pytest.mark.parametrize("n_mol", [1, 20, 64, 150])
def test_exported_bonds_add_up(n_mol, scale, many):
    from xreac_gb300 import Calculator, ForceField
    from xreac_gb300.workloads import water_cluster

    s = water_cluster(n_mol=n_mol, box=max(4.0, (30.0 * n_mol) ** (1 / 3)), min_oo=2.4, seed=n_mol, jitter=0.05)
    r = Calculator(ForceField.bundled(s.force_field)).evaluate(s.symbols, s.positions * scale)
    i, j, shift, order = r.bonds
    n = len(s.symbols)
    if many and n_mol >= 64:
        assert len(i) > 4 * n + 64
    keys = list(zip(i, j))
    assert keys == sorted(keys) and len(set(keys)) == len(keys) and (i < j).all() and (shift == 0).all()
    assert (order > 0).all()
    np.testing.assert_allclose(r.bond_orders.sum(axis=1), r.total_bond_orders, rtol=1e-13, atol=1e-13)
