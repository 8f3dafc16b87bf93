"""Edges placed from rows kept by the count pass (image scan or cell list), against the oracle's list edge for edge.

Covers rows that fill their slots and rows that do not fit (a dense cluster in a large cell: the call scans again),
one and several images a pair, partly periodic cells, unwrapped positions, and sizes on both sides of the
warps' 32 targets and of the 1,024-atom strides of the row bitmaps.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FF = "ffield.reax.HO.2015"


def _check(symbols, x, cell=None, pbc=None, cells=None, calls=2):
    from oracle import reaxff_oracle as oracle
    from xreac_gb300 import Calculator, ForceField

    ff = ForceField.bundled(FF)
    calc = Calculator(ff, max_expanded_atoms=1 << 30)
    calc.set_cell_list(cells)
    want = oracle.neighbor_list(x, float(ff.general[12]), cell, pbc)
    first = None
    for _ in range(calls):
        r = calc.evaluate(symbols, x, cell=cell, pbc=pbc)
        for got, ref in zip(calc.neighbor_list(), want):
            np.testing.assert_array_equal(got, ref)
        first = first or r
        assert r.energy == first.energy
        np.testing.assert_array_equal(r.total_bond_orders, first.total_bond_orders)
    return calc


def _water(n_mol, seed, side=None):
    from xreac_gb300.workloads import water_cluster

    s = water_cluster(n_mol=n_mol, box=side or max(4.0, (30.0 * n_mol) ** (1 / 3)), min_oo=2.4, seed=seed, jitter=0.05)
    return list(s.symbols), np.array(s.positions)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 191, 300])
def test_open_systems(n):
    symbols, x = _water((n + 2) // 3, seed=n)
    _check(symbols[:n], np.ascontiguousarray(x[:n]))


@pytest.mark.parametrize("cells", [False, True])
@pytest.mark.parametrize("side,pbc", [(9.0, True), (12.0, True), (17.0, True), (21.0, True), (30.0, True),
                                      (12.0, (True, False, True)), (21.0, (False, True, False))])
def test_periodic_systems(side, pbc, cells):
    symbols, x = _water(20 if side < 12 else 50, seed=int(side), side=side if side < 12 else min(side, 12.0))
    shear = np.array([[side, 0, 0], [0.2 * side, side, 0], [-0.1 * side, 0.15 * side, side]])
    rng = np.random.default_rng(2)
    x = x + rng.integers(-2, 3, (len(x) // 3, 3)).repeat(3, axis=0) * np.where(pbc, 1, 0) @ shear
    calc = _check(symbols, x, shear, pbc, cells=cells)
    assert calc.list_info()[0] == ("cells" if cells else "scan")


@pytest.mark.parametrize("cells,n_mol", [(False, 200), (True, 200), (None, 400)])
def test_rows_longer_than_the_mean_density_suggests(cells, n_mol):
    symbols, x = _water(n_mol, seed=7)  # liquid density in a corner of a nearly empty cell
    _check(symbols, x, np.diag([90.0] * 3), True, cells=cells, calls=3)


@pytest.mark.parametrize("n_mol", [341, 342, 683, 1025])
def test_row_bitmaps(n_mol):
    from xreac_gb300.workloads import water_box

    s = water_box(n_mol=n_mol, box=max(20.5, (31.0 * n_mol) ** (1 / 3)), min_oo=2.4, seed=n_mol)
    _check(list(s.symbols), np.array(s.positions), s.cell, True, cells=True, calls=1)


# far more row slots than edges: 298 molecules 8 A apart, alone and in a periodic cell, by image scan and cell list
@pytest.mark.parametrize("cells", [False, True])
@pytest.mark.parametrize("periodic", [False, True])
def test_calls_within_a_reservation_allocate_nothing(periodic, cells):
    from oracle import reaxff_oracle as oracle
    from xreac_gb300 import Calculator, ForceField
    from xreac_gb300.workloads import MOLECULES

    ff = ForceField.bundled(FF)
    symbols, water = MOLECULES["H2O"]()
    sites = 8.0 * np.stack(np.unravel_index(np.arange(298), (7, 7, 7)), axis=1)
    x = (sites[:, None, :] + np.asarray(water)).reshape(-1, 3)
    symbols = list(symbols) * 298
    cell = np.diag([56.0] * 3) if periodic else None
    want = oracle.neighbor_list(x, float(ff.general[12]), cell, periodic or None)
    calc = Calculator(ff)
    calc.set_cell_list(cells)
    calc.reserve(894, 1, edges_per_atom=len(want[0]) / 894, bonds_per_atom=3)
    before = calc.memory()
    calc.evaluate(symbols, x, cell=cell, pbc=periodic)
    assert calc.memory() == before
    for got, ref in zip(calc.neighbor_list(), want):
        np.testing.assert_array_equal(got, ref)


def test_slots_follow_the_longest_row():
    """Rows that did not fit once fit from the next call on, and other systems keep their slots."""
    from xreac_gb300 import Calculator, ForceField

    calc = Calculator(ForceField.bundled(FF), max_expanded_atoms=1 << 30)
    calc.set_cell_list(False)
    symbols, x = _water(200, seed=7)  # liquid density in a corner of a nearly empty cell
    cell = np.diag([90.0] * 3)
    for _ in range(2):
        calc.evaluate(symbols, x, cell=cell, pbc=True)
    held = calc.memory()
    longest = np.bincount(calc.neighbor_list()[0]).max()
    assert 2 * held["candidates"] >= len(x) * longest
    for _ in range(10):
        calc.evaluate(symbols, x, cell=cell, pbc=True)
    assert calc.memory() == held
    symbols, x = _water(100, seed=8)
    calc.evaluate(symbols, x, cell=np.diag([14.5] * 3), pbc=True)
    assert calc.memory()["candidates"] == held["candidates"]


def test_threads_whose_rows_need_different_shared_memory():
    """Row bitmaps of more than 48 KB a block, of two sizes, from two contexts at once (the limit is a setting of
    the process)."""
    import threading

    from test_gpu_qeq_rows import lattice_water

    from xreac_gb300 import Calculator, ForceField

    got, errors = {}, []

    def work(n_mol):
        try:
            calc = Calculator(ForceField.bundled(FF))
            symbols, x, cell = lattice_water(n_mol, seed=n_mol)
            got[n_mol] = [calc.evaluate(symbols, x, cell=cell, pbc=True).energy for _ in range(12)]
        except Exception as exc:  # noqa: BLE001 (reported by the main thread)
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(n,)) for n in (11000, 13800)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert all(len(set(v)) == 1 for v in got.values()) and len(got) == 2


def test_a_second_smaller_reservation_keeps_the_first():
    from xreac_gb300 import Calculator, ForceField

    calc = Calculator(ForceField.bundled(FF))
    calc.set_cell_list(False)
    rng = np.random.default_rng(3)
    x = 8.0 * np.stack(np.unravel_index(np.arange(800), (10, 10, 8)), axis=1) + rng.uniform(-0.1, 0.1, (800, 3))
    calc.reserve(800, 1, edges_per_atom=20, bonds_per_atom=1)
    calc.reserve(10, 1, edges_per_atom=20, bonds_per_atom=1)
    before = calc.memory()
    calc.evaluate(["O"] * 800, x)
    assert calc.memory() == before
