"""The native bookkeeping of a batch against its Python restatement: request tuples, cells, result fields."""

import copy
import pickle

import numpy as np
import pytest

host = pytest.importorskip("xreac_gb300._lib._xr_host")


def test_request_tuples():
    from xreac_gb300.calculator import _request_tuples

    full = dict(symbols=["H"], positions=[[0, 0, 0]], total_charge=1, cell=[9.0] * 3, pbc=True, initial_charges=[1.0])
    assert _request_tuples([full, dict(symbols="a", positions="b")]) == [
        (["H"], [[0, 0, 0]], 1, [9.0] * 3, True, [1.0]), ("a", "b", 0, None, None, None)]
    assert _request_tuples(iter([full]))[0][2] == 1  # another container takes the Python path
    with pytest.raises(KeyError, match="positions"):
        _request_tuples([dict(symbols=["H"])])


def _cells():
    rng = np.random.default_rng(0)
    out = [(None, None), (None, False), (np.eye(3) * 20, False), (np.eye(3) * 20, True), (np.eye(3) * 20, None),
           (np.full(3, 4.0), True), ([20.0] * 3, True), (np.eye(3) * 20, (True, True, False)), (np.eye(3) * 10.0, True),
           (-np.eye(3), True), (np.zeros(3), True), (np.full((3, 3), np.nan), True), (np.eye(3, dtype=np.float32) * 20, True),
           (np.asfortranarray(np.triu(np.full((3, 3), 20.0))), True), (np.eye(2), True), (None, True), (np.eye(3) * 1e-7, True)]
    for scale in (3.0, 8.0, 25.0):
        out += [(np.eye(3) * scale + rng.normal(0, 0.2 * scale, (3, 3)), True) for _ in range(30)]
    return out


@pytest.mark.parametrize("atoms,limit", [(3, 512), (100, 512), (3, 1)])
def test_cells(atoms, limit):
    from xreac_gb300.geometry import periodic_cell

    cells = _cells()
    items = [(["H"] * atoms, None, 0, c, p, None) for c, p in cells]
    block = np.full((len(items), 3, 3), 7.0)
    taken, rest = host.cells(items, 10.0, limit, block)
    done = dict(taken)
    for k, (c, p) in enumerate(cells):
        if (p is None and c is None) or p is False:
            assert k not in done and k not in rest
            continue
        want = periodic_cell(c, p, 10.0, atoms, limit)
        array = isinstance(c, np.ndarray) and c.dtype == np.float64 and c.flags.c_contiguous
        if want is None or not array:
            assert k in rest and k not in done  # the Python path decides, or rejects
        else:
            assert done[k] == want[2]
            np.testing.assert_array_equal(block[k], want[1])


def test_fields():
    from xreac_gb300.calculator import COMPONENTS, Evaluation, _BatchResults

    rng = np.random.default_rng(1)
    offsets, cut = [0, 3, 3 + 5], [0, 2, 9]
    batch = _BatchResults(rng.normal(size=(2, 15)), rng.normal(size=(8, 3)), rng.normal(size=(3, 8)),
                          rng.integers(0, 5, 8).astype(np.int32), rng.normal(size=(2, 3)), offsets,
                          tuple(rng.normal(size=9) for _ in range(4)), cut)
    etot = batch.energy[:, 14].tolist()
    evs = host.evaluations(Evaluation, etot, True, [(1, 1, 1), (2, 2, 2)], "replicated", batch)
    for k, ev in enumerate(evs):
        assert type(ev) is Evaluation and ev.energy == etot[k] and ev.full_derivative is True
        assert ev.cell_repetitions == [(1, 1, 1), (2, 2, 2)][k] and ev.neighbor_backend == "replicated"
        for name in ("forces", "charges", "total_bond_orders", "lone_pairs", "bond_counts", "dipole"):
            want, got = batch.field(name, k), getattr(ev, name)
            np.testing.assert_array_equal(got, want)
            assert got.dtype == want.dtype and getattr(ev, name) is got  # kept
        assert ev.components == batch.field("components", k) and tuple(ev.components) == COMPONENTS
        for got, want in zip(ev.bonds, batch.field("bonds", k)):
            np.testing.assert_array_equal(got, want)
        for name in ("nothing", "_batch2", "__deepcopy__x"):
            with pytest.raises(AttributeError, match=name):
                getattr(ev, name)
        assert not hasattr(ev, "other")
    fresh = host.evaluations(Evaluation, etot, False, [(1, 1, 1)] * 2, "x", batch)[1]
    for other in (copy.copy(fresh), copy.deepcopy(fresh), pickle.loads(pickle.dumps(fresh))):
        np.testing.assert_array_equal(getattr(other, "".join(["for", "ces"])), batch.forces[3:8])
    with pytest.raises(AttributeError):
        object.__new__(Evaluation).forces
