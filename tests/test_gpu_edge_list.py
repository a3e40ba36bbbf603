"""The FP64 path computes a bond once for both of its nodes (the edge list built at creation): rows
that do not mirror each other, repeated entries, unsorted rows, differing intact bits of the two
directions and a last chunk that is not full give the oracle's bits, as mirrored rows do."""
import numpy as np
import pytest

import _oracle
from perigrain_gb300 import Simulation, setups

pytestmark = pytest.mark.gpu


def _rows(s):
    off = s.bond_offset.astype(np.int64)
    return [s.bond_local[off[i]:off[i + 1]].copy() for i in range(s.n_nodes)]


def _with_rows(s, rows):
    s = s.copy()
    s.bond_local = np.concatenate(rows).astype(np.uint32)
    s.bond_offset = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    return s


def _setup(dim, change):
    s = setups.small_pair(dim=dim, r=2.5e-4 if dim == 2 else 1.6e-4)
    rng = np.random.default_rng(3)
    rows = _rows(s)
    if change == "one_sided":  # a third of the entries dropped, each direction by itself
        rows = [r[rng.random(len(r)) > 1 / 3] for r in rows]
    elif change == "repeated":  # some entries twice in a row, not always in the other row too
        rows = [np.concatenate([r, r[rng.random(len(r)) < 0.2]]) for r in rows]
    elif change == "shuffled":
        rows = [rng.permutation(r) for r in rows]
    elif change == "empty":  # nodes without bonds
        rows = [r if i % 3 else r[:0] for i, r in enumerate(rows)]
    return _with_rows(s, rows)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("change", ["mirrored", "one_sided", "repeated", "shuffled", "empty", "alive_differs"])
def test_any_rows_bit_exact(dim, change):
    s = _setup(dim, change)
    kw = dict(dt=2e-8, enable_fracture=1)
    gpu, ref = Simulation(s, **kw), _oracle.OracleSim(s, **kw)
    if change == "alive_differs":
        alive = (np.random.default_rng(4).random(s.n_bonds) > 0.3).astype(np.uint8)
        gpu.set_bond_alive(alive)
        rows = _rows(s)
        off = s.bond_offset.astype(np.int64)
        kept = [r[alive[off[i]:off[i + 1]] == 1] for i, r in enumerate(rows)]
        ref = _oracle.OracleSim(_with_rows(s, kept), **kw)
    gpu.step(60)
    ref.step(60)
    for f in ("CurrPos", "vel", "acc", "force"):
        assert np.array_equal(gpu.field(f), ref.field(f)), f
    if change == "alive_differs":
        assert np.array_equal(gpu.bond_alive()[alive == 1], ref.bond_alive())
        assert not gpu.bond_alive()[alive == 0].any()
    else:
        assert np.array_equal(gpu.bond_alive(), ref.bond_alive())


@pytest.mark.parametrize("dim", [2, 3])
def test_breaking_bonds_bit_exact(dim):
    """Bonds that break in the run: both directions' intact bits and break steps."""
    s = setups.small_pair(dim=dim, r=2.5e-4 if dim == 2 else 1.6e-4, speed=120.0)
    s.snot = s.snot * 0.05
    kw = dict(dt=2e-8, enable_fracture=1)
    gpu, ref = Simulation(s, **kw), _oracle.OracleSim(s, **kw)
    gpu.step(150)
    ref.step(150)
    assert 0 < (gpu.bond_alive() == 0).sum()
    assert np.array_equal(gpu.bond_alive(), ref.bond_alive())
    assert np.array_equal(gpu.break_step() == 0, gpu.bond_alive() == 1)
    assert np.array_equal(gpu.field("vel"), ref.field("vel"))
