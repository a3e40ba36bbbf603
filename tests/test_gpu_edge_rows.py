"""The edge list of an FP64 handle where it is built in two ways: rows that ascend are searched by
halves, others entry by entry, in any node layout, and either kind may be the other's partner."""
import numpy as np
import pytest

import _oracle
from perigrain_gb300 import Simulation, setups
from test_gpu_edge_list import _rows, _with_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["input", "shuffle", "cell"])
@pytest.mark.parametrize("dim", [2, 3])
def test_ascending_and_other_rows_together(dim, order):
    s = setups.small_pair(dim=dim, r=2.5e-4 if dim == 2 else 1.6e-4)
    rng = np.random.default_rng(dim)
    rows = []
    for i, r in enumerate(_rows(s)):
        kind = rng.integers(0, 5)
        if kind == 1:
            r = rng.permutation(r)
        elif kind == 2:  # one entry repeated, the row still in order
            r = np.sort(np.concatenate([r, r[:1]]))
        elif kind == 3:  # ascending with gaps
            r = r[rng.random(len(r)) < 0.7]
        elif kind == 4 and i % 7 == 0:
            r = r[:1]
        rows.append(r)
    s = _with_rows(s, rows)
    kw = dict(dt=2e-8, enable_fracture=1)
    gpu, ref = Simulation(s, node_order=order, **kw), _oracle.OracleSim(s, **kw)
    gpu.step(60)
    ref.step(60)
    for f in ("CurrPos", "vel", "acc", "force"):
        assert np.array_equal(gpu.field(f), ref.field(f)), f
    assert np.array_equal(gpu.bond_alive(), ref.bond_alive())
