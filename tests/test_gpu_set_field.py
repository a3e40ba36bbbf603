"""State written through set_field is in place when the call returns, whatever the next step's kernels
read: a handle whose field is written equals one created with it, at sizes above a pinned staging
buffer's."""
import numpy as np
import pytest

from perigrain_gb300 import Simulation, setups

pytestmark = pytest.mark.gpu


def _large(dim):
    if dim == 2:
        return setups.settling_2d(n_grains=40, nodes_per_grain=300)
    return setups.spheres_3d(n=8, nodes_per_grain=1200)


@pytest.mark.parametrize("order", ["input", "shuffle"])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("field,precision", [("acc", "mixed"), ("vel", "mixed"), ("acc", "fp64"), ("disp", "fp64")])
def test_written_field_equals_created_one(field, precision, dim, order):
    s = _large(dim)
    assert s.n_nodes * dim * 8 > 2 * 65536
    rng = np.random.default_rng(dim)
    scale = dict(acc=1e6, disp=1e-9, vel=2.0)[field]
    for k in range(4):
        t = s.copy()
        value = rng.uniform(-scale, scale, (s.n_nodes, dim))
        setattr(t, field, np.ascontiguousarray(value).reshape(-1))
        # (a mixed handle's fixed origin is the middle of pos + disp at creation, so its displacements
        # written later are equal to created ones only within rounding: FP64 for these)
        kw = dict(dt=1e-8, precision=precision, node_order=order)
        a, b = Simulation(s, **kw), Simulation(t, **kw)
        a.set_field(field, value)
        got = value.astype(np.float32).astype(np.float64) if (field, precision) == ("acc", "mixed") else value
        assert np.array_equal(a.field(field), got)
        a.step(3)
        b.step(3)
        for f in ("CurrPos", "vel", "acc", "force"):
            assert np.array_equal(a.field(f), b.field(f)), (f, k)
        a.close()
        b.close()
