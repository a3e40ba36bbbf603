"""A grain that is not movable: no force, no motion, no broken bond, whatever its neighbours do."""
import numpy as np
import pytest

from perigrain_gb300 import Simulation, setups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(block_size=64), dict(contact_skin=0.0)])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fixed_grain_has_no_force(precision, dim, kw):
    s = setups.small_pair(dim=dim, speed=60.0)
    s.movable = s.movable.copy()
    s.movable[1] = 0
    n0, b0 = int(s.grain_node_offset[1]), int(s.bond_offset[int(s.grain_node_offset[1])])
    sim = Simulation(s, dt=2e-8, precision=precision, **kw)
    for n in (1, 7, 60, 200):
        sim.step(n)
        assert not sim.field("force")[n0:].any() and np.isfinite(sim.field("force")).all()
        assert np.array_equal(sim.field("CurrPos")[n0:], s.pos.reshape(-1, dim)[n0:])
        assert sim.bond_alive()[b0:].all()
    assert sim.field("force")[:n0].any()
