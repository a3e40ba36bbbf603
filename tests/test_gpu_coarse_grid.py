"""Contact search where the grid is coarser than the contact radius (few cells for a wide box, as with
debris that flies apart), so that rows of cells hold from none to hundreds of nodes: FP64 against the
oracle, mixed against the same run with more cells."""
import numpy as np
import pytest

import _oracle as O
from perigrain_gb300 import Simulation, setups

pytestmark = pytest.mark.gpu
FIELDS = ("CurrPos", "vel", "acc", "force")


def _scene(dim, far):
    """Two grains that collide and fracture, a third one `far` away."""
    s = setups.small_pair(dim=dim, r=2.5e-4 if dim == 2 else 1.6e-4, speed=60.0, n_grains=3)
    s.pos = s.pos.copy()
    s.pos.reshape(-1, dim)[int(s.grain_node_offset[2]):, 0] += far
    return s


@pytest.mark.parametrize("far", [0.0, 2e-2, 2.0])
@pytest.mark.parametrize("dim", [2, 3])
def test_grid_search_in_coarse_cells(dim, far):
    s = _scene(dim, far)
    kw = dict(dt=2e-8, enable_fracture=1)
    r = O.OracleSim(s, **kw)
    r.step(250)
    assert r.pair_log_all()[0].sum() > 0
    for cells in (1, 0):
        g = Simulation(s, record_pairs=True, contact_skin=0.0, cells_per_node=cells, **kw)
        g.step(250)
        for f in FIELDS:
            assert np.array_equal(g.field(f), r.field(f)), f
        assert np.array_equal(g.break_step(), r.break_step())
        assert np.array_equal(np.array(g.pair_log(250)), np.array(r.pair_log_all()))
    sims = [Simulation(s, precision="mixed", contact_skin=0.0, cells_per_node=c, **kw) for c in (1, 64)]
    for sim in sims:
        sim.step(250)
    for f in FIELDS:
        assert np.array_equal(sims[0].field(f), sims[1].field(f)), f


def test_grid_search_reports_a_full_contact_list():
    s = setups.small_pair(dim=2, gap=-2e-5, speed=60.0)
    for precision in ("fp64", "mixed"):
        sim = Simulation(s, dt=2e-8, precision=precision, contact_skin=0.0, max_contacts=1)
        with pytest.raises(Exception):
            sim.step(300)
            sim.synchronize()


@pytest.mark.parametrize("skin", [0.25, 0.02])
@pytest.mark.parametrize("far", [0.0, 2e-2, 2.0])
@pytest.mark.parametrize("dim", [2, 3])
def test_lists_from_coarse_cells(dim, far, skin):
    s = _scene(dim, far)
    kw = dict(dt=2e-8, enable_fracture=1)
    r = O.OracleSim(s, **kw)
    r.step(250)
    for cells in (1, 0):
        g = Simulation(s, record_pairs=True, contact_skin=skin, cells_per_node=cells, **kw)
        g.step(250)
        for f in FIELDS:
            assert np.array_equal(g.field(f), r.field(f)), f
        assert np.array_equal(g.break_step(), r.break_step())
        assert np.array_equal(np.array(g.pair_log(250)), np.array(r.pair_log_all()))
    sims = [Simulation(s, precision="mixed", contact_skin=k, cells_per_node=1, **kw) for k in (skin, 0.0)]
    for sim in sims:
        sim.step(250)
    for f in FIELDS:
        assert np.array_equal(sims[0].field(f), sims[1].field(f)), f


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_full_candidate_list_is_reported(precision):
    s = setups.two_disk_collision(gap=-2e-4)
    s.contact_radius = s.contact_radius * 6.0
    sim = Simulation(s, dt=2e-8, precision=precision, self_contact=0)
    with pytest.raises(Exception):
        sim.step(2)
        sim.synchronize()
