"""The mixed force kernel with a team of warps per chunk against the one with a warp per chunk (any
block_size but 128): the same bonds and contacts added in the same order, so the same bits. Rows of
bonds below, at and above what a team forms between two barriers, several rounds of contact entries,
breaking, clamps, worm, torque, walls, the pair log, per-grain parameters, a contact list that
overflows."""
import ctypes as C

import numpy as np
import pytest

from perigrain_gb300 import Simulation, setups
from perigrain_gb300 import _native as N

pytestmark = pytest.mark.gpu
FIELDS = ("disp", "vel", "acc", "force", "CurrPos")


def _state(sim):
    out = {f: sim.field(f).copy() for f in FIELDS}
    out.update(alive=sim.bond_alive().copy(), broken=sim.break_step().copy(), status=np.array(sim.device_status()))
    return out


def _same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


CASES = {
    "pair": lambda: (setups.small_pair(dim=2, wall=True, speed=40.0), {}),
    "clamp, torque": lambda: (setups.small_pair(dim=2, clamp=True, torque=True, extforce=True), dict(enable_torque=1)),
    "worm": lambda: (setups.small_pair(dim=2, clamp=True, extforce=True), dict(timeloop=1)),
    "boundary only": lambda: (setups.small_pair(dim=2, wall=True, speed=40.0), dict(nl_bdry_only=1)),
    "no damping": lambda: (setups.small_pair(dim=2, wall=True, speed=40.0), dict(allow_damping=0)),
    "no friction": lambda: (setups.small_pair(dim=2, wall=True, speed=40.0), dict(allow_friction=0)),
    "input order": lambda: (setups.small_pair(dim=2, wall=True, speed=40.0), dict(node_order="input")),
    "3d": lambda: (setups.small_pair(dim=3, r=2.0e-4, wall=True, speed=40.0), {}),
    "32 nodes a grain": lambda: (setups.settling_2d(n_grains=4, nodes_per_grain=32), {}),
    "many contacts": lambda: (setups.small_pair(dim=2, gap=-2e-5, speed=60.0, n_grains=4), {}),
}


@pytest.mark.parametrize("name", CASES)
def test_team_equals_lone_warps(name):
    s, kw = CASES[name]()
    sims = [Simulation(s, dt=2e-8, precision="mixed", block_size=b, record_pairs=True, **kw) for b in (128, 64)]
    for n in (1, 2, 150, 250):
        got = []
        for sim in sims:
            sim.step(n)
            got.append(_state(sim))
        _same(*got)
    logs = [np.asarray(sim.pair_log(403)) for sim in sims]
    assert np.array_equal(logs[0], logs[1])


def test_team_per_grain_parameters():
    s = setups.small_pair(dim=2, wall=True, speed=40.0)
    got = []
    for b in (128, 64):
        sim = Simulation(s, dt=2e-8, precision="mixed", block_size=b)
        kn = np.array([1.0 + 0.1 * k for k in range(s.n_grains)]) * float(s.normal_stiffness[0])
        kn = np.ascontiguousarray(kn)
        N.check(N.lib().pg_set_grain_params(sim.h, None, None, N.ptr(kn, C.c_double), None, None))
        sim.step(400)
        got.append(_state(sim))
    _same(*got)


def test_team_reports_a_full_contact_list():
    s = setups.small_pair(dim=2, gap=-2e-5, speed=60.0)
    for b in (128, 64):
        sim = Simulation(s, dt=2e-8, precision="mixed", block_size=b, max_contacts=1)
        with pytest.raises(N.PerigrainError):
            sim.step(300)
            sim.synchronize()
