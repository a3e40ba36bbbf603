"""A run of n steps, whose force kernels make the next step's position update, against n runs of one
step: the same bits, at run lengths below, at and above the captured graph's, with what ends or
changes a step inside a run (walls, clamps, torque, worm, the pair log, rebuilt lists, no lists)."""
import numpy as np
import pytest

from perigrain_gb300 import Simulation, setups

pytestmark = pytest.mark.gpu
FIELDS = ("disp", "vel", "acc", "force", "CurrPos")

CASES = {
    "walls": (dict(wall=True, speed=40.0), dict(record_pairs=True)),
    "clamp, torque": (dict(clamp=True, torque=True, extforce=True), dict(enable_torque=1)),
    "worm": (dict(clamp=True, extforce=True), dict(timeloop=1)),
    "small skin": (dict(wall=True, speed=80.0), dict(contact_skin=0.02)),
    "grid search": (dict(wall=True, speed=40.0), dict(contact_skin=0.0)),
}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", CASES)
def test_run_equals_single_steps(name, precision, dim):
    scene, kw = CASES[name]
    s = setups.small_pair(dim=dim, **scene)
    a = Simulation(s, dt=2e-8, precision=precision, **kw)
    b = Simulation(s, dt=2e-8, precision=precision, **kw)
    for n in (1, 2, 3, 7, 8, 9, 16, 17, 25, 90):
        a.step(n)
        for _ in range(n):
            b.step(1)
        for f in FIELDS:
            assert np.array_equal(a.field(f), b.field(f)), (n, f)
        assert np.array_equal(a.bond_alive(), b.bond_alive()) and np.array_equal(a.break_step(), b.break_step())
        assert np.array_equal(a.wall(), b.wall()) and np.array_equal(a.reaction(), b.reaction())
        assert a.device_status() == b.device_status()
