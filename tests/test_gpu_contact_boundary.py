"""Mixed contact decisions at the last bit: pairs of single nodes whose squared distance lies within the
contact radius in one order of rounding and beyond it in another. Every variant of the force kernel
(teams, lone warps, the grid search, the one for seven blocks an SM) decides by the same sum,
fma(z, z, fma(x, x, y y))."""
from fractions import Fraction

import numpy as np
import pytest

from perigrain_gb300 import Simulation, setups

pytestmark = pytest.mark.gpu
K = 300


def _fl(x):
    return x.numerator / x.denominator  # correctly rounded


def _sums(d):
    f = [Fraction(float(x)) for x in d]
    s = _fl(f[0] * f[0] + Fraction(float(d[1]) * float(d[1])))
    other = float(d[0]) * float(d[0]) + float(d[1]) * float(d[1])
    if len(d) == 3:
        s, other = _fl(f[2] * f[2] + Fraction(s)), other + float(d[2]) * float(d[2])
    return s, other


def _largest_within(r):
    x = r * r
    while np.sqrt(x) <= r:
        x = np.nextafter(x, np.inf)
    while np.sqrt(x) > r:
        x = np.nextafter(x, 0.0)
    return x


def _pairs(dim):
    rng = np.random.default_rng(dim)
    at, radius, hit = [], [], []
    while len(at) < K:
        d = rng.uniform(0.3, 1.0, dim) * 1e-4
        a, b = _sums(d)
        r = float(np.sqrt(min(a, b)))
        top = _largest_within(r)
        if (a <= top) != (b <= top):
            at.append(d)
            radius.append(r)
            hit.append(a <= top)
    return np.array(at), np.array(radius), np.array(hit)


def _two_nodes(dim):
    g = [setups.make_grain("disk" if dim == 2 else "sphere", 1e-4, 1.2e-4, (0.0,) * dim, dim=dim) for _ in range(2)]
    b = setups.build_setup(g, dim, 1e-4, 1e10, 0.5, 0.5, allow_wall=0)
    keep = [0, int(b.grain_node_offset[1])]
    s = b.copy()
    for k in ("pos", "disp", "vel", "acc", "extforce"):
        setattr(s, k, np.zeros(2 * dim))
    s.vol = b.vol[keep].copy()
    s.grain_node_offset = np.array([0, 1, 2], np.uint32)
    s.bond_offset, s.bond_local = np.zeros(3, np.uint64), np.zeros(0, np.uint32)
    s.bdry_offset, s.bdry_nodes = np.array([0, 1, 2], np.uint32), np.zeros(2, np.uint32)
    s.clamped_offset, s.clamped_nodes = np.zeros(3, np.uint32), np.zeros(0, np.uint32)
    return s


@pytest.mark.parametrize("dim,repeat,kw", [(2, 1, {}), (3, 1, {}), (2, 1, dict(block_size=64)), (3, 1, dict(block_size=64)),
                                           (2, 1, dict(contact_skin=0.0)), (3, 1, dict(contact_skin=0.0)),
                                           (2, 200, {}), (3, 200, {})])
def test_same_decision_in_every_variant(dim, repeat, kw):
    at, radius, hit = _pairs(dim)
    assert 0.1 < hit.mean() < 0.9
    n = K * repeat
    s = setups.concat([_two_nodes(dim)] * n)
    x = np.zeros((n, 2, dim))
    x[:, 1] = np.tile(at, (repeat, 1))
    s.pos, s.vel = x.reshape(-1), -1e5 * x.reshape(-1)  # damping acts at full strength where there is contact
    s.contact_radius = np.tile(radius, repeat)
    sim = Simulation(s, dt=1e-30, precision="mixed", self_contact=0, **kw)  # the positions do not move
    sim.step(1)
    f = (sim.field("force").reshape(repeat, K, 2, dim) != 0).any(axis=3)
    assert (f[..., 0] == hit).all() and (f[..., 1] == hit).all()
