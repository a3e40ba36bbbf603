"""The maximin packing pass treats its nodes by classes of their numbers of elements and boundary
edges and shares the constraints of 32 nodes out over a warp: fans around nodes of every class's
edge, nodes with up to four boundary edges, and node counts that do not fill a warp, bit-identical
to the oracle's plain loop."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import packing_oracle as PO  # noqa: E402

from perigrain_gb300.packing import PackMesh, get_incenter_mesh_loc  # noqa: E402

pytestmark = pytest.mark.gpu


def _fans(valences, rng):
    """Fans of `v` triangles around a centre, side by side; the rim is the boundary."""
    pos, T, bn, be = [], [], [], []
    for c, v in enumerate(valences):
        o = len(pos)
        a = 2 * np.pi * (np.arange(v) + 0.25 * rng.uniform(-1, 1, v)) / v
        r = rng.uniform(0.7, 1.3, v)
        at = np.array([3.0 * c, 0.5 * c])
        pos += [at + rng.uniform(-0.1, 0.1, 2)] + [at + r[k] * np.array([np.cos(a[k]), np.sin(a[k])]) for k in range(v)]
        for k in range(v):
            i, j = o + 1 + k, o + 1 + (k + 1) % v
            T.append((o, i, j))
            bn.append(i)
            be.append((i, j))
    return pos, T, bn, be


def _same(pos, T, bn, be, gen=True):
    m = PackMesh(np.array(pos), np.array(T), bn, np.array(be))
    out = get_incenter_mesh_loc(m, modify_nodal_circles=True, gen_bdry=gen)
    inc, rad, ok = PO.incenter_mesh_loc(m.pos, m.T, m.bdry_nodes, m.bdry_edges, True, gen)
    assert np.array_equal(out.incenter, inc) and np.array_equal(out.incircle_rad, rad)
    assert out.unpolished == int((~ok).sum())


@pytest.mark.parametrize("valences", [[4], [5, 6], [7, 8, 9], [12, 13], [16], [3] * 9 + [8, 4, 16, 6, 12]])
@pytest.mark.parametrize("gen", [True, False])
def test_fans_of_every_class(valences, gen):
    _same(*_fans(valences, np.random.default_rng(sum(valences))), gen=gen)


def test_node_with_four_boundary_edges():
    rng = np.random.default_rng(5)
    pos, T, bn, be = _fans([6, 7], rng)
    # the second fan's first rim node becomes the first fan's: two fans that touch in one node
    a, b = 1, 1 + 6 + 1
    swap = lambda t: tuple(a if k == b else k for k in t)
    shift = np.array(pos[a]) - np.array(pos[b])
    for k in range(7, len(pos)):
        pos[k] = pos[k] + shift
    # the node left over is dropped
    T, be = [swap(t) for t in T], [swap(t) for t in be]
    drop = lambda k: k - 1 if k > b else k
    pos = pos[:b] + pos[b + 1:]
    T, be = [tuple(map(drop, t)) for t in T], [tuple(map(drop, t)) for t in be]
    _same(pos, T, sorted({drop(k) for k in bn if k != b}), be)
