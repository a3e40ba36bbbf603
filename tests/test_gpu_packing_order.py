"""The ascents of the packing classes run into one another on the stream; what follows them needs them
all. A mesh whose first class is the longest and whose last is one short warp, against the oracle."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import packing_oracle as PO  # noqa: E402

from perigrain_gb300.packing import PackMesh, get_incenter_mesh_loc  # noqa: E402

pytestmark = pytest.mark.gpu


def fans(valences, rng):
    """Fans of `v` triangles around a centre (node), side by side; the rim is the boundary."""
    v = np.asarray(valences)
    first = np.concatenate([[0], np.cumsum(v + 1)[:-1]])
    of = np.repeat(np.arange(len(v)), v)
    k = np.arange(len(of)) - np.repeat(np.cumsum(v) - v, v)
    a = 2 * np.pi * (k + 0.25 * rng.uniform(-1, 1, len(of))) / v[of]
    r = rng.uniform(0.7, 1.3, len(of))
    at = np.stack([3.0 * (np.arange(len(v)) % 64), 3.0 * (np.arange(len(v)) // 64)], 1)
    pos = np.zeros((int((v + 1).sum()), 2))
    pos[first] = at + rng.uniform(-0.1, 0.1, at.shape)
    i, j = first[of] + 1 + k, first[of] + 1 + (k + 1) % v[of]
    pos[i] = at[of] + r[:, None] * np.stack([np.cos(a), np.sin(a)], 1)
    return PackMesh(pos, np.stack([first[of], i, j], 1), i, np.stack([i, j], 1)), first


def same_circles(m, out, nodes, sample):
    """Circles of the nodes `sample` (positions in `nodes`, the nodes that have one) as the oracle's."""
    inc, rad = PO.element_circles(m.pos, m.T)
    ne = len(m.T)
    assert np.array_equal(out.incenter[:ne], inc) and np.array_equal(out.incircle_rad[:ne], rad)
    assert out.count() == ne + len(nodes)
    order = np.argsort(m.T, axis=None, kind="stable")
    flat, elem = m.T.ravel()[order], order // 3
    for p in sample:
        i = int(nodes[p])
        elems = sorted(elem[np.searchsorted(flat, i):np.searchsorted(flat, i, side="right")].tolist())
        c, r, _ = PO.maximin_node(m.pos, i, elems, inc, rad, [], False)
        assert tuple(out.incenter[ne + p]) == c and out.incircle_rad[ne + p, 0] == r, i


@pytest.mark.parametrize("last", [4, 6])
def test_short_class_behind_a_long_one(last):
    rng = np.random.default_rng(last)
    m, centres = fans([16] * 4000 + [last], rng)
    for _ in range(3):
        out = get_incenter_mesh_loc(m, modify_nodal_circles=True, gen_bdry=False)
        same_circles(m, out, centres, np.concatenate([rng.integers(0, 4000, 60), [0, 3999, 4000]]))
