"""Kernel variants that only large inputs reach: force kernels compiled for six and seven blocks an SM,
the packing ascent with full warps of nodes, the bond builder above its kept scratch."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

from perigrain_gb300 import Simulation, setups
from perigrain_gb300 import _native as N
from perigrain_gb300.packing import PackMesh, get_incenter_mesh_loc, rect_mesh

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
pytestmark = pytest.mark.gpu


def _copies(one, blocks):
    """Copies of a small scene as one batch whose chunks fill the GPU to `blocks` blocks an SM."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (sms * 4 * blocks * 32 - 32) // one.n_nodes
    return setups.concat([one] * n), n


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("blocks", [6, 7])
@pytest.mark.parametrize("skin", [0.25, 0.0])
def test_batch_of_copies_equals_one(skin, blocks, dim):
    # (walls in 2D only: a handle holds 16384 wall records a step, and 3D scenes touch theirs all over)
    one = setups.small_pair(dim=dim, r=2.5e-4 if dim == 2 else 1.6e-4, wall=dim == 2, speed=60.0)
    one.snot = one.snot * 0.1
    s, n = _copies(one, blocks)
    for precision in ("mixed", "fp64"):
        kw = dict(dt=2e-8, precision=precision, contact_skin=skin)
        a, b = Simulation(one, **kw), Simulation(s, **kw)
        for steps in (1, 200):
            a.step(steps)
            b.step(steps)
        for f in ("CurrPos", "vel", "acc", "force"):
            want = a.field(f)
            got = b.field(f).reshape((n,) + want.shape)
            assert (got == want).all(), (precision, f)
        assert (b.break_step().reshape(n, -1) == a.break_step()).all() and a.break_step().any()
        assert a.device_status()[0] == b.device_status()[0] == 0
        a.close()
        b.close()


def test_ascent_with_full_warps():
    import packing_oracle as PO
    from test_gpu_packing_order import fans

    rng = np.random.default_rng(3)
    m = rect_mesh(335, 305, width=2.0, height=1.9, jitter=0.25, seed=5)
    f, _ = fans([4, 5, 9, 10, 12, 13, 16] * 5 + [3], rng)  # classes with a last warp that is not full
    k = len(m.pos)
    mesh = PackMesh(np.concatenate([m.pos, f.pos + 10.0]), np.concatenate([m.T, f.T + k]),
                    np.concatenate([m.bdry_nodes, f.bdry_nodes + k]), np.concatenate([m.bdry_edges, f.bdry_edges + k]))
    inner = np.setdiff1d(np.arange(len(mesh.pos)), mesh.bdry_nodes)
    assert len(inner) > 100000 and len(inner) % 32
    out = get_incenter_mesh_loc(mesh, modify_nodal_circles=True, gen_bdry=False)
    inc, rad = PO.element_circles(mesh.pos, mesh.T)
    ne = len(mesh.T)
    assert np.array_equal(out.incenter[:ne], inc) and out.count() == ne + len(inner)
    order = np.argsort(mesh.T, axis=None, kind="stable")
    flat, elem = mesh.T.ravel()[order], order // 3
    sample = np.concatenate([rng.integers(0, len(inner), 400), np.arange(len(inner) - 36, len(inner)), [0]])
    for p in sample:
        i = int(inner[p])
        elems = sorted(elem[np.searchsorted(flat, i):np.searchsorted(flat, i, side="right")].tolist())
        c, r, _ = PO.maximin_node(mesh.pos, i, elems, inc, rad, [], False)
        assert tuple(out.incenter[ne + p]) == c and out.incircle_rad[ne + p, 0] == r, i


@pytest.mark.parametrize("dim,n", [(2, 262144), (2, 262145), (2, 300000), (3, 270000)])
def test_bonds_above_the_kept_scratch(dim, n):
    import torch

    rng = np.random.default_rng(n)
    side = int(round(n ** (1 / dim))) + 1
    p = np.stack([a.ravel() for a in np.meshgrid(*[np.arange(side)] * dim, indexing="ij")], 1)[:n]
    p = p + rng.uniform(-0.1, 0.1, p.shape)
    delta = 2.0 if dim == 2 else 1.5
    ref = setups.bond_pairs(p, delta)
    d_pos = torch.from_numpy(np.ascontiguousarray(p)).cuda()
    d_pairs = torch.empty((len(ref), 2), dtype=torch.int32, device="cuda")
    count = C.c_uint64()
    rc = N.lib().pg_build_bonds(C.c_void_p(d_pos.data_ptr()), n, dim, delta, C.c_void_p(d_pairs.data_ptr()), len(ref),
                                C.byref(count), None)
    assert rc == N.PG_OK and count.value == len(ref)
    assert np.array_equal(d_pairs.cpu().numpy(), ref)
