"""The work a user of perigrain_gb300 has it do, as cases that can be timed and compared.

Each case is one pass of a program that keeps its handle: an output interval of a simulation
(`modulo` = 100 steps, then the tc_/wall_ snapshot), a forward and backward pass of the gradient
path, a bond list, a packing, a post-processing call. The scenes and their sizes are those of
`perigrain_gb300.setups` (the five benchmark configurations and their generators) and of bench.py.

`exact` restates the reference's time step in torch, in 64 bits and without the engine.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from perigrain_gb300 import Simulation, grad, packing, setups
from perigrain_gb300 import _native as N

STEPS = 100  # the configurations' `modulo`: steps between two outputs


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def _run(name, scene, precision, steps=STEPS, skin=0.25, bdry_only=False, **size):
    return dict(name=name, kind="run", scene=scene, precision=precision, steps=steps, skin=skin,
                bdry_only=bdry_only, **size)


def listed():
    return [
        # one two-disk impact (configuration 0): 2,498 nodes. The smallest runs of the reference's
        # own experiments; a step is launches and latency. Both precisions: FP64 is the default and
        # the drop-in's, mixed the fast path.
        _run("pair_mixed", "pair", "mixed", h=5e-5),
        _run("pair_fp64", "pair", "fp64", h=5e-5),
        # 500 grains compressed in a box, about 30 thousand nodes: the size of the reference's own
        # logged bulk run (499 grains); walls, friction and contact from the first step.
        _run("bulk_fp64", "bulk", "fp64", grains=500, nodes=55),
        # mixed shapes in a walled box under gravity (configuration 1): 115,899 nodes
        _run("settling_mixed", "settling", "mixed", grains=400, nodes=300),
        # 64 spheres in three dimensions (configuration 2): 128,448 nodes, 84 bonds each
        _run("spheres_mixed", "spheres", "mixed", grains=64, nodes=2000),
        _run("spheres_fp64", "spheres", "fp64", grains=64, nodes=2000),
        # 256 independent two-grain impacts in one handle (configuration 3): 390,419 nodes, ten
        # million bonds, the largest batch
        _run("ensemble_mixed", "ensemble", "mixed", grains=256, h=6.25e-5),
        _run("ensemble_fp64", "ensemble", "fp64", grains=256, h=6.25e-5),
        # objectives and parameter gradients of the 50-grain compaction (configuration 4)
        dict(name="grad_mixed", kind="grad", precision="mixed", grains=50, nodes=400, steps=300, every=100),
        # the bond list of one large grain (bench.py's bond builder size)
        dict(name="bonds_200k", kind="bonds", dim=2, nodes=200_000),
        # incircle packing of a mesh, nodal circles included (bench.py's packing size)
        dict(name="pack_400k", kind="pack", nx=800, ny=500, modify=True),
        # the time series of an output step without files: grain means, damage, volume fraction
        dict(name="post_390k", kind="post", grains=256, h=6.25e-5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["grad", "bonds", "pack", "post"])
    if kind == "run":
        scene = rng.choice(["pair", "bulk", "settling", "spheres", "ensemble"])
        precision = rng.choice(["mixed", "fp64"])
        c = dict(kind="run", scene=scene, precision=precision, steps=int(_log(rng, 5, 101)),
                 skin=rng.choice([0.25, 0.25, 0.25, 0.5, 0.0]), bdry_only=rng.random() < 0.15)
        if scene == "pair":
            c["h"] = _log(rng, 1.5e-5, 2.5e-4)
        elif scene == "ensemble":
            c.update(grains=int(_log(rng, 1, 200)), h=rng.uniform(6.25e-5, 1.5e-4))
        elif scene == "spheres":
            c.update(grains=int(_log(rng, 1, 60)), nodes=int(_log(rng, 60, 1900)))
        else:
            c.update(grains=int(_log(rng, 4, 390)), nodes=int(_log(rng, 30, 300)))
        return c
    if kind == "grad":
        return dict(kind="grad", precision=rng.choice(["mixed", "fp64"]), grains=int(_log(rng, 2, 50)),
                    nodes=int(_log(rng, 60, 400)), steps=rng.randint(20, 200), every=rng.choice([25, 50, 100]))
    if kind == "bonds":
        return dict(kind="bonds", dim=rng.choice([2, 2, 3]), nodes=int(_log(rng, 100, 180_000)))
    if kind == "pack":
        return dict(kind="pack", nx=int(_log(rng, 6, 700)), ny=int(_log(rng, 6, 480)), modify=rng.random() < 0.7)
    return dict(kind="post", grains=int(_log(rng, 1, 200)), h=rng.uniform(6.25e-5, 1.5e-4))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _scene(scene, h, grains, nodes):
    """The meshes, bonds and material of a scene, as a setup file holds them."""
    if scene == "pair":
        return setups.two_disk_collision(h=h)
    if scene == "ensemble":
        return setups.collision_ensemble(n_inst=grains, h=h)
    if scene == "settling":
        return setups.settling_2d(n_grains=grains, nodes_per_grain=nodes)
    if scene == "spheres":
        return setups.spheres_3d(n=grains, nodes_per_grain=nodes)
    return setups.compaction_2d(n_grains=grains, nodes_per_grain=nodes)


def _base(case):
    scene = case.get("scene") or ("bulk" if case["kind"] == "grad" else "ensemble")
    return _scene(scene, case.get("h"), case.get("grains"), case.get("nodes")), scene


def _setup(case, seed):
    """The scene with this seed's velocities: the impact speeds vary by 10 %, grains at rest get a
    velocity of up to 4 m/s per component, as poured or stirred ones have, and every grain spins and
    deforms at about 1 m/s at its edge, as grains do once they have touched others."""
    base, scene = _base(case)
    s = base.copy()
    rng = np.random.default_rng(seed)
    of = np.repeat(np.arange(s.n_grains), np.diff(s.grain_node_offset.astype(np.int64)))
    v = s.vel.reshape(-1, s.dim)
    if scene in ("pair", "ensemble"):
        v = v * (1 + rng.uniform(-0.1, 0.1, s.n_grains))[of, None]
    else:
        v = rng.uniform(-4, 4, (s.n_grains, s.dim))[of]
    x = s.pos.reshape(-1, s.dim)
    count = np.bincount(of).astype(np.float64)
    x = x - np.stack([np.bincount(of, x[:, c]) / count for c in range(s.dim)], 1)[of]
    size = np.sqrt(np.maximum(np.bincount(of, (x * x).sum(1)) / count, 1e-30))[of]
    v = v + np.einsum("nij,nj->ni", rng.uniform(-1, 1, (s.n_grains, s.dim, s.dim))[of], x / size[:, None])
    s.vel = np.ascontiguousarray(v).reshape(-1)
    if case["kind"] == "post":  # gravity: without it a grain's summed force is its rounding alone
        s.extforce.reshape(-1, s.dim)[:, 1] = -9.8 * setups.RHO
    return s


def _dt(scene):
    return 1e-8 if scene in ("settling", "spheres") else 2e-8


def _sim(case, seed):
    s = _setup(case, seed)
    return Simulation(s, dt=_dt(_base(case)[1]), precision=case.get("precision", "fp64"),
                      contact_skin=case.get("skin", 0.25), nl_bdry_only=int(case.get("bdry_only", False)))


def _grain_points(case, seed):
    """One disk or ball of about `nodes` jittered grid nodes of spacing 1, and its horizon."""
    dim, n = case["dim"], case["nodes"]
    r = math.sqrt(n / math.pi) if dim == 2 else (0.75 * n / math.pi) ** (1 / 3)
    pos, _ = setups.grid_nodes("disk" if dim == 2 else "sphere", r, 1.0, dim=dim, jitter=0.1,
                               rng=np.random.default_rng(seed))
    return np.ascontiguousarray(pos), 3.0


def _bond_capacity(n, dim):
    return max(16, n * (20 if dim == 2 else 64))


def _mesh(case, seed):
    return packing.rect_mesh(case["nx"], case["ny"], width=2.0, height=1.25, jitter=0.25, seed=seed)


def _intact(case, seed):
    """A fractured state's bonds: 5 % broken, both directions of a bond alike."""
    s = _base(case)[0]
    i, j = _bond_ends(s)
    lo, hi = np.minimum(i, j).astype(np.uint64), np.maximum(i, j).astype(np.uint64)
    with np.errstate(over="ignore"):
        x = (lo * np.uint64(0x9E3779B97F4A7C15)) ^ (hi * np.uint64(0xC2B2AE3D27D4EB4F)) ^ np.uint64(seed + 1)
        x = (x ^ (x >> np.uint64(29))) * np.uint64(0xBF58476D1CE4E5B9)
    return ((x >> np.uint64(40)) % np.uint64(20) != 0).astype(np.uint8)


def prepare(case, seed):
    if case["kind"] == "run":
        sim = _sim(case, seed)
        items = ["CurrPos", "vel", "acc", "force", "bond_alive"]
        if sim.setup.allow_wall.any():
            items += ["wall", "reaction"]
        return dict(kind="run", sim=sim, steps=case["steps"], items=items, out=sim.snapshot_buffers(items))
    if case["kind"] == "grad":
        sim = _sim(case, seed)
        rng = np.random.default_rng(seed + 1)
        run_ = grad.GradRun(sim, case["steps"], checkpoint_every=case["every"])
        return dict(kind="grad", run=run_, rbar=rng.uniform(-1, 1, (run_.I, 2 * run_.dim, run_.dim)),
                    kbar=rng.uniform(0.5, 1.5, run_.I))
    if case["kind"] == "bonds":
        pos, delta = _grain_points(case, seed)
        cap = _bond_capacity(len(pos), case["dim"])
        return dict(kind="bonds", pos=torch.from_numpy(pos).cuda(), delta=delta, cap=cap,
                    pairs=torch.zeros((cap, 2), dtype=torch.int32, device="cuda"))
    if case["kind"] == "pack":
        m = _mesh(case, seed)
        dev = [torch.from_numpy(m.pos).cuda()]
        dev += [torch.from_numpy(np.ascontiguousarray(a, np.int64).astype(np.uint32).view(np.int32)).cuda()
                for a in (m.T, m.bdry_nodes, m.bdry_edges)]
        return dict(kind="pack", dev=dev, modify=case["modify"], elems=len(m.T))
    sim = _sim(case, seed)
    sim.set_bond_alive(_intact(case, seed))
    sim.step(1)
    sim.synchronize()
    return dict(kind="post", sim=sim)


def run(state):
    if state["kind"] == "run":
        state["sim"].step(state["steps"])
        return state["sim"].snapshot(state["items"], out=state["out"]).wait()
    if state["kind"] == "grad":
        r = state["run"]
        reaction, ke = r.forward()
        g = r.backward(reaction_bar=state["rbar"], ke_bar=state["kbar"])
        return dict(reaction=reaction, ke=ke, grad=g)
    if state["kind"] == "bonds":
        pos, pairs = state["pos"], state["pairs"]
        count = C.c_uint64()
        N.check(N.lib().pg_build_bonds(C.c_void_p(pos.data_ptr()), pos.shape[0], pos.shape[1], state["delta"],
                                       C.c_void_p(pairs.data_ptr()), state["cap"], C.byref(count), None))
        return dict(pairs=pairs, count=count.value)
    if state["kind"] == "pack":
        d_pos, d_T, d_bn, d_be = state["dev"]
        cen, rad, unpolished = packing.pack_device(d_pos, d_T, d_bn, d_be, modify_nodal_circles=state["modify"])
        n = state["elems"]
        return dict(elem_centers=cen[:n], elem_radii=rad[:n], node_centers=cen[n:], node_radii=rad[n:],
                    unpolished=unpolished)
    return state["sim"].postprocess(node_damage=True)


def work(case):
    """Bytes and operations of one pass. A step reads and writes each node's state once and reads
    each directed bond's neighbour and intact bit (FP64 also its reference length); about 40
    operations per bond in 2D, 55 in 3D."""
    if case["kind"] in ("run", "grad"):
        s = _base(case)[0]
        d, mixed = s.dim, case["precision"] == "mixed"
        node = 56 * d + 4 if mixed else 72 * d + 16
        step = s.n_nodes * node + s.n_bonds * (4.125 if mixed else 12.125)
        flops = s.n_bonds * (40 if d == 2 else 55)
        n = case["steps"] * (3 if case["kind"] == "grad" else 1)  # forward, recomputation, reverse
        return dict(bytes=step * n + s.n_nodes * d * 32, flops=flops * n)
    if case["kind"] == "bonds":
        n, d = case["nodes"], case["dim"]
        pairs = n * (13 if d == 2 else 52)
        return dict(bytes=n * d * 8 + pairs * 8, flops=pairs * 3 * d)
    if case["kind"] == "pack":
        nn, ne = (case["nx"] + 1) * (case["ny"] + 1), 2 * case["nx"] * case["ny"]
        # an ascent of about 66 iterations over 6 circles per node
        return dict(bytes=nn * 40 + ne * 36, flops=ne * 40 + (nn * 66 * 6 * 12 if case["modify"] else nn * 40))
    s = _base(case)[0]
    return dict(bytes=s.n_nodes * (s.dim * 32 + 20) + s.n_bonds / 8, flops=s.n_nodes * 20 + s.n_bonds)


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def _bond_ends(s):
    """Global node pairs (i, j) of the directed bonds, in the setup's order."""
    off = s.bond_offset.astype(np.int64)
    i = np.repeat(np.arange(s.n_nodes), np.diff(off))
    first = np.repeat(s.grain_node_offset[:-1].astype(np.int64), np.diff(s.grain_node_offset.astype(np.int64)))
    return i, s.bond_local.astype(np.int64) + first[i]


def _near(x, inst, r):
    """All ordered pairs (p, q), p != q, of nodes of one instance in adjacent cells of edge r."""
    n, d = x.shape
    c = torch.floor((x - x.amin(0)) / r).long() + 1
    size = c.amax(0) + 2
    stride = [1]
    for a in range(d - 1):
        stride.append(stride[-1] * int(size[a]))
    total = stride[-1] * int(size[d - 1])
    key = inst * total + sum(c[:, a] * stride[a] for a in range(d))
    key, order = torch.sort(key)
    own = torch.empty_like(key)
    own[order] = key
    got = []
    rows = [0] if d == 1 else [dy * stride[1] for dy in (-1, 0, 1)]
    if d == 3:
        rows = [a + dz * stride[2] for a in rows for dz in (-1, 0, 1)]
    for o in rows:  # three cells along x are consecutive
        b = torch.searchsorted(key, own + o - 1)
        e = torch.searchsorted(key, own + o + 1, right=True)
        cnt = e - b
        p = torch.repeat_interleave(torch.arange(n, device=x.device), cnt)
        k = torch.arange(len(p), device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
        q = order[b[p] + k]
        got.append(torch.stack([p, q])[:, p != q])
    return torch.cat(got, 1)


class _Exact:
    """The reference's time step (positions, bonds with breaking, contact with damping and
    friction, walls, external force, velocities) in torch float64."""

    def __init__(self, s, dt, bdry_only=False, alive=None):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        self.s, self.dt, self.d, n, d = s, dt, s.dim, s.n_nodes, s.dim
        v = lambda a: t(np.asarray(a, np.float64).reshape(n, d))
        self.pos, self.disp, self.vel, self.acc, self.ext = map(v, (s.pos, s.disp, s.vel, s.acc, s.extforce))
        self.grain = t(np.repeat(np.arange(s.n_grains), np.diff(s.grain_node_offset.astype(np.int64))))
        self.ginst = t(s.grain_instance.astype(np.int64))
        self.inst = self.ginst[self.grain]
        self.vol, self.rho, self.cnot, self.snot = t(s.vol), t(s.rho), t(s.cnot), t(s.snot)
        self.rc, self.kn = t(s.contact_radius), t(s.normal_stiffness)
        self.mu, self.zeta = t(s.friction_coefficient), t(s.damping_ratio)
        self.wall = t(s.wall_geom.reshape(-1, 2 * d).copy())
        self.wall_speed = t(s.wall_speed.reshape(-1, 2 * d))
        self.has_wall = t(s.allow_wall.astype(bool))
        deg = np.diff(s.bond_offset.astype(np.int64))
        self.bi, self.bj = _bond_ends(s)
        self.slot = np.arange(len(self.bi)) - np.repeat(s.bond_offset[:-1].astype(np.int64), deg)
        K = max(1, int(deg.max()) if len(deg) else 1)
        nb, ok = np.zeros((K, n), np.int64), np.zeros((K, n), bool)
        nb[self.slot, self.bi] = self.bj
        ok[self.slot, self.bi] = True if alive is None else alive.astype(bool)
        self.nb, self.alive = t(nb), t(ok)
        xi = self.pos[self.nb] - self.pos
        self.xi_norm = torch.where(self.alive, self._norm(xi), 1.0)
        bdry = np.zeros(n, bool)
        for g in range(s.n_grains):
            bdry[int(s.grain_node_offset[g]) + s.bdry_nodes[s.bdry_offset[g]:s.bdry_offset[g + 1]].astype(np.int64)] = True
        self.bdry = t(bdry) if bdry_only else torch.ones(n, dtype=torch.bool, device=dev)
        self.cand, self.at = None, None
        self.force = torch.zeros_like(self.pos)
        self.cur = self.pos + self.disp

    @staticmethod
    def _norm(v):
        s = v[..., 0] * v[..., 0]
        for c in range(1, v.shape[-1]):
            s = s + v[..., c] * v[..., c]
        return torch.sqrt(s)

    def _bonds(self):
        f = torch.zeros_like(self.pos)
        cnot, snot = self.cnot[self.grain], self.snot[self.grain]
        for k in range(len(self.nb)):
            j, use = self.nb[k], self.alive[k]
            e = (self.disp[j] - self.disp) + (self.pos[j] - self.pos)
            en = self._norm(e)
            st = (en - self.xi_norm[k]) / self.xi_norm[k]
            add = ((cnot * st) * self.vol[j])[:, None] * (e / en[:, None])
            f += torch.where(use[:, None], add, torch.zeros((), dtype=f.dtype, device=f.device))
            self.alive[k] = use & ~(st > snot)
        return f

    def _candidates(self):
        r = float(self.rc.max())
        if self.cand is None or float((self.cur - self.at).abs().max()) > 0.2 * r:
            self.at = self.cur.clone()
            p, q = _near(self.cur, self.inst, 2.0 * r)
            keep = self.bdry[p] & self.bdry[q] & (self._norm(self.cur[p] - self.cur[q]) < 1.9 * r)
            self.cand = torch.stack([p[keep], q[keep]])
        return self.cand

    def _contact(self, f):
        p, q = self._candidates()
        near = self._norm(self.cur[q] - self.cur[p]) <= self.rc[self.inst[p]]
        p, q = p[near], q[near]
        same = self.grain[p] == self.grain[q]
        bonded = ((self.nb[:, p] == q) & self.alive[:, p]).any(0) & same
        p, q, same = p[~bonded], q[~bonded], same[~bonded]
        if not len(p):
            return f
        gi, g = self.inst[p], self.grain[p]
        rc = self.rc[gi]
        rc = torch.where(same, torch.minimum(self._norm(self.pos[p] - self.pos[q]), rc), rc)
        kn = torch.where(same, self.cnot[g] / rc, self.kn[gi])
        y = self.cur[q] - self.cur[p]
        dn = self._norm(y)
        hit = dn <= rc
        p, q, gi, g, rc, kn, y, dn = (a[hit] for a in (p, q, gi, g, rc, kn, y, dn))
        u, rho, vq = y / dn[:, None], self.rho[g], self.vol[q]
        s1 = -kn * (rc - dn) * vq
        out = s1[:, None] * u
        rv = self.vel[p] - self.vel[q]
        ru = (rv * u).sum(1)
        out = out - (2 * self.zeta[gi] * torch.sqrt(kn * rho) * torch.sqrt(vq) * ru)[:, None] * u
        tg = rv - ru[:, None] * u
        tn, mu = self._norm(tg), self.mu[gi]
        fr = torch.where(tn < mu * s1.abs() * self.dt / rho, -tn / rho / self.dt, -mu * s1.abs())
        out = out + torch.where(tn > 0, fr / tn.clamp_min(1e-300), 0.0)[:, None] * tg
        return f.index_add(0, p, out)

    def _walls(self, f):
        d, I = self.d, len(self.rc)
        self.reaction = torch.zeros((I, 2 * d, d), dtype=f.dtype, device=f.device)
        for side in range(2 * d):
            ax = (0 if side < 2 else 1) if d == 2 else side % 3
            on = self.has_wall[self.inst] & self.bdry
            dist = self.cur[:, ax] - self.wall[self.inst, side]
            p = torch.nonzero(on & (dist.abs() <= self.rc[self.inst]))[:, 0]
            if not len(p):
                continue
            gi, rho = self.inst[p], self.rho[self.grain[p]]
            r, dd, sign = self.rc[gi], dist[p].abs(), torch.where(dist[p] > 0, 1.0, -1.0).to(f.dtype)
            if d == 2:
                area = math.pi * r * r / 2 - r * r * torch.asin(dd / r) - torch.sqrt(r * r - dd * dd) * dd
                cen = torch.zeros_like(area)
            else:
                area = math.pi / 3 * (r - dd) ** 2 * (2 * r - dd)
                cen = math.pi / 4 * (r * r - dd * dd) ** 2 / area
            F = self.kn[gi] * (r - cen).clamp_min(0) * area
            w = torch.zeros((len(p), d), dtype=f.dtype, device=f.device)
            w[:, ax] += sign * F
            rv = self.vel[p].clone()
            rv[:, ax] -= self.wall_speed[gi, side]
            mu = self.mu[gi]
            tan = [a for a in range(d) if a != ax]
            vn = self._norm(rv[:, tan])
            stick = -vn * rho / self.dt if d == 2 else -vn / rho / self.dt
            fr = torch.where(vn < mu * F.abs() * self.dt / rho, stick, -mu * F.abs())
            for a in tan:
                w[:, a] += torch.where(vn > 0, fr * rv[:, a] / vn.clamp_min(1e-300), 0.0)
            w[:, ax] -= 2 * self.zeta[gi] * torch.sqrt(self.kn[gi] * rho) * torch.sqrt(area.abs()) * rv[:, ax]
            f = f.index_add(0, p, w)
            self.reaction[:, side].index_add_(0, gi, -self.vol[p][:, None] * w)
        return f

    def step(self):
        dt = self.dt
        self.disp = self.disp + ((dt * self.vel) + (dt * dt * 0.5) * self.acc)
        self.cur = self.pos + self.disp
        f = self._walls(self._contact(self._bonds())) + self.ext
        acc = (1 / self.rho)[self.grain][:, None] * f
        self.vel = self.vel + 0.5 * dt * (self.acc + acc)
        self.acc, self.force = acc, f
        self.wall = self.wall + self.wall_speed * dt

    def go(self, n):
        for _ in range(n):
            self.step()
        return self

    def intact(self):
        a = self.alive.cpu().numpy()
        return a[self.slot, self.bi].astype(np.uint8)


def _exact_post(case, seed):
    s = _setup(case, seed)
    e = _Exact(s, _dt("ensemble"), alive=_intact(case, seed)).go(1)
    G, I, d, n = s.n_grains, s.n_instances, s.dim, s.n_nodes
    per = torch.bincount(e.grain, minlength=G).to(e.vol.dtype)

    def total(a, of, k):
        return torch.zeros((k,) + a.shape[1:], dtype=a.dtype, device=a.device).index_add(0, of, a)

    deg0 = torch.from_numpy(np.diff(s.bond_offset.astype(np.int64))).to(e.vol)
    damage = (deg0 - e.alive.sum(0)) / deg0
    w = e.wall
    out = dict(grain_mean_vel=total(e.vel, e.grain, G) / per[:, None], grain_mean_acc=total(e.acc, e.grain, G) / per[:, None],
               grain_mean_currpos=total(e.cur, e.grain, G) / per[:, None], grain_force=total(e.force, e.grain, G),
               grain_damage=total(damage, e.grain, G) / per,
               inertial_force=total((e.vol * e.rho[e.grain])[:, None] * e.acc, e.inst, I),
               volume_fraction=total(e.vol, e.inst, I) / ((w[:, 1] - w[:, 0]) * (w[:, 2] - w[:, 3])), node_damage=damage)
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_pack(case, seed):
    m = _mesh(case, seed)
    a, b, c = (m.pos[m.T[:, k]] for k in range(3))
    la, lb, lc = (np.sqrt(((p - q) ** 2).sum(1)) for p, q in ((c, b), (c, a), (b, a)))
    sl = la + lb + lc
    cen = (la[:, None] * a + lb[:, None] * b + lc[:, None] * c) / sl[:, None]
    rad = 2 * (0.25 * np.sqrt(sl * (la - lb + lc) * (lb - lc + la) * (lc - la + lb))) / sl
    return dict(elem_centers=cen, elem_radii=rad, node_centers=None, node_radii=None, unpolished=None)


def exact(case, seed):
    if case["kind"] == "bonds":
        return None  # whole numbers
    if case["kind"] == "pack":
        return _exact_pack(case, seed)
    if case["kind"] == "post":
        return _exact_post(case, seed)
    s = _setup(case, seed)
    if s.n_bonds * case["steps"] > 1.2e9:
        return None  # over about 20 seconds
    e = _Exact(s, _dt(_base(case)[1]), case.get("bdry_only", False)).go(case["steps"])
    if case["kind"] == "grad":
        mass = (e.rho[e.grain] * e.vol * (e.vel * e.vel).sum(1) * 0.5)
        ke = torch.zeros(len(e.rc), dtype=mass.dtype, device=mass.device).index_add(0, e.inst, mass)
        return dict(reaction=e.reaction.cpu().numpy(), ke=ke.cpu().numpy(), grad=None)
    out = dict(CurrPos=e.cur, vel=e.vel, acc=e.acc, force=e.force, bond_alive=None)
    if s.allow_wall.any():
        out.update(wall=e.wall, reaction=e.reaction)
    out = {k: (None if v is None else v.cpu().numpy()) for k, v in out.items()}
    return dict(out, too_close_events=None, last_step=None)
