"""The bond builder where its passes can go wrong: rows longer than the shared-memory list, the row
that crosses the buffer's capacity, scan tiles, lengths at exactly delta (FP64 decides), scales at
which no fixed-point test is made, degenerate boxes and horizons. The oracle is the rule of the
reference (exp_dict.py:171-222) over all pairs in numpy; whole numbers, so equality."""
import ctypes as C

import numpy as np
import pytest

from perigrain_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _oracle(p, delta):
    i, j = np.triu_indices(len(p), 1)
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        s = np.zeros(len(i))
        for c in range(p.shape[1]):
            s = s + (p[j, c] - p[i, c]) * (p[j, c] - p[i, c])
        keep = np.sqrt(s) <= delta
    return np.stack([i[keep], j[keep]], 1)


def _call(p, delta, capacity, entry="pg_build_bonds"):
    import torch

    d_pos = torch.from_numpy(np.ascontiguousarray(p, np.float64)).cuda()
    d_pairs = torch.full((capacity + 8, 2), -7, dtype=torch.int32, device="cuda")
    m = C.c_uint64()
    rc = getattr(N.lib(), entry)(C.c_void_p(d_pos.data_ptr()), len(p), p.shape[1], float(delta),
                                 C.c_void_p(d_pairs.data_ptr()), capacity, C.byref(m), None)
    out = d_pairs.cpu().numpy()
    assert (out[min(m.value, capacity):] == -7).all()  # nothing written past the rows
    return rc, m.value, out[:min(m.value, capacity)]


def _grid(dim, k, h=1.0, at=0.0):
    return np.stack([a.ravel() for a in np.meshgrid(*[np.arange(k)] * dim, indexing="ij")], 1) * h + at


CASES = {
    "two": (np.array([[0.0, 0.0], [1.0, 0.0]]), 1.0),
    "same point": (np.zeros((70, 2)), 0.0),
    "same point 3d": (np.zeros((70, 3)), 1.0),
    "a line": (np.stack([np.arange(900.0), np.zeros(900)], 1), 3.0),
    "a line on y": (np.stack([np.zeros(900), np.arange(900.0)], 1), 3.0),
    "lattice": (_grid(2, 40, 1e-4, 0.3), 3e-4),
    "lattice 3d": (_grid(3, 11, 1e-4, -0.3), 2e-4),
    "long rows": (np.random.default_rng(1).random((1500, 2)), 0.4),
    "long rows 3d": (np.random.default_rng(2).random((2300, 3)), 0.9),
    "scan tile - 1": (np.random.default_rng(3).random((4095, 2)), 0.02),
    "scan tile": (np.random.default_rng(4).random((4096, 2)), 0.02),
    "scan tile + 1": (np.random.default_rng(5).random((4097, 3)), 0.07),
    "far apart": (np.concatenate([np.random.default_rng(6).random((300, 2)), 1e6 + np.random.default_rng(7).random((300, 2))]), 0.1),
    "tiny scale": (_grid(2, 20, 1e-150), 3e-150),
    "large scale": (_grid(2, 20, 1e150), 3e150),
    "horizon 0": (np.random.default_rng(8).random((300, 2)), 0.0),
    "horizon below 0": (np.random.default_rng(8).random((300, 2)), -1.0),
    "horizon least": (np.zeros((40, 2)), 5e-324),
    "horizon inf": (np.random.default_rng(9).random((90, 3)), np.inf),
    "horizon nan": (np.random.default_rng(9).random((90, 2)), np.nan),
}


@pytest.mark.parametrize("name", CASES)
def test_rows(name):
    p, delta = CASES[name]
    ref = _oracle(p, delta)
    rc, m, got = _call(p, delta, len(ref) + 3)
    assert rc == N.PG_OK and m == len(ref) and np.array_equal(got, ref)
    rc, m, got = _call(p, delta, len(ref) + 3, "pg_build_bonds_noalloc")
    assert rc == N.PG_OK and m == len(ref) and np.array_equal(got, ref)


@pytest.mark.parametrize("name", ["lattice", "lattice 3d", "long rows", "long rows 3d"])
def test_row_that_crosses_the_capacity(name):
    p, delta = CASES[name]
    ref = _oracle(p, delta)
    for cap in (1, len(ref) // 2, len(ref) - 1):
        rc, m, got = _call(p, delta, cap)
        assert rc == N.PG_ECAPACITY and m == len(ref) and np.array_equal(got, ref[:cap])


@pytest.mark.parametrize("bad", [np.nan, -np.nan, np.inf, -np.inf])
def test_non_finite_position(bad):
    p = np.random.default_rng(10).random((200, 2))
    p[77, 1] = bad
    rc, m, _ = _call(p, 0.1, 100)
    assert rc == N.PG_EINVAL and m == 0 and b"non-finite" in N.lib().pg_bond_last_error()


def test_too_many_partners_and_too_many_cells():
    rc, m, _ = _call(np.zeros((4200, 2)), 1.0, 16)
    assert rc == N.PG_ECAPACITY and m == 4200 * 4199 // 2 and b"4096 partners" in N.lib().pg_bond_last_error()
    rc, m, _ = _call(np.random.default_rng(11).random((200, 3)), 1e-60, 16)
    assert rc == N.PG_ECAPACITY and m == 0 and b"grid" in N.lib().pg_bond_last_error()


def test_builds_side_by_side():
    """Calls of several threads, each on its own stream: one holds the kept scratch at a time, the
    others bring their own; every one gives its grain's rows."""
    import threading

    import torch

    grains = [(np.random.default_rng(20 + k).random((3000 + 500 * k, 2 + k % 2)), 0.05 + 0.05 * (k % 2)) for k in range(4)]
    refs = [_oracle(p, d) for p, d in grains]
    wrong = []

    def work(k):
        p, delta = grains[k]
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            d_pos = torch.from_numpy(p).cuda()
            d_pairs = torch.empty((len(refs[k]), 2), dtype=torch.int32, device="cuda")
            for _ in range(20):
                d_pairs.fill_(-7)
                m = C.c_uint64()
                rc = N.lib().pg_build_bonds(C.c_void_p(d_pos.data_ptr()), len(p), p.shape[1], delta,
                                            C.c_void_p(d_pairs.data_ptr()), len(refs[k]), C.byref(m),
                                            C.c_void_p(stream.cuda_stream))
                if rc != N.PG_OK or m.value != len(refs[k]) or not np.array_equal(d_pairs.cpu().numpy(), refs[k]):
                    wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
