"""Tile plans in the request server: made beside the requests, from room that no
system needs, given up before a system is evicted; results are those of the
level kernels throughout."""
from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest

from helpers import system
from tflows import TFS_CG, TFS_FP64, TFS_MIXED, Server, Solver
from tflows.lib import TFS_OPT_DIC_TILES, check, load_library
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu


def est(s):   # tfs_estimate_bytes
    n_pad = (s.n + 1023) // 1024 * 1024 + 32 * 64
    return n_pad * 200 + s.n * 20 + s.nnz * 29 + (64 << 10)


class Arrays:
    def __init__(self, s):
        self.lib, self.s, self.p = load_library(), s, {}
        for name, a in (("val", s.val), ("b", s.b), ("x", np.zeros(s.n)), ("r", np.zeros(s.n))):
            q = C.c_void_p()
            check(self.lib.tfs_device_alloc(a.nbytes, C.byref(q)), "alloc")
            self.p[name] = q.value
            check(self.lib.tfs_memcpy(C.c_void_p(q.value), a.ctypes.data_as(C.c_void_p), a.nbytes), "copy")

    def get(self, name):
        a = np.empty(self.s.n)
        check(self.lib.tfs_memcpy(a.ctypes.data_as(C.c_void_p), C.c_void_p(self.p[name]), a.nbytes), "copy")
        return a

    def free(self):
        for q in self.p.values():
            self.lib.tfs_device_free(C.c_void_p(q))


def want(s, mode, limit):
    with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 0}) as sol:
        x, r = np.zeros(s.n), s.b.copy()
        res = sol.solve(TFS_CG, s.val, x, r, 2, limit, 1e-8 * float(np.linalg.norm(s.b)))
        return x, r, res.niter


def ask(srv, sid, a, mode, limit):
    return srv.submit(sid, TFS_CG, 2, a.p["val"], a.p["x"], a.p["r"], limit, 1e-8 * float(np.linalg.norm(a.s.b)), mode,
                      d_b=a.p["b"], x0_zero=True)


def until(cond, limit_s=30.0):
    t0 = time.perf_counter()
    while not cond():
        assert time.perf_counter() - t0 < limit_s
        time.sleep(0.002)


@pytest.fixture(scope="module")
def pool(gpu):
    out = [system(POISSON, nx, ny, nz, seed=sd) for nx, ny, nz, sd in
           ((24, 24, 24, 1), (26, 25, 24, 2), (28, 26, 25, 3), (40, 40, 38, 4))]
    yield out


@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
def test_a_budget_for_the_systems_alone_evicts_none(pool, mode):
    """Room for the three systems and a little, not for their plans."""
    systems = pool[:3]
    arrs = [Arrays(s) for s in systems]
    try:
        with Server(int(1.02 * sum(est(s) for s in systems)), max_inflight=4) as srv:
            ids = [srv.add_system(s.n, s.row, s.col, s.dia) for s in systems]
            for rounds in range(6):
                for sid, a in zip(ids, arrs):
                    assert srv.wait(ask(srv, sid, a, mode, 40))["status"] == 0
                time.sleep(0.05)
            st = srv.stats()
        assert st["evictions"] == 0 and st["registrations"] == 3, st
        for a in arrs:
            x, r, _ = want(a.s, mode, 40)
            assert np.array_equal(a.get("x"), x) and np.array_equal(a.get("r"), r)
    finally:
        for a in arrs:
            a.free()


@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
def test_plans_arrive_and_give_way(pool, mode):
    """Plans take spare room once they are made; a system added later gets it
    back from them, and nobody is evicted."""
    first, late = pool[:3], pool[3]
    arrs = [Arrays(s) for s in pool]
    expected = [want(s, mode, 40) for s in pool]

    def good(k):
        return np.array_equal(arrs[k].get("x"), expected[k][0]) and np.array_equal(arrs[k].get("r"), expected[k][1])

    try:
        budget = sum(est(s) for s in first) + int(1.05 * est(late))
        with Server(budget, max_inflight=4) as srv:
            ids = [srv.add_system(s.n, s.row, s.col, s.dia) for s in first]
            assert srv.wait(ask(srv, ids[0], arrs[0], mode, 40))["status"] == 0
            assert good(0)
            bare = srv.stats()["resident_bytes"]
            until(lambda: srv.stats()["resident_bytes"] > bare)         # the first system's plan
            for k in range(3):
                for _ in range(3):
                    assert srv.wait(ask(srv, ids[k], arrs[k], mode, 40))["status"] == 0
                    assert good(k)
                    time.sleep(0.05)
            with_plans = srv.stats()["resident_bytes"]
            ids.append(srv.add_system(late.n, late.row, late.col, late.dia))
            tickets = [ask(srv, ids[k], arrs[k], mode, 40) for k in (3, 0, 1, 2)]
            for t in tickets:
                assert srv.wait(t)["status"] == 0
            time.sleep(0.2)
            st = srv.stats()
            assert all(good(k) for k in range(4))
        assert st["evictions"] == 0 and st["registrations"] == 4, st
        assert st["resident_bytes"] <= budget and with_plans > bare
    finally:
        for a in arrs:
            a.free()


def test_a_server_closed_while_it_plans(pool):
    a = Arrays(pool[3])
    try:
        for _ in range(3):
            with Server(1 << 34) as srv:
                sid = srv.add_system(a.s.n, a.s.row, a.s.col, a.s.dia)
                assert srv.wait(ask(srv, sid, a, TFS_MIXED, 30))["status"] == 0
    finally:
        a.free()
