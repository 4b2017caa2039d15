"""Tiled DIC sweeps that have nothing to do: a solve that ends inside a loop
body leaves that body's other sweeps idle.

CPU: the walk of the lane that copies a tile's rounds leaves nothing in flight,
whenever the sweep is called off.  GPU: solves that end at every place of a
body, back to back and from several threads, bitwise equal to the level
kernels', on systems of one tile whose rounds all fit its ring (the lane has
issued them before it can know that there is nothing to sweep), of a few tiles
and of many."""
from __future__ import annotations

import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import pytest

from helpers import system
from tflows import TFS_CG, TFS_CGS, TFS_FP64, TFS_MIXED, Solver
from tflows.lib import TFS_OPT_DIC_TILES
from tflows.synth import CONVDIFF, POISSON

REPO = Path(__file__).resolve().parents[1]


def test_copy_walk_leaves_nothing_in_flight(tmp_path):
    exe = tmp_path / "tile_copy_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", str(REPO / "t-flows_gb300" / "csrc"),
                    str(REPO / "tests" / "native" / "tile_copy_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def _solve(sol, s, method, limit):
    x, r = np.zeros(s.n), s.b.copy()
    res = sol.solve(method, s.val, x, r, 2, limit, 1e-12 * float(np.linalg.norm(s.b)))
    return x, r, np.array([res.niter, res.status]), np.array([res.ini_res, res.fin_res])


@pytest.mark.gpu
@pytest.mark.parametrize("kind,shape", [(POISSON, (12, 11, 10)), (CONVDIFF, (20, 20, 20)), (POISSON, (40, 40, 40)),
                                        (POISSON, (64, 64, 64))])
@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
def test_solves_that_end_inside_a_body(kind, shape, mode, gpu):
    s = system(kind, *shape)
    method = TFS_CG if kind == POISSON else TFS_CGS
    limits = [1, 2, 3, 5, 13, 14, 15, 16, 17]     # singly, then in bodies of four
    with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 0}) as sol:
        want = [_solve(sol, s, method, n) for n in limits]

    def run(_):
        out = []
        with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 1}) as sol:
            for _ in range(4):
                out.append([_solve(sol, s, method, n) for n in limits])
            assert sol.stats()["dic_tiles"] > 0
        return out

    with ThreadPoolExecutor(3) as pool:
        for got in pool.map(run, range(3)):
            for series in got:
                for a, c in zip(series, want, strict=True):
                    assert all(np.array_equal(u, v) for u, v in zip(a, c, strict=True))
