"""A tile plan of the DIC sweeps that cannot be had -- no memory on the host, a
thread that the system does not start, no device memory -- leaves the level
kernels, which need none of it: the solve gives what it gives without tiles,
and what the plan had taken is given back."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import system
from tflows import TFS_CG, TFS_FP64, TFS_MIXED, Solver
from tflows.lib import TFS_ERR_ARG, TFS_OPT_DIC_TILES, last_error, load_library
from tflows.synth import POISSON

REPO = Path(__file__).resolve().parents[1]


def test_plan_without_threads_or_memory(tmp_path):
    exe = tmp_path / "tile_plan_failures_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-pthread", "-I", str(REPO / "t-flows_gb300" / "csrc"),
                    str(REPO / "tests" / "native" / "tile_plan_failures_check.cpp"), "-o", str(exe), "-ldl"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_diag_alloc_failure_rejects_without_a_device():
    lib = load_library()
    assert lib.tfs_diag_alloc_failure(None, 1) == TFS_ERR_ARG
    assert "tfs_diag_alloc_failure" in last_error()


def _solve(sol, s):
    x, r = np.zeros(s.n), s.b.copy()
    res = sol.solve(TFS_CG, s.val, x, r, 2, 60, 1e-10 * float(np.linalg.norm(s.b)))
    return x, r, np.array([res.niter, res.status])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
def test_solves_without_device_memory_for_the_plan(mode, gpu):
    lib = load_library()
    s = system(POISSON, 24, 23, 22)
    with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 0}) as sol:
        want = _solve(sol, s)
        plain_bytes = sol.stats()["device_bytes"]
    for nth in (1, 2, 5, 9, 14, 18, 0):     # the plan has nine arrays a direction
        with Solver(s.matrix(), precision=mode) as sol:
            sol.levels()                    # the layout's own allocations
            assert lib.tfs_diag_alloc_failure(sol.h, nth) == 0
            for _ in range(2):
                for a, c in zip(_solve(sol, s), want, strict=True):
                    assert np.array_equal(a, c)
                st = sol.stats()
                assert (st["dic_tiles"] > 0) == (nth == 0)
                assert (st["device_bytes"] > plain_bytes) == (nth == 0)
            assert lib.tfs_diag_alloc_failure(sol.h, 0) == 0
