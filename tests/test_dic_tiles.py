"""The tiled DIC sweeps (TFS_OPT_DIC_TILES).

CPU: the plan (partition, closures, packed rounds, list rounds) compiled on
the host, and the two-FMA form of the backward start values.  GPU: Prec_Solve
bitwise equal to the oracle, and whole DIC solves -- CG in both arithmetics,
CGS in binary64, the drop-in BiCG -- bitwise equal to the level kernels', on
systems of one tile and of many, with sizes at the edges of a round (512
rows), of the one-tile limit and of a tile per multiprocessor."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import system
from oracle import tfs_oracle as O
from tflows import TFS_BICG, TFS_CG, TFS_CGS, TFS_FP64, TFS_MIXED, Solver
from tflows.lib import TFS_ERR_TIMEOUT, TFS_OPT_DIC_TILES, TFS_OPT_FUSE_L0, TFS_OPT_LAUNCH, TfsError, load_library
from tflows.synth import CONVDIFF, POISSON

REPO = Path(__file__).resolve().parents[1]


def _native(tmp_path, name, *flags):
    exe = tmp_path / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-ffp-contract=off", *flags, "-I",
                    str(REPO / "t-flows_gb300" / "csrc"), str(REPO / "tests" / "native" / f"{name}.cpp"), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def test_plan_sweeps_bitwise_and_refuses_long_closures(tmp_path):
    _native(tmp_path, "dic_tiles_plan_check")


def test_quotient_of_a_rounded_product_is_the_division(tmp_path):
    _native(tmp_path, "tile_quotient_check")


# rows: one tile (8 .. 3071), two and more, a tile per multiprocessor
SHAPES = [(POISSON, (2, 2, 2)), (POISSON, (8, 8, 8)), (POISSON, (19, 9, 3)), (POISSON, (16, 16, 12)),
          (CONVDIFF, (13, 15, 16)), (POISSON, (40, 41, 39)), (CONVDIFF, (62, 62, 62))]


def _solves(s, tiles, **more):
    """Everything a DIC caller can see, with or without the tiles."""
    out, used = [], []
    tol = 1e-8 * float(np.linalg.norm(s.b))
    opts = {TFS_OPT_DIC_TILES: tiles, **more.get("options", {})}
    b = np.random.default_rng(4).uniform(-1, 1, s.n)
    for mode in (TFS_FP64, TFS_MIXED):
        with Solver(s.matrix(), precision=mode, options=opts) as sol:
            if mode == TFS_FP64:
                out.append(sol.prec_solve(s.val, 2, b))
                used.append(sol.stats()["dic_tiles"])
            methods = (TFS_CG, TFS_BICG) if s.kind == POISSON else (TFS_CGS,)
            for method in methods:
                x, r = np.zeros(s.n), s.b.copy()
                res = sol.solve(method, s.val, x, r, 2, 60, tol)
                used.append(sol.stats()["dic_tiles"])
                out += [x, r, np.array([res.niter, res.status]), np.array([res.ini_res, res.fin_res])]
    return out, used


@pytest.mark.gpu
@pytest.mark.parametrize("kind,shape", SHAPES)
def test_tiles_bitwise(kind, shape, gpu):
    s = system(kind, *shape)
    got, used = _solves(s, 1)
    want, none = _solves(s, 0)
    assert all(u > 0 for u in used) and not any(none), (used, none)
    assert np.array_equal(got[0], O.prec_solve(s.n, s.row, s.col, s.dia, s.val, 2,
                                               np.random.default_rng(4).uniform(-1, 1, s.n)))
    for a, c in zip(got, want):
        assert np.array_equal(a, c)


@pytest.mark.gpu
@pytest.mark.parametrize("options", [{TFS_OPT_FUSE_L0: 0}, {TFS_OPT_LAUNCH: 1}])
def test_tiles_bitwise_with_options(options, gpu):
    s = system(POISSON, 24, 23, 22)
    got, used = _solves(s, 1, options=options)
    want, none = _solves(s, 0, options=options)
    assert all(u > 0 for u in used) and not any(none)
    for a, c in zip(got, want):
        assert np.array_equal(a, c)


@pytest.mark.gpu
def test_structured_numbering_keeps_the_level_kernels(gpu):
    """Closures under a lexicographic numbering reach through the mesh: no
    tiles, and the solve is the level kernels'."""
    s = system(POISSON, 30, 28, 26, permute=False)
    got, used = _solves(s, 1)
    want, _ = _solves(s, 0)
    assert not any(used)
    for a, c in zip(got, want):
        assert np.array_equal(a, c)


@pytest.mark.gpu
def test_values_outside_the_quotients_range(gpu):
    """Diagonals and right-hand sides far from 1 take the division itself:
    Prec_Solve still equals the oracle."""
    s = system(POISSON, 9, 10, 11)
    for scale_a, scale_b in ((1e-200, 1.0), (1e180, 1.0), (1.0, 1e-300), (1.0, 1e290), (1e-30, 0.0)):
        val = s.val * scale_a
        b = np.random.default_rng(5).uniform(-1, 1, s.n) * scale_b
        with Solver(s.matrix()) as sol:
            z = sol.prec_solve(val, 2, b)
            assert sol.stats()["dic_tiles"] > 0
        with np.errstate(all="ignore"):
            assert np.array_equal(z, O.prec_solve(s.n, s.row, s.col, s.dia, val, 2, b), equal_nan=True)


@pytest.mark.gpu
def test_tile_wait_runs_out(gpu):
    """With nothing staged and a 2 ms limit the tiles' waits run out: the
    solve returns TFS_ERR_TIMEOUT, and the same handle then solves as before."""
    lib = load_library()
    s = system(POISSON, 24, 24, 24)
    tol = 1e-8 * float(np.linalg.norm(s.b))
    with Solver(s.matrix()) as sol:
        x, r = np.zeros(s.n), s.b.copy()
        good = sol.solve(TFS_CG, s.val, x, r, 2, 500, tol)
        assert good.status == 0 and sol.stats()["dic_tiles"] > 0
        assert lib.tfs_diag_dic_timeout(sol.h, 2_000_000) == 0
        with pytest.raises(TfsError) as e:
            sol.solve(TFS_CG, s.val, np.zeros(s.n), s.b.copy(), 2, 500, tol)
        assert e.value.status == TFS_ERR_TIMEOUT
        assert lib.tfs_diag_dic_timeout(sol.h, 0) == 0
        x2, r2 = np.zeros(s.n), s.b.copy()
        again = sol.solve(TFS_CG, s.val, x2, r2, 2, 500, tol)
        assert again.status == 0 and np.array_equal(x2, x) and np.array_equal(r2, r)
