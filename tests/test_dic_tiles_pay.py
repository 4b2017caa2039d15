"""TFS_OPT_DIC_TILES = 2 (the default): tiles where they are the faster way, by
the system's size and the iterations a solve is expected to take -- its limit, or
what the last one took to its tolerance --, with the level kernels' or the
one-block kernel's bits either way."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import system
from tflows import TFS_CG, TFS_FP64, TFS_MIXED, Matrix_Type, Solver
from tflows.lib import TFS_OPT_DIC_TILES
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu


def _solve(sol, s, limit, rel=1e-30):
    x, r = np.zeros(s.n), s.b.copy()
    res = sol.solve(TFS_CG, s.val, x, r, 2, limit, rel * float(np.linalg.norm(s.b)))
    return [x, r, np.array([res.niter, res.ini_res, res.fin_res])], sol.stats()["dic_tiles"]


# (shape, arithmetic, iterations expected -> tiles?), both sides of every line:
# the one-block DIC's rows, one iteration from 2^17 rows, fewer than four from
# 1.65 M, than eight with two tiles a multiprocessor (from 2.19 M)
LINES = [((14, 15, 14), TFS_MIXED, {1: 0, 40: 0}), ((15, 15, 14), TFS_MIXED, {1: 1, 40: 1}),
         ((10, 9, 9), TFS_FP64, {1: 0, 40: 0}), ((10, 10, 9), TFS_FP64, {1: 1, 40: 1}),
         ((51, 51, 50), TFS_FP64, {1: 1, 2: 1}), ((51, 51, 51), TFS_FP64, {1: 0, 2: 1}),
         ((119, 119, 117), TFS_MIXED, {3: 0, 4: 1}), ((131, 131, 130), TFS_MIXED, {7: 0, 8: 1}),
         ((131, 131, 130), TFS_FP64, {7: 0, 8: 1}),
         # one tile a multiprocessor by its rows, but in binary64 they do not fit: two
         ((129, 129, 129), TFS_FP64, {3: 0, 4: 1})]


@pytest.mark.parametrize("shape,mode,asked", LINES)
def test_lines(shape, mode, asked, gpu):
    s = system(POISSON, *shape)
    want = {}
    with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 0}) as sol:
        for limit in asked:
            want[limit], none = _solve(sol, s, limit)
            assert none == 0
    with Solver(s.matrix(), precision=mode) as sol:
        assert sol.get_option(TFS_OPT_DIC_TILES) == 2
        for limit in sorted(asked) + sorted(asked, reverse=True):
            got, tiles = _solve(sol, s, limit)
            assert (tiles > 0) == bool(asked[limit]), (limit, tiles)
            assert all(np.array_equal(a, b) for a, b in zip(got, want[limit], strict=True))
    with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 1}) as sol:
        for limit in asked:
            got, tiles = _solve(sol, s, limit)
            assert tiles > 0
            assert all(np.array_equal(a, b) for a, b in zip(got, want[limit], strict=True))


def test_short_solves_are_expected_to_be_short_again(gpu):
    s = system(POISSON, 51, 51, 51)                     # tiles from two iterations on
    with Solver(s.matrix()) as sol:
        first, tiles = _solve(sol, s, 500, 0.99)        # nothing known: its limit
        assert tiles > 0
        it = sol.stats()["iterations"]
        for _ in range(2):
            again, tiles = _solve(sol, s, 500, 0.99)
            assert (tiles > 0) == (it >= 2)
            assert all(np.array_equal(a, b) for a, b in zip(first, again, strict=True))
        _solve(sol, s, 500, 1e-6)                       # a long one
        again, tiles = _solve(sol, s, 500, 0.99)
        assert tiles > 0 and all(np.array_equal(a, b) for a, b in zip(first, again, strict=True))
        _solve(sol, s, 3)                               # ended by its limit: says nothing of the next
        assert _solve(sol, s, 500, 0.99)[1] > 0


@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
@pytest.mark.parametrize("n,tiles", [(12, 0), (15, 1)])     # 1,728 and 3,375 rows
def test_rows_of_more_than_eight_entries(n, tiles, mode, gpu):
    """A randomly numbered mesh with two diagonal neighbour pairs besides the six
    faces (rows of up to eleven entries): one block below 3,072 rows in both
    arithmetics, tiles above, with the level kernels' bits."""
    num = np.random.default_rng(n).permutation(n ** 3).reshape(n, n, n)
    rows, cols = [np.arange(n ** 3)], [np.arange(n ** 3)]
    for dx, dy, dz in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (0, 1, 1)):
        a, b = num[: n - dx, : n - dy, : n - dz].ravel(), num[dx:, dy:, dz:].ravel()
        rows += [a, b]
        cols += [b, a]
    i, j = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((j, i))
    i, j = i[order], j[order]
    deg = np.bincount(i, minlength=n ** 3)
    val = np.where(i == j, deg[i] - 1 + 0.01, -1.0)
    row = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    A = Matrix_Type(n ** 3, row, (j + 1).astype(np.int32), (np.flatnonzero(i == j) + 1).astype(np.int32), val)
    b = np.random.default_rng(1).uniform(-1, 1, n ** 3)
    got = []
    for option in (0, 1, 2):
        with Solver(A, precision=mode, options={TFS_OPT_DIC_TILES: option}) as sol:
            x, r = np.zeros(n ** 3), b.copy()
            res = sol.solve(TFS_CG, val, x, r, 2, 30, 1e-10)
            used = sol.stats()["dic_tiles"]
            assert (used > 0) == (option == 1 or (option == 2 and bool(tiles))), (option, used)
            got.append((x, r, np.array([res.niter, res.ini_res, res.fin_res])))
    for other in got[1:]:
        assert all(np.array_equal(p, q) for p, q in zip(got[0], other, strict=True))
