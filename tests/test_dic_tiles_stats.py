"""dic_tiles and dic_kernel describe the last solve's DIC applications, also
when its graph was captured before those of other solves."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import system
from tflows import TFS_BICG, TFS_CG, TFS_FP64, TFS_MIXED, Solver
from tflows.lib import TFS_OPT_BICG
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu


def _solve(sol, s, method, prec):
    x, r = np.zeros(s.n), s.b.copy()
    sol.solve(method, s.val, x, r, prec, 20, 1e-10 * float(np.linalg.norm(s.b)))
    st = sol.stats()
    return x, st["dic_tiles"], st["dic_kernel"]


def test_statistics_of_the_graph_that_ran(gpu):
    s = system(POISSON, 24, 23, 22)
    with Solver(s.matrix(), options={TFS_OPT_BICG: 1}) as sol:
        x, tiles, kernel = _solve(sol, s, TFS_CG, 2)
        assert tiles > 0 and kernel == 0
        assert _solve(sol, s, TFS_BICG, 2)[1:] == (0, 0)       # two vectors a sweep: by levels
        again = _solve(sol, s, TFS_CG, 2)
        assert again[1:] == (tiles, 0) and np.array_equal(again[0], x)
        _solve(sol, s, TFS_CG, 1)
        sol.profile_prec(s.val)                                # stamps the level launches
        again = _solve(sol, s, TFS_CG, 2)
        assert again[1:] == (tiles, 0) and np.array_equal(again[0], x)
        sol.set_precision(TFS_MIXED)
        assert _solve(sol, s, TFS_CG, 2)[1] > 0
        sol.set_precision(TFS_FP64)
        _solve(sol, s, TFS_CG, 1)
        assert _solve(sol, s, TFS_CG, 2)[1:] == (tiles, 0)
