"""Loop bodies of one iteration or of four, whichever the solve is expected to
fill: whatever came before on the handle, every solve gives the bits of the same
solve launched kernel by kernel on a handle of its own."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import system
from tflows import TFS_BICG, TFS_CG, TFS_CGS, TFS_FP64, TFS_MIXED, Solver
from tflows.lib import TFS_OPT_BICG, TFS_OPT_DIC_TILES, TFS_OPT_LAUNCH
from tflows.synth import CONVDIFF, POISSON

pytestmark = pytest.mark.gpu

# (limit, relative tolerance): long and short in turn, ended by either
SERIES = [(40, 1e-30), (1, 1e-30), (2, 1e-30), (3000, 0.5), (3000, 1e-6), (13, 1e-30), (11, 1e-30), (3000, 0.2),
          (0, 1e-6), (3000, 1e-3), (5, 1e-30), (3000, 2.0), (3000, 1e-2), (12, 1e-30), (3, 1e-30), (3000, 1e-4)]


def _solve(sol, s, method, prec, limit, rel):
    x, r = np.zeros(s.n), s.b.copy()
    res = sol.solve(method, s.val, x, r, prec, limit, rel * float(np.linalg.norm(s.b)))
    return [x, r, np.array([res.niter, res.status, sol.stats()["iterations"]]), np.array([res.ini_res, res.fin_res])]


@pytest.mark.parametrize("kind,shape,permute,method,literal", [
    (POISSON, (12, 11, 10), True, TFS_CG, 0), (POISSON, (30, 28, 26), True, TFS_CG, 0),
    (POISSON, (14, 13, 12), False, TFS_CG, 0), (POISSON, (50, 50, 50), True, TFS_CG, 0),
    (CONVDIFF, (20, 20, 20), True, TFS_CGS, 0), (POISSON, (16, 15, 14), True, TFS_BICG, 1)])
@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
@pytest.mark.parametrize("prec", [1, 2])
def test_bodies_whatever_came_before(kind, shape, permute, method, literal, mode, prec, gpu):
    s = system(kind, *shape, permute=permute)
    opts = {TFS_OPT_BICG: literal}
    with Solver(s.matrix(), precision=mode, options={**opts, TFS_OPT_LAUNCH: 1}) as sol:
        want = [_solve(sol, s, method, prec, n, rel) for n, rel in SERIES]
    with Solver(s.matrix(), precision=mode, options=opts) as sol:
        for _ in range(2):
            for (n, rel), w in zip(SERIES, want, strict=True):
                for a, b in zip(_solve(sol, s, method, prec, n, rel), w, strict=True):
                    assert np.array_equal(a, b), (n, rel)


@pytest.mark.parametrize("mode,prec", [(TFS_MIXED, 1), (TFS_FP64, 2)])
def test_kernel_launches_count_whole_bodies(mode, prec, gpu):
    """A solve's launches: those around the loop and an iteration's, times the
    iterations launched -- in bodies of four also those past the solve's end."""
    s = system(POISSON, 30, 28, 26)

    def count(sol, limit, rel):
        it = _solve(sol, s, TFS_CG, prec, limit, rel)[2][2]
        return it, sol.stats()["kernel_launches"]

    # (tiles whatever the limit: without iterations the level kernels are the default)
    with Solver(s.matrix(), precision=mode, options={TFS_OPT_DIC_TILES: 1}) as sol:
        assert count(sol, 0, 1e-30)[0] == 0
        around = sol.stats()["kernel_launches"]
        one = count(sol, 1, 1e-30)[1] - around
        assert one >= 3 and count(sol, 7, 1e-30) == (7, around + 7 * one)       # singly
        for limit in (12, 13, 14, 40, 41):
            assert count(sol, limit, 1e-30) == (limit, around + (limit + 3) // 4 * 4 * one)
        seen = set()
        for rel in (1e-3, 1e-4, 1e-5, 1e-6):
            it, launched = count(sol, 3000, rel)
            assert it >= 12 and launched == around + (it + 3) // 4 * 4 * one
            seen.add(it % 4)
        assert seen - {0}
