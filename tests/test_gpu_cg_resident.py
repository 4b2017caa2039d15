"""The binary64 CG loop of small systems in one kernel (diagonal or no
preconditioner): bitwise what the launches of the per-iteration kernels
(TFS_OPT_LAUNCH = 1) give, at the edges of a block (256 rows), of a row's width
(4, 8), of a block per multiprocessor and past the last size it takes."""
from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from helpers import system
from tflows import TFS_CG, TFS_FP64, Solver
from tflows.lib import TFS_OPT_LAUNCH, TfsError
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu

# (shape, whether one kernel solves it)
SHAPES = [((1, 1, 1), 1), ((2, 2, 2), 1), ((300, 1, 1), 1), ((16, 16, 1), 1), ((17, 16, 1), 1), ((16, 16, 16), 1),
          ((20, 21, 19), 1), ((36, 36, 30), 1), ((37, 36, 30), 1), ((42, 41, 40), 1), ((50, 50, 50), 0)]


def _solves(s, launch):
    out, kernels = [], []
    norm = float(np.linalg.norm(s.b))
    with Solver(s.matrix(), precision=TFS_FP64, options={TFS_OPT_LAUNCH: launch}) as sol:
        for prec, limit, rel in ((1, 1, 1e-8), (0, 30, 1e-8), (1, 25, 1e-30), (1, 2000, 1e-8), (1, 0, 1e-8), (1, 40, 2.0)):
            x, r = np.zeros(s.n), s.b.copy()
            res = sol.solve(TFS_CG, s.val, x, r, prec, limit, rel * norm)
            st = sol.stats()
            kernels.append(st["kernel_launches"])
            out += [x, r, np.array([res.niter, res.status, st["iterations"], st["spmv_launches"]]),
                    np.array([res.ini_res, res.fin_res])]
        bad = s.val.copy()
        bad[s.n // 2] = np.nan
        x, r = np.zeros(s.n), s.b.copy()
        try:
            res = sol.solve(TFS_CG, bad, x, r, 1, 20, 1e-8 * norm)
            out.append(np.array([res.niter, res.status]))
        except TfsError as e:
            out.append(np.array([-1, e.status]))
        x, r = np.zeros(s.n), s.b.copy()      # and a good solve after it
        sol.solve(TFS_CG, s.val, x, r, 1, 20, 1e-8 * norm)
        out += [x, r]
    return out, kernels


@pytest.mark.parametrize("shape,one", SHAPES)
def test_one_kernel_bitwise(shape, one, gpu):
    s = system(POISSON, *shape)
    got, kernels = _solves(s, 0)
    want, _ = _solves(s, 1)
    assert (len(set(kernels)) == 1) == bool(one), kernels
    for a, c in zip(got, want, strict=True):
        assert np.array_equal(a, c, equal_nan=True)


def test_one_kernel_from_several_threads(gpu):
    """Solves of several handles at once, a block per multiprocessor or two."""
    systems = [system(POISSON, *sh) for sh in ((32, 32, 32), (20, 20, 20), (42, 41, 40), (12, 11, 10), (36, 36, 30), (41, 40, 40))]

    def run(s, times):
        out = []
        with Solver(s.matrix(), precision=TFS_FP64) as sol:
            for _ in range(times):
                x, r = np.zeros(s.n), s.b.copy()
                sol.solve(TFS_CG, s.val, x, r, 1, 60, 1e-10 * float(np.linalg.norm(s.b)))
                out.append(x)
        return out

    want = [run(s, 1)[0] for s in systems]
    with ThreadPoolExecutor(len(systems)) as pool:
        for w, got in zip(want, pool.map(lambda s: run(s, 20), systems), strict=True):
            assert all(np.array_equal(w, x) for x in got)
