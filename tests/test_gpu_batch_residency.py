"""Batch kernels of one, two and three CTAs an SM, whichever the batch asks for:
every system's result is bitwise that of the system in a batch of its own."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import system
from tflows import TFS_BICG, TFS_CG, TFS_FP64, TFS_MIXED, Batch, Solver
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu


def _run(batch, systems, method, prec, mode):
    xs, rs = [np.zeros(s.n) for s in systems], [s.b.copy() for s in systems]
    res = batch.solve(method, prec, [s.val for s in systems], xs, rs, 40, [1e-8 * float(np.linalg.norm(s.b)) for s in systems],
                      mode=mode)
    return xs, rs, res.niter


# (systems, cluster, threads): CTAs of 512 threads asked for an SM 0.1, 1.3, 2.5, 5.1
@pytest.mark.parametrize("n,cluster,threads", [(2, 8, 512), (24, 8, 512), (24, 16, 512), (48, 16, 512), (96, 16, 256)])
@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
@pytest.mark.parametrize("method,prec", [(TFS_CG, 1), (TFS_CG, 2), (TFS_BICG, 2)])
def test_results_do_not_depend_on_what_is_resident(n, cluster, threads, mode, method, prec, gpu):
    shapes = [(4, 4, 4), (9, 8, 7), (13, 12, 11)]
    kinds = [system(POISSON, *sh) for sh in shapes]
    systems = [kinds[k % 3] for k in range(n)]
    solvers = [Solver(s.matrix()) for s in systems]
    alone = []
    for k in range(min(3, n)):
        with Batch([solvers[k]], cluster, threads) as b:
            alone.append(_run(b, [systems[k]], method, prec, mode))
    with Batch(solvers, cluster, threads) as b:
        xs, rs, its = _run(b, systems, method, prec, mode)
    for k in range(n):
        x, r, it = alone[k % 3] if n >= 3 else alone[k]
        assert np.array_equal(xs[k], x[0]) and np.array_equal(rs[k], r[0]) and its[k] == it[0], k
    for s in solvers:
        s.close()
