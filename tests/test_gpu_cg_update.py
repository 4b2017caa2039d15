"""The binary64 CG update's instances by the chunks of 256 rows a system has: one
chunk a block with four blocks a multiprocessor (up to five chunks each), with
eight, then two and four chunks a block -- both sides of every line against the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import SOL_REL, oracle_solve, rel_l2, system
from tflows import TFS_CG, Solver
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu


# 312 chunks; 752 and 764; 1212 and 1232; 2428 and 2456
@pytest.mark.parametrize("shape", [(43, 43, 43), (58, 58, 57), (58, 58, 58), (68, 68, 67), (68, 68, 68), (86, 86, 84),
                                   (86, 86, 85)])
@pytest.mark.parametrize("prec", [1, 2])
def test_update_against_the_oracle(shape, prec, gpu):
    s = system(POISSON, *shape)
    ref = oracle_solve(s, TFS_CG, prec, niter=12, rel=1e-30)
    with Solver(s.matrix()) as sol:
        x, r = np.zeros(s.n), s.b.copy()
        res = sol.solve(TFS_CG, s.val, x, r, prec, 12, ref["tol"])
    assert res.niter == ref["niter"] == 13
    assert rel_l2(x, ref["x"]) <= SOL_REL and rel_l2(r, ref["r"]) <= SOL_REL
    assert abs(res.fin_res - ref["fin"]) <= SOL_REL * ref["fin"]
