"""The waits of the binary64 CG in one kernel, each made to run out with a short
limit: a roll call that one block does not answer leaves the solve to the
launched kernels, to the same bits; a partial sum that one block withholds ends
the solve with TFS_ERR_TIMEOUT, whoever finds it, and the handle then solves as
before."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import system
from tflows import TFS_CG, Solver
from tflows.lib import TFS_ERR_ARG, TFS_ERR_TIMEOUT, TfsError, last_error, load_library
from tflows.synth import POISSON

SHAPES = [(2, 2, 2), (16, 16, 16), (20, 21, 19), (36, 36, 30), (42, 41, 40)]   # 1 block .. two a multiprocessor


def test_diag_resident_rejects_without_a_device():
    lib = load_library()
    assert lib.tfs_diag_resident(None, 1, 100) == TFS_ERR_ARG
    assert "tfs_diag_resident" in last_error()


def _solve(sol, s, limit=40, rel=1e-8):
    x, r = np.zeros(s.n), s.b.copy()
    res = sol.solve(TFS_CG, s.val, x, r, 1, limit, rel * float(np.linalg.norm(s.b)))
    return (x, r, np.array([res.niter, res.status, sol.stats()["iterations"]]), np.array([res.ini_res, res.fin_res]))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_a_roll_call_given_up(shape, gpu):
    lib = load_library()
    s = system(POISSON, *shape)
    with Solver(s.matrix()) as sol:
        for limit, rel in ((40, 1e-8), (3, 1e-30), (0, 1e-8), (40, 2.0)):   # .. both early exits
            want = _solve(sol, s, limit, rel)
            alone = sol.stats()["kernel_launches"]
            assert lib.tfs_diag_resident(sol.h, 1, 2000) == 0
            got = _solve(sol, s, limit, rel)
            if want[2][2]:
                assert sol.stats()["kernel_launches"] > alone
            assert lib.tfs_diag_resident(sol.h, 0, 0) == 0
            again = _solve(sol, s, limit, rel)
            assert sol.stats()["kernel_launches"] == alone
            for a, b, c in zip(want, got, again, strict=True):
                assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_a_withheld_partial_is_a_timeout(shape, gpu):
    lib = load_library()
    s = system(POISSON, *shape)
    with Solver(s.matrix()) as sol:
        want = _solve(sol, s)
        for _ in range(3):
            assert lib.tfs_diag_resident(sol.h, 2, 2000) == 0
            with pytest.raises(TfsError) as e:
                _solve(sol, s)
            assert e.value.status == TFS_ERR_TIMEOUT
            assert lib.tfs_diag_resident(sol.h, 0, 0) == 0
            for a, b in zip(want, _solve(sol, s), strict=True):
                assert np.array_equal(a, b)
        assert lib.tfs_diag_resident(sol.h, 3, 1) == TFS_ERR_ARG
        assert lib.tfs_diag_resident(sol.h, 1, 0) == TFS_ERR_ARG
