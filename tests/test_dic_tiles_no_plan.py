"""Nothing is planned, packed or kept for tiled DIC sweeps by calls that do not
sweep by tiles: the literal BiCG (two vectors a sweep), Prec_Form, a schedule
that the one-block DIC takes."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import system
from tflows import TFS_BICG, TFS_CG, TFS_FP64, TFS_MIXED, Solver
from tflows.lib import TFS_OPT_BICG, TFS_OPT_DIC_TILES
from tflows.synth import POISSON

pytestmark = pytest.mark.gpu


def _call(sol, s, what):
    if what == "form":
        return [sol.prec_form(s.val, 2)]
    x, r = np.zeros(s.n), s.b.copy()
    sol.solve(TFS_BICG if what == "literal" else TFS_CG, s.val, x, r, 2, 10, 1e-10 * float(np.linalg.norm(s.b)))
    return [x, r]


@pytest.mark.parametrize("what,shape,permute", [("literal", (24, 23, 22), True), ("form", (24, 23, 22), True),
                                                ("deep", (10, 9, 8), False)])
@pytest.mark.parametrize("mode", [TFS_FP64, TFS_MIXED])
def test_calls_without_tiled_sweeps_make_no_plan(what, shape, permute, mode, gpu):
    s = system(POISSON, *shape, permute=permute)
    seen = []
    for tiles in (0, 1):
        opts = {TFS_OPT_DIC_TILES: tiles, **({TFS_OPT_BICG: 1} if what == "literal" else {})}
        with Solver(s.matrix(), precision=mode, options=opts) as sol:
            out = _call(sol, s, what)
            st = sol.stats()
            assert st["dic_tiles"] == 0
            sol.solve(TFS_CG, s.val, np.zeros(s.n), s.b.copy(), 1, 1, 0.0)   # (fills device_bytes in)
            seen.append((out, sol.stats()["device_bytes"], st["kernel_launches"]))
    assert seen[0][1:] == seen[1][1:], [q[1:] for q in seen]
    assert all(np.array_equal(a, b) for a, b in zip(seen[0][0], seen[1][0], strict=True))
