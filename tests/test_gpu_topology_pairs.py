"""Device topology where several faces join the same pair of cells (two cells
across a periodic direction): columns as often as faces, mir of each of a pair's
entries the first of the mirrored ones, pos of each of its faces the last, and
the same on every call."""
from __future__ import annotations

import numpy as np
import pytest

from tflows.matrix_mod import Matrix_Mod_Topology_Device

pytestmark = pytest.mark.gpu


def _expected(n, faces):
    rows = [[c + 1] for c in range(n)]
    for c1, c2 in faces:
        if c2 > 0:
            rows[c1 - 1].append(c2)
            rows[c2 - 1].append(c1)
    rows = [sorted(r) for r in rows]
    row = np.concatenate([[1], 1 + np.cumsum([len(r) for r in rows])]).astype(np.int32)
    first = [{v: row[c] + r.index(v) for v in r} for c, r in enumerate(rows)]
    last = [{v: row[c + 1] - 1 - r[::-1].index(v) for v in r} for c, r in enumerate(rows)]
    mir = [first[v - 1][c + 1] for c, r in enumerate(rows) for v in r]
    pos = [(last[c1 - 1][c2], last[c2 - 1][c1]) if c2 > 0 else (0, 0) for c1, c2 in faces]
    dia = [last[c][c + 1] for c in range(n)]
    return row, np.concatenate(rows), np.array(dia), np.array(mir), np.array(pos)


@pytest.mark.parametrize("n,hub", [(2, 0), (7, 4), (300, 0), (300, 9), (5000, 40)])
def test_pairs_joined_twice(n, hub, gpu):
    """A chain, every third link of it twice and some three times (rows of up to
    seven entries, sorted in registers), and a first cell joined to cells 3 to
    hub (longer rows, sorted in place), the faces in any order and direction."""
    rng = np.random.default_rng(n + hub)
    pairs = [(c, c + 1) for c in range(1, n)] + [(c, c + 1) for c in range(1, n, 3)] + [(c, c + 1) for c in range(1, n, 9)]
    pairs += [(k, 1) for k in range(3, hub + 1)] + [(1, k) for k in range(3, hub + 1, 2)]
    pairs += [(c, -c) for c in range(1, n + 1, 5)]
    faces = np.array([p if p[1] < 0 or rng.integers(2) else p[::-1] for p in pairs], np.int32)
    faces = np.ascontiguousarray(faces[rng.permutation(len(faces))])
    row, col, dia, mir, pos = _expected(n, faces.tolist())
    for _ in range(3):
        dev = Matrix_Mod_Topology_Device(n, faces)
        assert np.array_equal(dev.row, row) and np.array_equal(dev.col, col) and np.array_equal(dev.dia, dia)
        assert np.array_equal(dev.mir, mir) and np.array_equal(dev.pos, pos)
