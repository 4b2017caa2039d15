"""Assembly of meshes whose cells come in their own order (a structured
numbering: rows in place, one a thread) and of those that do not, bitwise the
oracle's face loops: structured meshes, faces and cells partly shuffled on both
sides of the rule (half of the cells), rows of more than eight entries, sizes
around a warp's and a block's."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import tfs_oracle as O
from tflows import Matrix_Type, Solver

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, nz, shuffled, hub, seed):
    """nx x ny x nz cells numbered lexicographically, the first `shuffled` of them
    at random among themselves; cell hub joined to every seventh cell besides;
    boundary faces among the others."""
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    num = np.arange(n)
    num[:shuffled] = rng.permutation(shuffled)
    ids = num.reshape(nz, ny, nx) + 1
    faces = []
    for a, b in ((ids[:, :, :-1], ids[:, :, 1:]), (ids[:, :-1], ids[:, 1:]), (ids[:-1], ids[1:])):
        faces += list(zip(a.ravel(), b.ravel()))
    have = {tuple(sorted(f)) for f in faces}
    if hub:
        faces += [(hub, int(c)) for c in range(1, n + 1, 7) if c != hub and tuple(sorted((hub, c))) not in have]
    faces = [(min(f), max(f)) for f in faces]
    faces.sort()
    out = []
    for k, f in enumerate(faces):
        out.append(f)
        if k % 15 == 3:
            out.append((f[0], -1 - k))
    return n, np.array(out if out else [(1, -1)], np.int32)


@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 1, 1), (33, 1, 1), (8, 8, 4), (257, 1, 1), (20, 19, 18), (64, 33, 9)])
@pytest.mark.parametrize("shuffle,hub", [(0.0, 0), (0.45, 0), (0.55, 0), (1.0, 0), (0.0, 5), (0.6, 5)])
def test_ordered_and_scattered(dims, shuffle, hub, gpu):
    n = dims[0] * dims[1] * dims[2]
    n, faces = _mesh(*dims, int(shuffle * n), hub if n > 40 else 0, seed=n)
    row, col, dia, mir, pos = O.topology(n, faces)
    nf = len(faces)
    rng = np.random.default_rng(3)
    a12, a21, d12, d21 = (rng.uniform(0.1, 2.0, nf) for _ in range(4))
    d12[(faces[:, 1] <= 0) & (rng.uniform(size=nf) < 0.4)] = 0.0
    cell, start = rng.uniform(0.0, 1.0, n), rng.uniform(-1.0, 1.0, len(col))
    with Solver(Matrix_Type(n, row, col, dia, start.copy())) as sol:
        sol.faces_register(faces, pos)
        for c in (cell, None):
            want = O.assemble_faces(n, faces.reshape(-1), pos.reshape(-1), dia, a12, a21, d12, d21, c, start)
            assert np.array_equal(sol.assemble(a12, a21, d12, d21, c, start), want)
