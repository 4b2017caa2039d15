"""The work that users of this framework have it do, as cases that can be timed.

A flow solver registers its mesh once and then, every time step, hands over
new matrix values and right-hand sides: pressure systems (symmetric, Poisson
type) and momentum/scalar transport systems (non-symmetric), solved with a
small iteration limit or to a relative tolerance, from device arrays or from
the Fortran call's host arrays, one at a time, as a batch or through the
request server.  Around the solves stand the device assembly of the matrix
from face coefficients, the topology built from the faces of a mesh, and the
residual that allocates nothing.  The meshes are the repository's seeded
jittered hexahedra, numbered at random (as an unstructured generator leaves
them) or lexicographically (as a structured one does).

A case's mesh and the handle registered for it are kept for the process, as a
flow solver keeps them; every seed gives other cell diffusivities (hence other
matrix values) and another right-hand side.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

# (imported with the repository's root as the working folder)
sys.path.insert(0, str(Path("t-flows_gb300").resolve()))

import tflows  # noqa: E402
from tflows.synth import CONVDIFF, POISSON, SynthSystem  # noqa: E402

METHOD = {"cg": tflows.TFS_CG, "bicg": tflows.TFS_BICG, "cgs": tflows.TFS_CGS}
PREC = {"none": 0, "diag": 1, "dic": 2}
MODE = {"fp64": tflows.TFS_FP64, "mixed": tflows.TFS_MIXED}
TO_TOL = 5000          # iteration limit of the solves that run to their tolerance


def listed():
    solve = dict(kind="solve", numbering="random", arrays="device")
    return [
        # The headline workload: a two-million-cell pressure system solved to
        # 1e-8 with the reference's incomplete Cholesky, mixed precision.
        dict(solve, name="pressure 2M dic mixed", equation="pressure", nx=128, ny=128, nz=128,
             method="cg", prec="dic", mode="mixed", limit=TO_TOL, rel=1e-8),
        # The same pressure system as one time step of Process asks for it:
        # BiCG, at most 40 iterations, the reference's own arithmetic.
        dict(solve, name="pressure 2M dic fp64", equation="pressure", nx=128, ny=128, nz=128,
             method="bicg", prec="dic", mode="fp64", limit=40, rel=1e-8),
        # A transport equation to its tolerance with CGS and the diagonal.
        dict(solve, name="transport 2M cgs mixed", equation="transport", nx=128, ny=128, nz=128,
             method="cgs", prec="diag", mode="mixed", limit=TO_TOL, rel=1e-8),
        # One momentum component of a mid-sized run through the drop-in call:
        # host arrays, CG with a limit of 10, incomplete Cholesky, binary64.
        dict(solve, name="momentum 260k host", equation="transport", nx=65, ny=63, nz=64,
             method="cg", prec="dic", mode="fp64", limit=10, rel=1e-10, arrays="host"),
        # A small pressure system to tolerance, diagonal CG in binary64.
        dict(solve, name="pressure 32k diag fp64", equation="pressure", nx=32, ny=32, nz=32,
             method="cg", prec="diag", mode="fp64", limit=TO_TOL, rel=1e-8),
        # A structured mesh in its own numbering (long dependency chains in
        # the incomplete Cholesky), drop-in call.
        dict(solve, name="pressure 14k lexi host", equation="pressure", nx=25, ny=24, nz=24,
             numbering="lexicographic", method="cg", prec="dic", mode="mixed", limit=40, rel=1e-8,
             arrays="host"),
        # The smallest call: a test-sized mesh through the drop-in call.
        dict(solve, name="pressure 1k host", equation="pressure", nx=12, ny=11, nz=10, method="cg",
             prec="dic", mode="fp64", limit=20, rel=1e-8, arrays="host"),
        # Many independent pressure systems solved together.
        dict(kind="batch", name="batch of 24", systems=24, lo=5000, hi=100000, prec="diag", mode="mixed",
             limit=TO_TOL, rel=1e-8),
        # Requests arriving at the server together, sizes mixed.
        dict(kind="serve", name="serve 16 requests", systems=8, requests=16, lo=10000, hi=200000,
             mode="mixed", limit=300, rel=1e-8),
        # Matrix values assembled from face coefficients, every time step.
        dict(kind="assemble", name="assemble 2M", nx=128, ny=128, nz=128),
        # The topology of a mesh held on the device, once per mesh.
        dict(kind="topology", name="topology 2M", nx=128, ny=128, nz=128),
        # The residual a coupling loop computes without allocating.
        dict(kind="residual", name="residual 2M", nx=128, ny=128, nz=128),
    ]


def _dims(rng, lo, hi):
    """A mesh of roughly log-uniform size between lo and hi cells, sides uneven."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = n ** (1.0 / 3.0)
    nx = max(2, round(side * rng.uniform(0.75, 1.25)))
    ny = max(2, round(side * rng.uniform(0.75, 1.25)))
    return dict(nx=nx, ny=ny, nz=max(2, round(n / (nx * ny))))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["batch", "serve", "assemble", "topology", "residual"])
    if kind == "batch":
        lo = rng.randrange(2000, 10000)
        return dict(kind=kind, systems=rng.randrange(3, 29), lo=lo, hi=lo * rng.randrange(2, 16),
                    prec=rng.choice(["diag", "diag", "dic"]), mode=rng.choice(["mixed", "mixed", "fp64"]),
                    limit=rng.choice([60, 150]), rel=1e-8)
    if kind == "serve":
        lo = rng.randrange(5000, 20000)
        systems = rng.randrange(2, 9)
        return dict(kind=kind, systems=systems, requests=rng.randrange(systems, 3 * systems), lo=lo,
                    hi=lo * rng.randrange(2, 12), mode=rng.choice(["mixed", "mixed", "fp64"]),
                    limit=rng.choice([60, 150]), rel=1e-8)
    if kind in ("assemble", "topology", "residual"):
        return dict(kind=kind, **_dims(rng, 1000, 1900000))
    equation = rng.choice(["pressure", "pressure", "transport"])
    numbering = rng.choice(["random", "random", "random", "lexicographic"])
    arrays = rng.choice(["device", "device", "host"])
    method = rng.choice(["cg", "bicg"] if equation == "pressure" else ["cg", "bicg", "cgs"])
    prec = rng.choice(["dic", "dic", "diag", "none"] if equation == "pressure" else ["dic", "diag"])
    hi = 200000 if numbering == "lexicographic" else 400000 if arrays == "host" else 1500000
    size = _dims(rng, 1000, hi)
    # Small systems to their tolerance or a limit, large ones to a limit.
    small = size["nx"] * size["ny"] * size["nz"] < 200000 and numbering == "random"
    limit = rng.choice([40, 100, TO_TOL] if small and equation == "pressure" and prec != "none" else [10, 40])
    return dict(kind=kind, equation=equation, numbering=numbering, arrays=arrays, method=method, prec=prec,
                mode=rng.choice(["mixed", "fp64"]), limit=limit, rel=1e-8, **size)


# ---------------------------------------------------------------- meshes

_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


class _Mesh:
    """A seeded system and, per stored entry, its row and column (0-based)."""

    def __init__(self, equation, nx, ny, nz, numbering):
        s = SynthSystem(CONVDIFF if equation == "transport" else POISSON, nx, ny, nz,
                        permute=numbering == "random")
        self.s, self.n, self.nnz, self.equation = s, s.n, s.nnz, equation
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        to = lambda a: torch.from_numpy(a).to(self.dev)  # noqa: E731
        self.row0 = to(s.row).long() - 1
        self.cols = to(s.col).long() - 1
        self.rows = torch.repeat_interleave(torch.arange(s.n, device=self.dev), self.row0.diff())
        self.dia0 = to(s.dia).long() - 1
        v = to(s.val)
        self.off = v.clone()
        self.off[self.dia0] = 0.0
        # what a row's diagonal holds beyond its neighbours' coefficients
        self.rest = (v[self.dia0] + self.row_sums(self.off)).clamp(min=0.0)

    def row_sums(self, entries):
        """The sum of every row's entries, in their order (the same on every run)."""
        total = entries.new_zeros(self.n)
        begin, end = self.row0[:-1], self.row0[1:]
        for k in range(int((end - begin).max())):
            total += torch.where(begin + k < end, entries[(begin + k).clamp(max=self.nnz - 1)], 0.0)
        return total

    def values(self, rng):
        """Matrix values with cell diffusivities in [0.5, 2] (their harmonic
        mean on every face) and a right-hand side in [-1, 1]."""
        g = torch.from_numpy(rng.uniform(0.5, 2.0, self.n)).to(self.dev)
        off = self.off * (2.0 * g[self.rows] * g[self.cols] / (g[self.rows] + g[self.cols]))
        val = off.clone()
        val[self.dia0] = self.rest - self.row_sums(off)
        b = torch.from_numpy(rng.uniform(-1.0, 1.0, self.n)).to(self.dev)
        x0 = torch.zeros_like(b)
        if self.equation == "transport":     # the previous time step's field
            x0 = torch.from_numpy(rng.uniform(-1.0, 1.0, self.n)).to(self.dev)
        return val, b, x0


def _mesh(c):
    numbering = c.get("numbering", "random")
    key = ("mesh", c.get("equation", "pressure"), c["nx"], c["ny"], c["nz"], numbering)
    return _keep(key, lambda: _Mesh(key[1], c["nx"], c["ny"], c["nz"], numbering))


def _sizes(c):
    """The meshes of a batch or a server's systems: log-uniform in [lo, hi],
    k x k x m cells."""
    out = []
    for k in range(c["systems"]):
        u = (0.5 + (k * 0.6180339887498949)) % 1.0
        n = c["lo"] * (c["hi"] / c["lo"]) ** u
        side = max(2, round(n ** (1.0 / 3.0)))
        out.append((side, side, max(1, round(n / (side * side)))))
    return out


def _many(c):
    """The meshes of a batch or server case: a served pool holds pressure and
    (every fourth) transport systems."""
    out = []
    for k, (nx, ny, nz) in enumerate(_sizes(c)):
        equation = "transport" if c["kind"] == "serve" and k % 4 == 3 else "pressure"
        out.append(_mesh(dict(equation=equation, nx=nx, ny=ny, nz=nz)))
    return out


def _solver(c, m, prec, mode):
    """The handle that a program keeps for a mesh."""
    key = ("solver", c["kind"], m.equation, m.s.dims, c.get("numbering", "random"), prec, mode)
    return _keep(key, lambda: tflows.Solver(m.s.matrix(), precision=MODE[mode]))


# ------------------------------------------------------- prepare and run

def prepare(case, seed):
    return {"solve": _prepare_solve, "batch": _prepare_batch, "serve": _prepare_serve,
            "assemble": _prepare_assemble, "topology": _prepare_topology,
            "residual": _prepare_residual}[case["kind"]](case, np.random.default_rng(seed))


def run(state):
    return state["run"](state)


def _prepare_solve(c, rng):
    m = _mesh(c)
    val, b, x0 = m.values(rng)
    tol = c["rel"] * float(b.norm())
    st = dict(c=c, tol=tol, sol=_solver(c, m, c["prec"], c["mode"]))
    if c["arrays"] == "host":
        st.update(run=_run_host, val=val.cpu().numpy(), b=b.cpu().numpy(), x0=x0.cpu().numpy(),
                  x=np.zeros(m.n), r=np.zeros(m.n))
    else:
        st.update(run=_run_device, val=val, b=b, x0=x0, x=torch.zeros_like(b), r=torch.zeros_like(b))
    return st


def _run_host(st):
    """One drop-in call: x and r1 = b set by the caller, both overwritten."""
    c, sol = st["c"], st["sol"]
    np.copyto(st["x"], st["x0"])
    np.copyto(st["r"], st["b"])
    res = sol.solve(METHOD[c["method"]], st["val"], st["x"], st["r"], PREC[c["prec"]], c["limit"], st["tol"])
    return {"x": st["x"], "r1": st["r"], "niter": res.niter, "ini_res": res.ini_res, "fin_res": res.fin_res}


def _p(t):
    return C.c_void_p(t.data_ptr())


def _run_device(st):
    """The same on device arrays, x and r1 set by copies on the handle's stream."""
    c, sol, nb = st["c"], st["sol"], 8 * st["x"].numel()
    sol.lib.tfs_copy(sol.h, _p(st["x"]), _p(st["x0"]), nb)
    sol.lib.tfs_copy(sol.h, _p(st["r"]), _p(st["b"]), nb)
    res = sol.solve_device(METHOD[c["method"]], st["val"].data_ptr(), st["x"].data_ptr(), st["r"].data_ptr(),
                           PREC[c["prec"]], c["limit"], st["tol"])
    return {"x": st["x"], "r1": st["r"], "niter": res.niter, "ini_res": res.ini_res, "fin_res": res.fin_res}


def _flat(ms, rng):
    """Every system's arrays one after the other: (values, b, x0, their views)."""
    parts = [m.values(rng) for m in ms]
    flat = [torch.cat([p[k] for p in parts]) for k in range(3)]
    return flat, [float(p[1].norm()) for p in parts]


def _views(flat, lengths):
    return list(torch.split(flat, lengths))


def _prepare_batch(c, rng):
    ms = _many(c)
    (val, b, x0), norms = _flat(ms, rng)
    key = ("batch",) + tuple(sorted((k, v) for k, v in c.items() if k != "name"))
    batch = _keep(key, lambda: tflows.Batch([_solver(c, m, c["prec"], c["mode"]) for m in ms], 16, 512))
    x, r = torch.zeros_like(b), torch.zeros_like(b)
    ns, zs = [m.n for m in ms], [m.nnz for m in ms]
    ptrs = lambda flat, ls: [v.data_ptr() for v in _views(flat, ls)]  # noqa: E731
    return dict(run=_run_batch, c=c, batch=batch, val=val, b=b, x0=x0, x=x, r=r,
                p_val=ptrs(val, zs), p_x=ptrs(x, ns), p_r=ptrs(r, ns), tol=[c["rel"] * t for t in norms])


def _run_batch(st):
    c, batch, nb = st["c"], st["batch"], 8 * st["x"].numel()
    two = lambda *v: (C.c_void_p * 2)(*v)  # noqa: E731
    batch.lib.tfs_batch_copy(batch.b, 2, two(st["x"].data_ptr(), st["r"].data_ptr()),
                             two(st["x0"].data_ptr(), st["b"].data_ptr()), (C.c_size_t * 2)(nb, nb))
    res = batch.solve_device(tflows.TFS_CG, PREC[c["prec"]], st["p_val"], st["p_x"], st["p_r"], c["limit"],
                             st["tol"], mode=MODE[c["mode"]])
    return {"x": st["x"], "r1": st["r"], "niter": res.niter, "ini_res": res.ini_res, "fin_res": res.fin_res,
            "status": res.status}


def _served(c):
    """(system, method, preconditioner, limit) of every request: pressure
    systems by CG, transport systems by BiCG with the call sites' limit of
    10; incomplete Cholesky and the diagonal in turn."""
    out = []
    for q in range(c["requests"]):
        k = (q * 3) % c["systems"] if c["systems"] % 3 else q % c["systems"]
        transport = k % 4 == 3
        out.append((k, "bicg" if transport else "cg", "dic" if k % 2 else "diag", 10 if transport else c["limit"]))
    return out


def _prepare_serve(c, rng):
    ms = _many(c)

    def make():
        server = tflows.Server(64 << 30, max_inflight=8)
        return server, [server.add_system(m.n, m.s.row, m.s.col, m.s.dia) for m in ms]

    server, ids = _keep(("serve",) + tuple(sorted((k, v) for k, v in c.items() if k != "name")), make)
    asked = _served(c)
    (val, b, _), norms = _flat([ms[k] for k, *_ in asked], rng)
    x, r = torch.zeros_like(b), torch.zeros_like(b)
    ns, zs = [ms[k].n for k, *_ in asked], [ms[k].nnz for k, *_ in asked]
    todo = [(ids[k], METHOD[me], PREC[pr], v.data_ptr(), xx.data_ptr(), rr.data_ptr(), li, c["rel"] * t, bb.data_ptr())
            for (k, me, pr, li), v, xx, rr, bb, t in zip(asked, _views(val, zs), _views(x, ns), _views(r, ns),
                                                         _views(b, ns), norms)]
    return dict(run=_run_serve, c=c, server=server, todo=todo, val=val, b=b, x=x, r=r)


def _run_serve(st):
    server, mode = st["server"], MODE[st["c"]["mode"]]
    tickets = [server.submit(i, me, pr, v, x, r, li, tol, mode=mode, d_b=b, x0_zero=True)
               for i, me, pr, v, x, r, li, tol, b in st["todo"]]
    res = [server.wait(t) for t in tickets]
    return {"x": st["x"], "r1": st["r"], "niter": np.array([q["niter"] for q in res]),
            "status": np.array([q["status"] for q in res]), "ini_res": np.array([q["ini_res"] for q in res]),
            "fin_res": np.array([q["fin_res"] for q in res])}


def _faces(c):
    """Every face of the mesh: the interior ones, and a boundary face for each
    seventh cell, spread among them; with the topology they give."""
    m = _mesh(c)

    def make():
        inner = m.s.faces_c
        nb = max(1, m.n // 7)
        outer = np.stack([np.arange(1, m.n + 1, dtype=np.int32)[::7][:nb],
                          -np.arange(1, nb + 1, dtype=np.int32)[:len(np.arange(m.n)[::7][:nb])]], axis=1)
        at = np.linspace(0, len(inner), len(outer)).astype(np.int64)
        faces = np.insert(inner, at, outer, axis=0).astype(np.int32)
        return faces, tflows.Matrix_Mod_Topology(m.n, faces)

    return (m,) + _keep(("faces", m.s.dims, m.equation), make)


def _prepare_assemble(c, rng):
    m, faces, A = _faces(c)

    def make():
        sol = tflows.Solver(A)
        sol.faces_register(faces, A.pos)
        return sol

    sol = _keep(("assembler", m.s.dims), make)
    coef = [torch.from_numpy(rng.uniform(0.1, 1.0, len(faces))).to(m.dev) for _ in range(4)]
    coef.append(torch.from_numpy(rng.uniform(0.1, 1.0, m.n)).to(m.dev))
    val0 = torch.zeros(A.nnz, dtype=torch.float64, device=m.dev)
    return dict(run=_run_assemble, sol=sol, coef=coef, val0=val0, val=torch.zeros_like(val0))


def _run_assemble(st):
    sol = st["sol"]
    sol.lib.tfs_copy(sol.h, _p(st["val"]), _p(st["val0"]), 8 * st["val"].numel())
    if sol.lib.tfs_assemble_faces_device(sol.h, *(_p(t) for t in st["coef"]), _p(st["val"])):
        raise RuntimeError(tflows.lib.last_error())
    return st["val"]


def _prepare_topology(c, rng):
    m, faces, _ = _faces(c)
    # the mesh as this seed orders its faces, each given from either side
    order = rng.permutation(len(faces)) if len(faces) < 200000 else np.roll(np.arange(len(faces)),
                                                                            int(rng.integers(1, len(faces))))
    f = faces[order].copy()
    flip = (f[:, 1] > 0) & (rng.random(len(f)) < 0.5)
    f[flip] = f[flip][:, ::-1]
    f = torch.from_numpy(f).to(m.dev)
    nf, cap = len(faces), m.n + 2 * len(faces)
    make = lambda k: torch.zeros(k, dtype=torch.int32, device=m.dev)  # noqa: E731
    return dict(run=_run_topology, lib=tflows.load_library(), n=m.n, nf=nf, faces=f, row=make(m.n + 1), col=make(cap),
                dia=make(m.n), mir=make(cap), pos=make(2 * nf))


def _run_topology(st):
    nnz = C.c_int32()
    if st["lib"].tfs_topology_build_device(st["n"], st["nf"], _p(st["faces"]), _p(st["row"]), _p(st["col"]),
                                           _p(st["dia"]), _p(st["mir"]), _p(st["pos"]), C.byref(nnz)):
        raise RuntimeError(tflows.lib.last_error())
    k = nnz.value                                  # col and mir are defined up to here
    return {"row": st["row"], "col": st["col"][:k], "dia": st["dia"], "mir": st["mir"][:k], "pos": st["pos"], "nnz": k}


def _prepare_residual(c, rng):
    m = _mesh(c)
    val, b, _ = m.values(rng)
    x = torch.from_numpy(rng.uniform(-1.0, 1.0, m.n)).to(m.dev)
    to = lambda a: torch.from_numpy(a).to(m.dev)  # noqa: E731
    row, col = _keep(("csr", m.s.dims, m.equation), lambda: (to(m.s.row), to(m.s.col)))
    return dict(run=_run_residual, lib=tflows.load_library(), n=m.n, row=row, col=col, val=val, x=x, b=b,
                r=torch.zeros_like(b), norm=torch.zeros(1, dtype=torch.float64, device=m.dev))


def _run_residual(st):
    st["r"].copy_(st["b"])
    s = torch.cuda.current_stream().cuda_stream
    if st["lib"].tfs_residual_norm_noalloc(st["n"], _p(st["row"]), _p(st["col"]), _p(st["val"]), _p(st["x"]),
                                           _p(st["r"]), _p(st["norm"]), C.c_void_p(s)):
        raise RuntimeError(tflows.lib.last_error())
    return {"r1": st["r"], "norm": st["norm"]}


# ------------------------------------------------------------------ work

def _iterations(equation, prec, method, limit, n):
    """Iterations of a solve: its limit, or about what its tolerance takes."""
    if limit < TO_TOL:
        return limit
    side = n ** (1.0 / 3.0)
    return 9 if equation == "transport" else round((2.9 if prec == "dic" else 7.5) * side)


def _solve_work(n, nnz, iterations, prec, method, mode):
    """Each iteration: one pass over the matrix per product (two for CGS), one
    more per incomplete Cholesky application, the iteration's vectors once."""
    v = 4 if mode == "mixed" else 8
    passes = 2 if method == "cgs" else 1
    sweep = passes if prec == "dic" else 0
    vectors = 14 if method == "cgs" else 10
    per = passes * (v + 4) * nnz + sweep * ((v + 4) * (nnz - n) + 3 * v * n) + vectors * v * n
    flops = (passes + sweep) * 2 * nnz + vectors * n
    once = 12 * nnz + 32 * n        # values and indices in, b and x in, x and r1 out
    return once + iterations * per, 2 * nnz + iterations * flops


def _cells(nx, ny, nz):
    n = nx * ny * nz
    inner = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
    return n, n + 2 * inner, inner


def work(case):
    c = case
    if c["kind"] in ("batch", "serve"):
        systems = [(_cells(*d), k) for k, d in enumerate(_sizes(c))]
        if c["kind"] == "batch":
            asked = [(k, "cg", c["prec"], c["limit"]) for k in range(c["systems"])]
        else:
            asked = _served(c)
        total = [_solve_work(systems[k][0][0], systems[k][0][1],
                             _iterations("pressure", pr, me, li, systems[k][0][0]), pr, me, c["mode"])
                 for k, me, pr, li in asked]
        return {"bytes": sum(t[0] for t in total), "flops": sum(t[1] for t in total)}
    n, nnz, inner = _cells(c["nx"], c["ny"], c["nz"])
    nf = inner + len(range(0, n, 7))
    if c["kind"] == "solve":
        its = _iterations(c["equation"], c["prec"], c["method"], c["limit"], n)
        by, fl = _solve_work(n, nnz, its, c["prec"], c["method"], c["mode"])
        return {"bytes": by, "flops": fl}
    if c["kind"] == "assemble":     # values set and updated, four coefficients and two cells a face
        return {"bytes": 8 * nnz * 2 + 40 * nf + 8 * n, "flops": 4 * nf + n}
    if c["kind"] == "topology":     # faces in; row, col, dia, mir, pos out
        return {"bytes": 8 * nf + 4 * (n + 1) + 8 * nnz + 4 * n + 8 * nf, "flops": 0}
    return {"bytes": 12 * nnz + 4 * (n + 1) + 32 * n, "flops": 2 * nnz + 2 * n}


# ----------------------------------------------------------------- exact

class _Dic:
    """Diagonal incomplete Cholesky by levels of independent rows, in torch."""

    def __init__(self, m, val):
        dev, n = m.dev, m.n
        low, up = m.cols < m.rows, m.cols > m.rows
        level = torch.zeros(n, dtype=torch.long, device=dev)
        r, k = m.rows[low], m.cols[low]
        while True:
            new = torch.zeros_like(level).scatter_reduce_(0, r, level[k] + 1, "amax")
            if bool((new == level).all()):
                break
            level = new
        order = torch.argsort(level, stable=True)
        self.at = [order[level[order] == v] for v in range(int(level.max()) + 1)] if int(level.max()) < 8 else \
            list(torch.split(order, torch.bincount(level).tolist()))
        place = torch.empty(n, dtype=torch.long, device=dev)
        for rows in self.at:
            place[rows] = torch.arange(len(rows), device=dev)

        def parts(mask):
            rr, kk, vv, lv = m.rows[mask], m.cols[mask], val[mask], level[m.rows[mask]]
            o = torch.argsort(lv, stable=True)
            sizes = torch.bincount(lv, minlength=len(self.at)).tolist()
            return list(zip(*(torch.split(t[o], sizes) for t in (place[rr], kk, vv))))

        self.low, self.up = parts(low), parts(up)
        self.d = torch.zeros(n, dtype=torch.float64, device=dev)
        diag = val[m.dia0]
        for rows, (q, k, v) in zip(self.at, self.low):
            self.d[rows] = 1.0 / diag[rows].index_add(0, q, -(self.d[k] * v * v))

    def __call__(self, b):
        y, d = torch.zeros_like(b), self.d
        for rows, (q, k, v) in zip(self.at, self.low):
            y[rows] = b[rows].index_add(0, q, -(v * y[k])) * d[rows]
        y = y / (d + 1e-30)
        z = torch.zeros_like(b)
        for rows, (q, k, v) in zip(reversed(self.at), reversed(self.up)):
            z[rows] = y[rows].index_add(0, q, -(v * z[k])) * d[rows]
        return z


def _plain_solve(m, val, b, x0, method, prec, limit, tol):
    """The reference's CG (its BiCG gives the same iterates) and CGS in 64 bits."""
    a = torch.sparse_csr_tensor(m.row0, m.cols, val, size=(m.n, m.n))
    diag = val[m.dia0]
    inv = _Dic(m, val) if prec == "dic" else (lambda r: r / diag) if prec == "diag" else (lambda r: r.clone())
    x, r = x0.clone(), b - a @ x0
    ini = fin = float(r.norm())
    if fin < tol:
        return x, r, ini, fin
    shadow, p, q, u2, rho_old = r.clone(), None, None, None, None
    for it in range(1, limit + 1):
        if method == "cgs":
            rho = shadow @ r
            if it == 1:
                u1, u2 = r.clone(), r.clone()
            else:
                beta = rho / rho_old
                u1 = r + beta * q
                u2 = u1 + beta * (q + beta * u2)
            v = a @ inv(u2)
            alpha = rho / (shadow @ v)
            q = u1 - alpha * v
            w = inv(u1 + q)
            x += alpha * w
            r -= alpha * (a @ w)
        else:
            z = inv(r)
            rho = r @ z
            p = z if it == 1 else z + (rho / rho_old) * p
            q = a @ p
            alpha = rho / (p @ q)
            x += alpha * p
            r -= alpha * q
        fin = float(r.norm())
        if fin < tol:
            break
        rho_old = rho
    return x, r, ini, fin


def _solved(x, r, ini, fin, limited):
    """A solve stopped by its tolerance leaves a residual of rounding noise:
    only its solution and first residual are values to compare."""
    return {"x": x, "r1": r if limited else None, "niter": None, "ini_res": ini, "fin_res": fin if limited else None}


def exact(case, seed):
    c, rng = case, np.random.default_rng(seed)
    if c["kind"] == "solve":
        m = _mesh(c)
        val, b, x0 = m.values(rng)
        x, r, ini, fin = _plain_solve(m, val, b, x0, c["method"], c["prec"], c["limit"], c["rel"] * float(b.norm()))
        limited = fin >= c["rel"] * float(b.norm()) and c["mode"] == "fp64"
        return _solved(x, r, ini, fin, limited)
    if c["kind"] in ("batch", "serve"):
        ms = _many(c)
        asked = _served(c) if c["kind"] == "serve" else [(k, "cg", c["prec"], c["limit"]) for k in range(len(ms))]
        xs, inis = [], []
        for k, me, pr, li in asked:
            m = ms[k]
            val, b, x0 = m.values(rng)
            x0 = torch.zeros_like(x0) if c["kind"] == "serve" else x0
            x, _, ini, _ = _plain_solve(m, val, b, x0, me, pr, li, c["rel"] * float(b.norm()))
            xs.append(x)
            inis.append(ini)
        return {"x": torch.cat(xs), "r1": None, "niter": None, "status": None, "ini_res": np.array(inis),
                "fin_res": None}
    if c["kind"] == "assemble":
        m, faces, A = _faces(c)
        f = [torch.from_numpy(rng.uniform(0.1, 1.0, len(faces))).to(m.dev) for _ in range(4)]
        cell = torch.from_numpy(rng.uniform(0.1, 1.0, m.n)).to(m.dev)
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(m.dev).long()  # noqa: E731
        fc, pos, dia = to(faces), to(A.pos), to(A.dia) - 1
        inner = fc[:, 1] > 0
        val = torch.zeros(A.nnz, dtype=torch.float64, device=m.dev)
        val.index_add_(0, pos[inner, 0] - 1, -f[0][inner])
        val.index_add_(0, pos[inner, 1] - 1, -f[1][inner])
        val.index_add_(0, dia[fc[:, 0] - 1], f[2])
        val.index_add_(0, dia[fc[inner, 1] - 1], f[3][inner])
        val.index_add_(0, dia, cell)
        return val
    if c["kind"] == "residual":
        m = _mesh(c)
        val, b, _ = m.values(rng)
        x = torch.from_numpy(rng.uniform(-1.0, 1.0, m.n)).to(m.dev)
        r = b - torch.sparse_csr_tensor(m.row0, m.cols, val, size=(m.n, m.n)) @ x
        return {"r1": r, "norm": r.norm().reshape(1)}
    return None
