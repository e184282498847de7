"""Performance cases: the work a user of this package has it do, through its
public entry points, over the range of sizes it is used at.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call (meshes,
contexts, right-hand sides), ``run(state)`` makes one pass and returns its
outputs whole, ``work(case)`` counts the bytes and operations no
implementation can do without (each input read once, each output written
once), ``exact(case, seed)`` gives the outputs where they are known in 64
bits: the linear systems are set up from a known solution.

Meshes are the jittered unit-square meshes of the benchmark (quadrilaterals,
triangles, or the mixed mesh).  A mesh and its matrix structure are built
once per process and shared by the states, as a program builds them once
and solves many systems on them; right-hand sides, matrix values, fields
and start states follow the seed.
"""
import functools

import numpy as np
import torch

from fortranfvcell_gb300 import Context, solver
from fortranfvcell_gb300 import autograd, cases, cells, mesh
from fortranfvcell_gb300.solver import make_opts, pack_block_diagonal


def listed():
    return [
        # the drop-in `solver` call on host arrays, as an unchanged host program
        # makes it: the p' system of a 48 x 48 cavity, Jacobi-PCG on CSRD
        dict(name="dropin_pcg_2k", op="dropin", nx=48, ny=48, kind="quad", system="pressure",
             matriz=1, code=1, tol=1e-10, precision="fp64"),
        # the same call for a momentum system in ELLPACK (the reference's
        # momentum storage and solver), warm-started from the last velocity
        dict(name="dropin_bicgstab_ell_40k", op="dropin", nx=211, ny=190, kind="quad",
             system="transport", matriz=4, code=2, tol=1e-11, precision="fp64", dom=0.05),
        # one FP64 matrix-vector product on the device, a mixed mesh of ~1M cells
        dict(name="spmv_f64_1m", op="spmv", nx=836, ny=836, kind="mixed", matriz=1, mode="fast"),
        # a pressure solve of ordinary size on device arrays, triangles, ELLPACK
        dict(name="pcg_f64_66k", op="solve", nx=181, ny=183, kind="tri", system="pressure",
             matriz=4, code=1, tol=1e-10, precision="fp64"),
        # the large pressure solve of the benchmark's family, plain FP64
        dict(name="pcg_f64_1m", op="solve", nx=836, ny=836, kind="mixed", system="pressure",
             matriz=1, code=1, tol=1e-8, precision="fp64"),
        # a large one in mixed precision (FP32 iterations, FP64 residuals), to a
        # residual at which the solution is FP64-accurate
        dict(name="pcg_mixed_1m", op="solve", nx=1024, ny=1021, kind="quad", system="pressure",
             matriz=1, code=1, tol=1e-12, precision="mixed"),
        # an enthalpy-sized transport solve: fresh values from the assembly, then
        # BiCGSTAB in FP64 (512 x 512 cells)
        dict(name="bicgstab_f64_262k", op="solve", nx=512, ny=512, kind="quad",
             system="transport", matriz=1, code=2, tol=1e-12, precision="fp64", dom=0.03),
        # a large unsymmetric solve in mixed precision
        dict(name="bicgstab_mixed_1m", op="solve", nx=836, ny=836, kind="mixed",
             system="transport", matriz=1, code=2, tol=1e-11, precision="mixed", dom=0.05),
        # many independent systems of uneven size in one call, pressure by PCG
        # and transport by BiCGSTAB side by side
        dict(name="batched_uneven_48", op="batched", nsys=48, lo=24, hi=140, kind="quad",
             tol=1e-12, precision="mixed"),
        # one gradient step through a differentiable solve: forward and adjoint
        dict(name="adjoint_66k", op="adjoint", nx=256, ny=257, kind="quad", tol=1e-12, dom=0.02),
        # the cell work of one SIMPLE outer iteration: gradients, both momentum
        # systems and the p' system of a mixed mesh
        dict(name="cells_200k", op="cells", nx=365, kind="mixed", geometry=True),
        # lid-driven cavity, 64 x 64: ten outer iterations from a saved state,
        # one CUDA graph launch each
        dict(name="simple_cavity_64", op="simple", nx=64, kind="quad", nit=10, tol=1e-10,
             gas=False),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    op = rng.choice(["dropin", "spmv", "solve", "solve", "batched", "adjoint", "cells", "simple"])
    log = lambda lo, hi: int(round(lo * (hi / lo) ** rng.random()))
    kind = rng.choice(["quad", "tri", "mixed"])
    if op == "dropin":
        nx = log(12, 200)
        system = rng.choice(["pressure", "transport"])
        matriz = 1 if kind == "mixed" else rng.choice([1, 4])
        return dict(op=op, nx=nx, ny=max(8, nx + rng.randint(-7, 7)), kind=kind, system=system,
                    matriz=matriz, code=1 if system == "pressure" else 2, tol=1e-11,
                    precision="fp64", dom=0.05)
    if op == "spmv":
        nx = log(60, 800)
        return dict(op=op, nx=nx, ny=nx + rng.randint(-9, 9), kind=kind, matriz=1,
                    mode=rng.choice(["fast", "reference", "f32"]))
    if op == "solve":
        system = rng.choice(["pressure", "transport"])
        nx = log(60, 620 if kind == "tri" else 800)
        matriz = 1 if kind == "mixed" else rng.choice([1, 4])
        precision = rng.choice(["fp64", "mixed"])
        return dict(op=op, nx=nx, ny=nx + rng.randint(-9, 9), kind=kind, system=system,
                    matriz=matriz, code=1 if system == "pressure" else 2,
                    tol=1e-9 if (system, precision) == ("pressure", "fp64") else 1e-12,
                    precision=precision,
                    dom=round(rng.uniform(0.02, 0.1), 3))
    if op == "batched":
        return dict(op=op, nsys=log(6, 48), lo=log(12, 24), hi=log(60, 140), kind=kind, tol=1e-12,
                    precision=rng.choice(["fp64", "mixed"]))
    if op == "adjoint":
        nx = log(40, 256)
        return dict(op=op, nx=nx, ny=nx + rng.randint(-9, 9), kind=kind, tol=1e-12,
                    dom=round(rng.uniform(0.02, 0.1), 3))
    if op == "cells":
        return dict(op=op, nx=log(24, 360), kind=kind, geometry=rng.random() < 0.7)
    return dict(op=op, nx=log(20, 64), kind=kind, nit=rng.randint(2, 8), tol=1e-10,
                gas=rng.random() < 0.5)


# ---- meshes and linear systems ---------------------------------------------

@functools.lru_cache(maxsize=3)
def _graph(nx, ny, kind):
    """Mesh, adjacency and RCM numbering of an nx x ny jittered unit square."""
    m = mesh.square_mesh(nx, ny, kind=kind, jitter=0.2, seed=1234)
    nelcon = mesh.adjacency(m)
    num = mesh.rcm(nelcon)
    return m, nelcon, num, mesh.numeq(num, nelcon)


@functools.lru_cache(maxsize=3)
def _pressure(nx, ny, kind, matriz):
    """The p' matrix (cell 1 pinned): ad, au, ia, ja, nad, the slots' rows and
    0-based columns, and the pinned row."""
    m, nelcon, num, ident = _graph(nx, ny, kind)
    ia, ja, nad = mesh.datastruc(ident, matriz, True)
    ad, au = mesh.assemble_pressure(m, nelcon, num, ia, ja, matriz, True, pin_cell=1)
    n = m.numel
    if matriz == 4:
        rows = np.repeat(np.arange(n), ja.shape[1])
    else:
        rows = np.repeat(np.arange(n), np.diff(ia))
    cols = ja.ravel()[: rows.size].astype(np.int64) - 1
    return ad, au, ia, ja, nad, rows, cols, int(num[0]) - 1


def _transport(ad, au, rows, n, seed, dom):
    """A convection-like unsymmetric matrix on a p' structure: off-diagonals
    scaled by 1 +- 0.4 per entry, the diagonal their absolute row sum plus
    the share dom (the time or relaxation term)."""
    au2 = au * (1.0 + 0.4 * np.random.default_rng(seed).uniform(-1.0, 1.0, au.size))
    ad2 = np.bincount(rows, weights=np.abs(au2[: rows.size]), minlength=n) * (1.0 + dom) + 1e-3
    return ad2, au2


def _field(n, seed):
    """A smooth field along the numbering with a little noise, of order 1."""
    rng = np.random.default_rng(seed)
    s = np.arange(n) / max(n - 1, 1)
    x = np.zeros(n)
    for k in range(1, 6):
        x += rng.normal() / k * np.cos(np.pi * k * s + rng.uniform(0, np.pi))
    return x + 0.01 * rng.normal(size=n)


def _linear(case, seed, x=None):
    """ad, au, structure, right-hand side and known solution of a case."""
    ad, au, ia, ja, nad, rows, cols, pin = _pressure(case["nx"], case["ny"], case["kind"],
                                                     case.get("matriz", 1))
    n = ad.size
    if x is None:
        x = _field(n, seed)
    if case.get("system", "transport") == "transport":
        ad, au = _transport(ad, au, rows, n, seed, case["dom"])
    else:
        x = x - x[pin]                       # the pin holds p' = 0 there
    b = ad * x + np.bincount(rows, weights=au[: rows.size] * x[cols], minlength=n)
    return dict(n=n, nad=nad, ad=ad, au=au, ia=ia, ja=ja, rows=rows, cols=cols, b=b, x=x)


def _cuda(a, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


def _context(s, matriz):
    c = Context()
    c.set_matrix(matriz, True, s["n"], s["nad"], s["ad"], s["au"], s["au"], s["ia"], s["ja"])
    c.set_stream(torch.cuda.current_stream())
    return c


# ---- the passes ------------------------------------------------------------

def _prepare_dropin(case, seed):
    s = _linear(case, seed)
    guess = s["x"] * (1.0 + 0.05 * np.random.default_rng(seed + 1).uniform(-1, 1, s["n"]))
    return dict(s, case=case, guess=guess, opts=make_opts(case["precision"]))


def _run_dropin(st):
    c = st["case"]
    x = st["guess"].copy()
    solver(st["ad"], st["au"], st["au"], x, st["b"], st["ia"], st["ja"], st["n"], st["nad"], True,
           c["tol"], 50000, c["code"], c["matriz"], 0, st["opts"])
    return x


def _prepare_spmv(case, seed):
    s = _linear(dict(case, system="pressure"), seed)
    f32 = case["mode"] == "f32"
    x = _cuda(s["x"], torch.float32 if f32 else torch.float64)
    return dict(ctx=_context(s, case["matriz"]), x=x, y=torch.empty_like(x), mode=case["mode"])


def _run_spmv(st):
    c = st["ctx"]
    {"fast": c.spmv_fast, "reference": c.spmv, "f32": c.spmv_f32}[st["mode"]](st["x"], st["y"])
    return st["y"]


def _prepare_solve(case, seed):
    s = _linear(case, seed)
    guess = s["x"] * (1.0 + 0.05 * np.random.default_rng(seed + 1).uniform(-1, 1, s["n"]))
    return dict(case=case, ctx=_context(s, case["matriz"]), b=_cuda(s["b"]), guess=_cuda(guess),
                x=torch.empty(s["n"], dtype=torch.float64, device="cuda"), ad=_cuda(s["ad"]),
                au=_cuda(s["au"]), opts=make_opts(case["precision"]))


def _run_solve(st):
    c = st["case"]
    st["x"].copy_(st["guess"])                   # ELLPACK solves start from it
    st["ctx"].update_values_async(st["ad"], st["au"], st["au"])
    st["ctx"].solve(c["code"], st["b"], st["x"], c["tol"], 50000, st["opts"])
    return st["x"]


def _batch_sides(case):
    """Grid sides spread over lo..hi (their logarithm), a fixed shuffle."""
    k = case["nsys"]
    f = np.random.default_rng(k).permutation(k) / max(k - 1, 1)
    return [int(round(case["lo"] * (case["hi"] / case["lo"]) ** v)) for v in f]


@functools.lru_cache(maxsize=8)
def _batch_system(nx, kind):
    m = mesh.square_mesh(nx, nx + 1, kind=kind, jitter=0.2, seed=nx)
    nelcon = mesh.adjacency(m)
    num = mesh.rcm(nelcon)
    ia, ja, nad = mesh.datastruc(mesh.numeq(num, nelcon), 1, True)
    ad, au = mesh.assemble_pressure(m, nelcon, num, ia, ja, 1, True, pin_cell=1)
    return ad, au, ia, ja, int(num[0]) - 1


def _batch(case, seed):
    systems, xs, bs, codes = [], [], [], []
    for k, nx in enumerate(_batch_sides(case)):
        ad, au, ia, ja, pin = _batch_system(nx, case["kind"])
        n = ad.size
        rows, cols = np.repeat(np.arange(n), np.diff(ia)), ja[: ia[-1] - 1].astype(np.int64) - 1
        x = _field(n, seed * 1000 + k)
        codes.append(1 + k % 2)
        if k % 2:
            ad, au = _transport(ad, au, rows, n, seed * 1000 + k, 0.05)
        else:
            x = x - x[pin]
        systems.append(dict(ad=ad, au=au, ia=ia, ja=ja))
        xs.append(x)
        bs.append(ad * x + np.bincount(rows, weights=au[: rows.size] * x[cols], minlength=n))
    p = pack_block_diagonal(systems)
    b, x = np.zeros(p["neq"]), np.zeros(p["neq"])
    for r, bk, xk in zip(p["rows"], bs, xs):
        b[r], x[r] = bk, xk
    return p, codes, b, x


def _prepare_batched(case, seed):
    p, codes, b, _ = _batch(case, seed)
    s = dict(n=p["neq"], nad=p["nad"], ad=p["ad"], au=p["au"], ia=p["ia"], ja=p["ja"])
    return dict(case=case, ctx=_context(s, 1), b=_cuda(b), row_start=p["row_start"], codes=codes,
                x=torch.zeros(p["neq"], dtype=torch.float64, device="cuda"),
                opts=make_opts(case["precision"], init=1))


def _run_batched(st):
    st["ctx"].solve_batched(st["row_start"], st["b"], st["x"], st["case"]["tol"], 50000,
                            st["opts"], codes=st["codes"])
    return st["x"]


def _adjoint(case, seed):
    """A system with known solution x, and the upstream gradient A^T lambda of a
    known adjoint solution lambda."""
    s = _linear(case, seed)
    lam = _field(s["n"], seed + 7)
    gx = s["ad"] * lam + np.bincount(s["cols"], weights=s["au"][: s["rows"].size] * lam[s["rows"]],
                                     minlength=s["n"])
    return s, lam, gx


def _prepare_adjoint(case, seed):
    s, _, gx = _adjoint(case, seed)
    sysm = autograd.CsrdSystem(s["ia"], s["ja"], s["n"], code=2, tol=case["tol"])
    leaf = lambda a: _cuda(a).requires_grad_()
    return dict(sys=sysm, ad=leaf(s["ad"]), au=leaf(s["au"][: s["nad"]]), b=leaf(s["b"]),
                gx=_cuda(gx))


def _run_adjoint(st):
    x = autograd.linear_solve(st["ad"], st["au"], st["b"], st["sys"])
    g = torch.autograd.grad(x, (st["ad"], st["au"], st["b"]), st["gx"])
    return [x.detach(), *g]


@functools.lru_cache(maxsize=3)
def _cavity(nx, kind, gas=False):
    """The lid-driven cavity, or the side-heated one of the ideal-gas loop."""
    if gas:
        return cases.natural_convection_cavity(nx, ra=1e5, kind=kind, jitter=0.1)
    return cases.lid_driven_cavity(nx, kind=kind, jitter=0.2 if kind != "quad" else 0.1)


def _flow(c, seed):
    """A recirculating start state: velocity (numel, 2) and pressure by cell."""
    rng = np.random.default_rng(seed)
    m = c["mesh"]
    used = (m.ix > 0)[..., None]
    xy = np.where(used, m.coor[np.maximum(m.ix, 1) - 1], 0.0).sum(1) / m.nsides[:, None]
    side = c.get("side", 1.0)
    a = rng.uniform(0.3, 1.0) * (0.05 if "side" in c else 1.0)   # air in a heated cavity is slow
    sx, sy = np.pi * xy[:, 0] / side, np.pi * xy[:, 1] / side
    w = a * np.stack([np.sin(sx) ** 2 * np.sin(2 * sy), -np.sin(2 * sx) * np.sin(sy) ** 2], 1)
    w += 0.01 * a * rng.normal(size=w.shape)
    p = a * a * (np.cos(sx) * np.cos(sy) + 0.01 * rng.normal(size=sx.size))
    return w, p


def _prepare_cells(case, seed):
    c = _cavity(case["nx"], case["kind"])
    n, nsh = c["numel"], c["nshared"]
    m = cells.CellMesh(c["coor"], c["ix"], c["nelcon"], c["num"], c["pedge"], c["sedge"], c["e"])
    if case["geometry"]:
        m.cache_geometry()
    ia4, ja4, _ = mesh.datastruc(c["ident"], 4, True)
    ia1, ja1, nad = mesh.datastruc(c["ident"], 1, True)
    w, p = _flow(c, seed)
    new = lambda *shape: torch.zeros(shape, dtype=torch.float64, device="cuda")
    st = dict(m=m, w=_cuda(w), u1=_cuda(w[:, 0]), u2=_cuda(w[:, 1]), p=_cuda(p), gp0=new(n, 2),
              ia4=_cuda(ia4, torch.int32), ja4=_cuda(ja4, torch.int32),
              ia1=_cuda(ia1, torch.int32), ja1=_cuda(ja1, torch.int32))
    cells.gradient(m, 2, 3, st["p"], st["gp0"])
    # the systems' padding slots are never written; they start at zero
    st["out"] = dict(gu1=new(n, 2), gu2=new(n, 2), gp=new(n, 2), im=new(n, 4), d=new(n, 2),
                     ad1=new(n), au1=new(n * nsh), b1=new(n), rc1=new(n), ad2=new(n),
                     au2=new(n * nsh), b2=new(n), rc2=new(n), adp=new(n), aup=new(max(nad, 1)),
                     bp=new(n), rcp=new(n))
    return st


def _run_cells(st):
    m, o = st["m"], st["out"]
    cells.gradient(m, 1, 1, st["u1"], o["gu1"])
    cells.gradient(m, 1, 2, st["u2"], o["gu2"])
    o["gp"].copy_(st["gp0"])                     # extrapolates with the last gradient
    cells.gradient(m, 2, 3, st["p"], o["gp"])
    for comp, u, own, oth in ((1, "u1", "gu1", "gu2"), (2, "u2", "gu2", "gu1")):
        cells.momentum(m, comp, 1, st[u], st["p"], st["w"], o[own], o[oth], o["gp"], 1e10,
                       st["ia4"], st["ja4"], 4, o["ad%d" % comp], o["au%d" % comp],
                       o["b%d" % comp], o["im"], o["d"], o["rc%d" % comp])
    cells.pressure_correction(m, st["w"], o["d"], st["p"], o["gp"], st["ia1"], st["ja1"], 1,
                              o["adp"], o["aup"], o["bp"], o["rcp"])
    return o


def _prepare_simple(case, seed):
    c = _cavity(case["nx"], case["kind"], case["gas"])
    opts = cells.simple_opts(tol_u=case["tol"], tol_pc=case["tol"])
    loop = cells.SimpleLoop(c["coor"], c["ix"], c["nelcon"], c["num"], c["pedge"], c["sedge"],
                            c["e"], opts)
    w, p = _flow(c, seed)
    start = dict(w=w, w0=w, p=p)
    if case["gas"]:
        loop.enable_energy(c["pedgeE"], c["sedgeE"], c["gravity"], c["t0"])
        s = loop.get_state(energy=True)
        en = s["en"] + 0.2 * cases.AIR[3] * np.random.default_rng(seed + 3).uniform(-1, 1, p.size)
        start.update(en=en, en0=en, ro=s["ro"])
    loop.use_graph(True)
    return dict(loop=loop, nit=case["nit"], gas=case["gas"], start=start)


def _run_simple(st):
    loop = st["loop"]
    loop.set_state(st["start"])
    res, _ = loop.iterate_energy(st["nit"]) if st["gas"] else loop.iterate(st["nit"])
    w, p = loop.fields()
    out = dict(w=w, p=p, residuals=res)
    if st["gas"]:
        out["temperature"], out["enthalpy"], out["density"] = loop.energy_fields()
    return out


_PREPARE = dict(dropin=_prepare_dropin, spmv=_prepare_spmv, solve=_prepare_solve,
                batched=_prepare_batched, adjoint=_prepare_adjoint, cells=_prepare_cells,
                simple=_prepare_simple)
_RUN = dict(dropin=_run_dropin, spmv=_run_spmv, solve=_run_solve, batched=_run_batched,
            adjoint=_run_adjoint, cells=_run_cells, simple=_run_simple)


def prepare(case, seed):
    return dict(_PREPARE[case["op"]](case, seed), op=case["op"])


def run(state):
    return _RUN[state["op"]](state)


# ---- what a pass cannot do without -----------------------------------------

def _cells_of(nx, ny, kind):
    """Cells and directed neighbour links of a mesh (mixed: half the quads cut)."""
    q = nx * ny
    cell = {"quad": q, "tri": 2 * q, "mixed": 1.5 * q}[kind]
    sides = {"quad": 4 * q, "tri": 6 * q, "mixed": 5 * q}[kind]
    return cell, sides - 2 * (nx + ny)


def work(case):
    op = case["op"]
    if op == "batched":
        sizes = [_cells_of(nx, nx + 1, case["kind"]) for nx in _batch_sides(case)]
        n, nnz = (sum(v) for v in zip(*sizes))
    else:
        n, nnz = _cells_of(case["nx"], case.get("ny", case["nx"]), case["kind"])
    if op == "spmv":
        v = 4 if case["mode"] == "f32" else 8     # values, columns, diagonal, x, y
        return dict(bytes=nnz * (v + 4) + n * (3 * v + 4), flops=2 * (n + nnz))
    if op in ("dropin", "solve", "batched"):
        # the matrix, its structure, b, the guess and x once; the iterations
        # between are the method's own
        return dict(bytes=nnz * 12 + n * 36, flops=2 * (n + nnz))
    if op == "adjoint":
        # forward and adjoint solve, and the three gradients
        return dict(bytes=2 * (nnz * 12 + n * 28) + nnz * 24 + n * 40, flops=6 * (n + nnz))
    if op == "cells":
        # mesh (nodes, links, numbers, codes), fields in; gradients, two
        # momentum systems, the p' system and their cell values out
        return dict(bytes=n * (16 + 20 + 16 + 4 + 20 + 56) + n * (48 + 96 + 64 + 24) + nnz * 12,
                    flops=900 * n)
    # the saved state in, the fields out, per outer iteration the three systems
    # written and read once
    return dict(bytes=n * 80 + case["nit"] * 2 * (3 * (n * 16 + nnz * 8)),
                flops=case["nit"] * 1500 * n)


def exact(case, seed):
    op = case["op"]
    if op in ("dropin", "solve"):
        return _linear(case, seed)["x"]
    if op == "spmv":
        if case["mode"] == "f32":
            x = _linear(dict(case, system="pressure"), seed)["x"]
            x = x.astype(np.float32).astype(np.float64)
            s = _exact_product(case, x)
            return s
        return _linear(dict(case, system="pressure"), seed)["b"]
    if op == "batched":
        return _batch(case, seed)[3]
    if op == "adjoint":
        s, lam, _ = _adjoint(case, seed)
        nad = s["nad"]
        return [s["x"], -lam * s["x"], -lam[s["rows"]][:nad] * s["x"][s["cols"]][:nad], lam]
    return None                                   # cells and loops: no closed form


def _exact_product(case, x):
    ad, au, _, _, _, rows, cols, _ = _pressure(case["nx"], case["ny"], case["kind"],
                                               case["matriz"])
    return ad * x + np.bincount(rows, weights=au[: rows.size] * x[cols], minlength=x.size)
