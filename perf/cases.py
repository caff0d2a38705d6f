"""Performance cases: the work a user of this framework has it do, through its public entry points.

Three families, after the three ways the framework is used.

``matrix``    the stand-alone solver functions of the C-ABI on device arrays (what the shadow
              functions of the MEX gateway call with gpuArray arguments): residual, symmetric
              natural-order Gauss-Seidel, DILU factor and application, the smoother loop
              ``cfdSolveAlgebraicSystem``, and one agglomeration level with its Galerkin product.
``plain``     one steady case on the reference's own algorithm in FP64 (``ufvm.GpuCase``): a
              run restarted from a checkpoint (U, p, mdot set from host arrays), continued for a
              few SIMPLE iterations and read back.
``service``   the batched steady-case service: ``requests`` takes a group of cases from submission
              through admission, AMG hierarchy builds and SIMPLE iterations to their read-back and
              release; ``ticks`` continues a batch that is already resident for a few SIMPLE
              iterations and reads its fields.

Sizes are those of the named workloads (the 20 x 20 and 64^3 cavities, the 6-tet channel, the
2D-cavity sweep of mesh edges 16..256, the serving mix) and of the solver tests, or lie between
them. Systems of the matrix family are finite-volume matrices: a face couples two cells, face
conductances vary by cell spacing and a random factor, the diagonal is the sum of the row's
off-diagonals over an under-relaxation factor.
"""
from __future__ import annotations

import ctypes as ct
import dataclasses
import functools
import math

import numpy as np
import torch

from matlab_ufvm_b200 import case as fv
from matlab_ufvm_b200 import meshgen, ufvm

MATRIX_OPS = ("residual", "sor", "ilu", "solve", "agglomerate")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # r = b - A x on a million-cell grid: what a solver loop written in MATLAB calls most
        dict(name="residual_1M", family="matrix", op="residual", grid="hex", nx=100, ny=100, nz=100),
        # one Gauss-Seidel sweep on the U or p matrix of a fine 2D case (long dependency chain)
        dict(name="sor_2d_62k", family="matrix", op="sor", grid="hex", nx=250, ny=250, nz=1),
        # DILU factor and one application on an unstructured 3D matrix
        dict(name="ilu_tet_136k", family="matrix", op="ilu", grid="tet", nx=70, ny=18, nz=18),
        # the smoother loop on a medium 2D matrix, as cfdSolveEquation('U') runs it
        dict(name="solve_ilu_16k", family="matrix", op="solve", grid="hex", nx=127, ny=129, nz=1, smoother="ILU"),
        # one agglomeration level and its Galerkin product on the 64^3 grid
        dict(name="agglomerate_262k", family="matrix", op="agglomerate", grid="hex", nx=64, ny=64, nz=64),
        # the tutorial-size case: five SIMPLE iterations of the 20 x 20 cavity, Gauss-Seidel V-cycles
        dict(name="plain_cavity_20", family="plain", mesh="cavity2d", nx=20, ny=0, nz=0, p_smoother="SOR",
             cycle="V-Cycle", iters=5),
        # a medium 2D case with the settings of the cylinder tutorial (W-cycles, DILU)
        dict(name="plain_cavity_97_W", family="plain", mesh="cavity2d", nx=97, ny=0, nz=0, p_smoother="ILU",
             cycle="W-Cycle", iters=1),
        # the large structured case: one SIMPLE iteration of the 64^3 cavity, DILU for p
        dict(name="plain_cavity_64cubed", family="plain", mesh="cavity3d", nx=64, ny=0, nz=0, p_smoother="ILU",
             cycle="V-Cycle", iters=1),
        # the unstructured case: inlet, outlet and walls on jittered tets, multicolour smoothing for p
        dict(name="plain_channel_136k", family="plain", mesh="channel", nx=70, ny=18, nz=18, p_smoother="MCGS",
             cycle="V-Cycle", iters=1),
        # a handful of small requests from submission to read-back
        dict(name="service_small", family="service", flow="requests", count=16, sizes=6, n_min=16, n_max=40,
             cubes=0, cube=0, tets=0, tet=0, iters=40),
        # the serving mix: 2D cavities beside 3D cavities and a tet channel
        dict(name="service_mixed", family="service", flow="requests", count=20, sizes=8, n_min=32, n_max=200,
             cubes=3, cube=33, tets=1, tet=14, iters=12),
        # a resident sweep batch over its whole size range, ten SIMPLE iterations on
        dict(name="service_sweep", family="service", flow="ticks", count=128, sizes=12, n_min=16, n_max=256,
             cubes=0, cube=0, tets=0, tet=0, iters=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(("matrix", "matrix", "plain", "service"))
    if family == "matrix":
        op = rng.choice(MATRIX_OPS)
        c = dict(family="matrix", op=op)
        if rng.random() < 0.35:
            s = rng.uniform(2.0, 17.0)
            c.update(grid="tet", nx=_log(rng, 3.0 * s, 4.2 * s), ny=max(2, round(s)), nz=max(2, round(s * rng.uniform(0.8, 1.1))))
        elif rng.random() < 0.5:
            n = _log(rng, 16, 256)
            c.update(grid="hex", nx=n, ny=max(8, round(n * rng.uniform(0.5, 1.0))), nz=1)
        else:
            n = _log(rng, 8, 100 if op == "residual" else 64)
            c.update(grid="hex", nx=n, ny=max(6, round(n * rng.uniform(0.6, 1.0))), nz=max(5, round(n * rng.uniform(0.6, 1.0))))
        if op == "solve":
            c["smoother"] = rng.choice(("ILU", "SOR", "MCGS"))
        return c
    if family == "plain":
        mesh = rng.choice(("cavity2d", "cavity2d", "cavity3d", "channel"))
        c = dict(family="plain", mesh=mesh, p_smoother=rng.choice(("SOR", "ILU", "MCGS")), cycle="V-Cycle", ny=0, nz=0)
        if mesh == "cavity2d":
            c["nx"] = _log(rng, 16, 160)
            if c["nx"] >= 64:  # the W- and F-cycles need four levels
                c["cycle"] = rng.choice(("V-Cycle", "W-Cycle", "F-Cycle"))
        elif mesh == "cavity3d":
            c["nx"] = _log(rng, 10, 48)
        else:
            s = rng.uniform(3.0, 17.0)
            c.update(nx=max(8, round(3.9 * s)), ny=max(3, round(s)), nz=max(3, round(s * rng.uniform(0.8, 1.1))))
        c["iters"] = rng.randint(1, 3) if mesh == "cavity2d" else 1
        return c
    flow = rng.choice(("requests", "ticks"))
    lo = _log(rng, 16, 64)
    hi = _log(rng, lo + 8, 256)
    c = dict(family="service", flow=flow, count=_log(rng, 2, 48 if hi > 128 else 128), sizes=rng.randint(2, 8), n_min=lo, n_max=hi,
             cubes=rng.choice((0, 0, 1, 2)), cube=rng.randint(12, 36), tets=rng.choice((0, 0, 1)), tet=rng.randint(5, 14),
             iters=rng.randint(4, 16))
    return c


# ------------------------------------------------------------------ topology and meshes (shared by all seeds)
@functools.lru_cache(maxsize=16)
def _topology(grid, nx, ny, nz):
    """Owner / neighbour lists of the interior faces (owner < neighbour, sorted) and a conductance
    per face that reflects the cell spacing."""
    if grid == "tet":
        m = meshgen.channel_tet(nx, ny, nz)
        own, nei = m.owner[:m.n_interior].astype(np.int64), m.neighbour.astype(np.int64)
        return m.n_cells, own, nei, np.ones(own.size)
    c = np.arange(nx * ny * nz, dtype=np.int64).reshape(nz, ny, nx)
    pairs = [(c[:, :, :-1], c[:, :, 1:], ny * nz / nx), (c[:, :-1, :], c[:, 1:, :], nx * nz / ny),
             (c[:-1], c[1:], nx * ny / nz)]
    own = np.concatenate([a.ravel() for a, _, _ in pairs])
    nei = np.concatenate([b.ravel() for _, b, _ in pairs])
    cond = np.concatenate([np.full(a.size, g) for a, _, g in pairs])
    o = np.lexsort((nei, own))
    return nx * ny * nz, own[o], nei[o], cond[o]


@functools.lru_cache(maxsize=16)
def _pattern(grid, nx, ny, nz):
    """cconn-ordered CSR pattern (a row lists its neighbours in face order) and each entry's face."""
    n, own, nei, _ = _topology(grid, nx, ny, nz)
    f = np.arange(own.size, dtype=np.int64)
    row, col, face = np.concatenate([own, nei]), np.concatenate([nei, own]), np.concatenate([f, f])
    o = np.lexsort((face, row))
    rowptr = np.zeros(n + 1, dtype=np.int32)
    rowptr[1:] = np.cumsum(np.bincount(row, minlength=n))
    return rowptr, col[o].astype(np.int32), face[o]


def _system(case, seed):
    """(rowptr, col, ac, anb, bc, dphi) as host arrays."""
    key = (case["grid"], case["nx"], case["ny"], case["nz"])
    n, own, _, cond = _topology(*key)
    rowptr, col, face = _pattern(*key)
    rng = np.random.default_rng([seed, 17])
    g = cond / cond.mean() * rng.uniform(0.4, 1.0, own.size)
    anb = -g[face]
    ac = -np.add.reduceat(anb, rowptr[:-1]) * (1.0 + 0.43 * rng.uniform(0.2, 1.0, n))
    return rowptr, col, ac, anb, rng.normal(size=n), 1e-2 * rng.normal(size=n)


@functools.lru_cache(maxsize=40)
def _base_spec(mesh, nx, ny, nz):
    q = dict(quirks=fv.QUIRKS_CONVERGING)
    if mesh == "cavity2d":
        return fv.cavity_case(nx, **q)
    if mesh == "cavity3d":
        return fv.cavity_case(nx, dim=3, **q)
    return fv.channel_case(nx, ny, nz, **q)


# ------------------------------------------------------------------ what a program has in hand
def _vp(t):
    return ct.c_void_p(t.data_ptr())


def _prepare_matrix(case, seed):
    host = _system(case, seed)
    dev = [torch.from_numpy(a).cuda() for a in host]
    st = dict(case=case, n=len(host[2]), rp=dev[0], col=dev[1], ac=dev[2], anb=dev[3], bc=dev[4], x0=dev[5])
    st["x"] = torch.empty_like(st["x0"])
    if case["op"] == "residual":
        st["r"] = torch.empty_like(st["x0"])
    if case["op"] == "ilu":
        st["dc"] = torch.empty_like(st["x0"])
    if case["op"] == "agglomerate":
        n, nnz = st["n"], st["col"].numel()
        st.update(par=torch.zeros(n, dtype=torch.int32, device="cuda"), crp=torch.zeros(n + 1, dtype=torch.int32, device="cuda"),
                  ccol=torch.zeros(nnz, dtype=torch.int32, device="cuda"),
                  cac=torch.zeros(n, dtype=torch.float64, device="cuda"),
                  canb=torch.zeros(nnz, dtype=torch.float64, device="cuda"))
    return st


def _prepare_plain(case, seed):
    rng = np.random.default_rng([seed, 29])
    base = _base_spec(case["mesh"], case["nx"], case["ny"], case["nz"])
    spec = dataclasses.replace(base, nu=1.0 / rng.uniform(50.0, 500.0), p_smoother=case["p_smoother"],
                               p_cycle=case["cycle"])
    g = ufvm.GpuCase(spec)
    g.cfdRunCase(1)  # the checkpoint: the fields after the first iteration, stirred by a smooth flow
    U, p, mdot = g.get("U"), g.get("p"), g.get("mdot")
    x = g.geometry("centroid_c")
    k = rng.integers(1, 4, size=(3, 3))
    rows = U.size // 3
    for c in range(3 if case["mesh"] != "cavity2d" else 2):
        U[c * rows:c * rows + g.Nc] += rng.uniform(0.02, 0.1) * np.prod(np.sin(math.pi * k[c] * x), axis=1)
    return dict(case=case, g=g, U=U, p=p, mdot=mdot)


def _service_specs(case, seed):
    rng = np.random.default_rng([seed, 31])
    s = max(case["sizes"], 1)
    edges = [int(round(math.exp(math.log(case["n_min"]) + (math.log(case["n_max"]) - math.log(case["n_min"])) * (i + 0.5) / s)))
             for i in range(s)]
    bases = [_base_spec("cavity2d", edges[i % s], 0, 0) for i in range(case["count"])]
    bases += [_base_spec("cavity3d", case["cube"], 0, 0) for _ in range(case["cubes"])]
    bases += [_base_spec("channel", 4 * case["tet"], case["tet"], case["tet"]) for _ in range(case["tets"])]
    return [dataclasses.replace(b, nu=1.0 / rng.uniform(50.0, 1000.0)) for b in bases]


def _prepare_service(case, seed):
    specs = _service_specs(case, seed)
    settings = ufvm.fast_settings(specs[0])
    st = dict(case=case, specs=specs)
    if case["flow"] == "ticks":
        settings.tol_u = settings.tol_p = 0.0  # a fixed number of iterations, no convergence stop
    svc = st["svc"] = ufvm.Service(settings, max_resident_cells=8_000_000)
    svc.set_schedule(4096)  # a program that serves one kind of load keeps its schedule
    # the host buffers that results are read into: U (3 components) and p over cells, boundary rows
    # and, behind an outlet, face-indexed rows
    rows = sum(s.mesh.n_cells + s.mesh.n_faces for s in specs)
    st["host"] = torch.zeros(4 * rows, dtype=torch.float64, pin_memory=True)
    if case["flow"] == "ticks":
        st["tickets"] = [svc.submit(s, 1_000_000) for s in specs]
        svc.admit()
        for _ in range(20):  # hierarchies built, the tick captured, the first transient over
            svc.step()
    return st


def prepare(case, seed):
    if case["family"] == "matrix":
        return _prepare_matrix(case, seed)
    if case["family"] == "plain":
        return _prepare_plain(case, seed)
    return _prepare_service(case, seed)


# ------------------------------------------------------------------ one pass
def _ok(code):
    if code != 0:
        raise ufvm.UfvmError(code, ufvm.lib().ufvm_last_error().decode())


def _run_matrix(st):
    L, op, n = ufvm.lib(), st["case"]["op"], st["n"]
    stream = ct.c_void_p(torch.cuda.current_stream().cuda_stream)
    rp, col, ac, anb, bc = (_vp(st[k]) for k in ("rp", "col", "ac", "anb", "bc"))
    if op == "residual":
        _ok(L.ufvm_compute_residuals_array(n, rp, col, ac, anb, bc, _vp(st["x0"]), _vp(st["r"]), stream))
        return {"r": st["r"]}
    if op == "agglomerate":
        nc, nnz = ct.c_int32(), ct.c_int32()
        _ok(L.ufvm_agglomerate_level(n, rp, col, ac, anb, _vp(st["par"]), _vp(st["crp"]), _vp(st["ccol"]), _vp(st["cac"]),
                                     _vp(st["canb"]), ct.byref(nc), ct.byref(nnz), stream))
        # the buffers at their capacity, as a caller holds them; the counts say how much is in use
        return {"parents": st["par"], "rowptr": st["crp"], "col": st["ccol"], "ac": st["cac"], "anb": st["canb"],
                "n_coarse": nc.value, "nnz_coarse": nnz.value}
    st["x"].copy_(st["x0"])
    x = _vp(st["x"])
    if op == "sor":
        _ok(L.ufvm_solve_sor(n, rp, col, ac, anb, bc, x, stream))
        return {"x": st["x"]}
    if op == "ilu":
        _ok(L.ufvm_factorize_ilu(n, rp, col, ac, anb, _vp(st["dc"]), fv.QUIRKS_CONVERGING, stream))
        _ok(L.ufvm_solve_ilu(n, rp, col, ac, anb, bc, _vp(st["dc"]), x, stream))
        return {"dc": st["dc"], "x": st["x"]}
    r0, r1, it = ct.c_double(), ct.c_double(), ct.c_int32()
    _ok(L.ufvm_solve_algebraic_system(n, rp, col, ac, anb, bc, x, fv.SMOOTHER[st["case"]["smoother"]], 10, 0.1,
                                      fv.QUIRKS_CONVERGING, ct.byref(r0), ct.byref(r1), ct.byref(it), stream))
    return {"x": st["x"], "r0": r0.value, "r1": r1.value, "iterations": it.value}


def _run_plain(st):
    g = st["g"]
    g.set("U", st["U"])
    g.set("p", st["p"])
    g.set("mdot", st["mdot"])
    it, res = g.cfdRunCase(st["case"]["iters"])
    return {"U": g.get("U"), "p": g.get("p"), "mdot": g.get("mdot"), "res": res, "iterations": it}


def _read(st, tickets):
    """Every case's U, then p, into the program's pinned buffer, one after another."""
    L, svc, host, off, n = ufvm.lib(), st["svc"], st["host"], 0, ct.c_int64()
    base = host.data_ptr()
    for name in (b"U", b"p"):
        for t in tickets:
            _ok(L.ufvm_service_get_field(svc.h, t, name, ct.cast(base + 8 * off, ufvm.D), host.numel() - off, ct.byref(n)))
            off += n.value
    status = [svc.status(t) for t in tickets]
    return {"fields": host, "res": np.array([s["res"] for s in status]),
            "iterations": np.array([s["iterations"] for s in status])}


def _run_service(st):
    svc, case = st["svc"], st["case"]
    if case["flow"] == "ticks":
        for _ in range(case["iters"]):
            svc.step()
        return _read(st, st["tickets"])
    tickets = [svc.submit(s, case["iters"]) for s in st["specs"]]
    svc.run()
    svc.poll()
    out = _read(st, tickets)
    for t in tickets:
        svc.release(t)
    return out


def run(state):
    family = state["case"]["family"]
    if family == "matrix":
        return _run_matrix(state)
    return _run_plain(state) if family == "plain" else _run_service(state)


# ------------------------------------------------------------------ what a pass cannot do without
def _iteration_work(spec):
    """One SIMPLE iteration: the mesh read once, the fields and gradients read and written once, and
    for each of the five equations (three U, two p) its matrix written, read by one solve and the
    correction added."""
    m = spec.mesh
    n, f, fi = m.n_cells, m.n_faces, m.n_interior
    rows, nnz = n + f - fi, 2 * fi
    mesh = 8 * 19 * f + 4 * (f + fi) + 8 * n
    fields = 8 * (2 * (3 + 1) * rows + 2 * 12 * rows + 2 * f)
    eq = 2 * 5 * (16 * n + 8 * nnz) + 5 * (4 * n + 4 * nnz + 24 * n)
    return {"bytes": float(mesh + fields + eq), "flops": float(400 * fi + 60 * (f - fi) + 5 * (4 * nnz + 20 * n))}


def work(case):
    if case["family"] == "matrix":
        n, own, _, _ = _topology(case["grid"], case["nx"], case["ny"], case["nz"])
        nnz, op = 2 * own.size, case["op"]
        matrix = 4 * (n + 1) + 12 * nnz + 8 * n  # pattern, off-diagonals, diagonal
        if op == "residual":
            return {"bytes": matrix + 24.0 * n, "flops": 2.0 * (nnz + n)}
        if op == "sor":
            return {"bytes": matrix + 24.0 * n, "flops": 4.0 * (nnz + n)}
        if op == "ilu":
            return {"bytes": 2.0 * matrix + 40.0 * n, "flops": 7.0 * nnz + 6.0 * n}
        if op == "solve":
            return {"bytes": matrix + 24.0 * n, "flops": 8.0 * (nnz + n)}
        return {"bytes": matrix + 4.0 * n + 0.3 * matrix, "flops": 4.0 * nnz}
    if case["family"] == "plain":
        w = _iteration_work(_base_spec(case["mesh"], case["nx"], case["ny"], case["nz"]))
        return {k: v * case["iters"] for k, v in w.items()}
    out = {"bytes": 0.0, "flops": 0.0}
    for s in _service_specs(case, 0):
        for k, v in _iteration_work(s).items():
            out[k] += v * case["iters"]
    return out


# ------------------------------------------------------------------ results in 64 bits, by plain loops
def _gs_row(i, x, rp, col, ac, anb, bc):
    v = bc[i]
    for k in range(rp[i], rp[i + 1]):
        v -= anb[k] * x[col[k]]
    x[i] = v / ac[i]


def _sor(x, n, *a):
    for i in range(n):
        _gs_row(i, x, *a)
    for i in range(n - 1, -1, -1):
        _gs_row(i, x, *a)


def _residual(x, rp, col, ac, anb, bc):
    r = bc - ac * x
    return r - np.add.reduceat(anb * x[col], rp[:-1])


def _dilu_factor(n, rp, col, ac, anb, skip):
    """1 / d_i with d_i = ac_i - sum over lower j of a_ij a_ji / d_j; `skip`: the reference's loop
    leaves out the contributions of its row N - 1."""
    a = [dict(zip(col[rp[i]:rp[i + 1]], anb[rp[i]:rp[i + 1]])) for i in range(n)]
    dc = [0.0] * n
    for i in range(n):
        d = ac[i]
        for j in sorted(j for j in a[i] if j < i):
            if not (skip and j == n - 2):
                d -= a[i][j] * dc[j] * a[j][i]
        dc[i] = 1.0 / d
    return dc, a


def _dilu_apply(n, r, dc, a):
    r = list(r)
    for i in range(n):
        v = r[i]
        for j in sorted(j for j in a[i] if j < i):
            v -= a[i][j] * (dc[j] * r[j])
        r[i] = v
    for i in range(n - 1, -1, -1):
        v = r[i]
        if i < n - 1:
            for j, w in a[i].items():
                if j > i:
                    v -= w * r[j]
        r[i] = dc[i] * v
    return np.array(r)


def exact(case, seed):
    if case["family"] != "matrix" or case["op"] == "agglomerate":
        return None  # whole solvers and the seed agglomeration have no value without their own loops
    rp, col, ac, anb, bc, x0 = _system(case, seed)
    n, op = len(ac), case["op"]
    if op == "residual":
        return {"r": _residual(x0, rp, col, ac, anb, bc)}
    if n > 300_000:
        return None
    lists = tuple(v.tolist() for v in (rp, col, ac, anb, bc))
    if op == "sor":
        x = x0.tolist()
        _sor(x, n, *lists)
        return {"x": np.array(x)}
    skip = bool(fv.QUIRKS_CONVERGING & fv.Q7_ILU_SKIP_ROW)
    if op == "ilu":
        dc, a = _dilu_factor(n, *lists[:4], skip)
        return {"dc": np.array(dc), "x": x0 + _dilu_apply(n, _residual(x0, rp, col, ac, anb, bc), dc, a)}
    if case["smoother"] == "MCGS" or n > 70_000:
        return None
    x, it = x0.copy(), 0
    r0 = r1 = float(np.abs(_residual(x, rp, col, ac, anb, bc)).sum()) / n
    if case["smoother"] == "ILU":
        dc, a = _dilu_factor(n, *lists[:4], skip)
    while it < 10 and r1 > 0.1 * r0:
        if case["smoother"] == "ILU":
            x = x + _dilu_apply(n, _residual(x, rp, col, ac, anb, bc), dc, a)
        else:
            y = x.tolist()
            _sor(y, n, *lists)
            x = np.array(y)
        r1 = float(np.abs(_residual(x, rp, col, ac, anb, bc)).sum()) / n
        it += 1
    return {"x": x, "r0": r0, "r1": r1, "iterations": it}
