"""Performance cases: the work a program gives this package, by entry point.

A case is a dict of plain values; `path` names the entry point:

  steady     ThermalModelA: init(), conductivity and source from host arrays,
             advance() to an outer residual ratio of 1e-10, temperature back
  transient  the same model with backward-Euler steps and updateTime()
  batch      BatchedThermal.solve(): independent quad meshes as one system
  csr        solve_csr() of AMG / CG / BCGStab on a host CSR system
  residual   fvm_csr_residual_device_noalloc() on device buffers
  train      LearnedCorrection.train() on harvested residual / error pairs

`solver` is one of the settings the package is run with: `default` (the
model's own default AMG), `plain` (FP64 AMG V(1,1), coarsest level of at most
100 rows smoothed), `plain_cg` (CG under it), `bcgstab` (BiCGStab under the
default AMG) and `mixed` (flexible CG under the FP32 cycle on the GPU-built
hierarchy, with Anderson mixing of depth 2 on tet meshes).
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from fvm_b200 import _lib, batch, fvmbaseExt, learned, meshgen, models

OUTER = 1e-10  # outer residual ratio of every thermal solve
MAX_OUTER = 500
DT = 1e-3


# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # the smallest whole solve: a first try of a model, a unit test, one
        # inner solve of a coupled program; latency and launches
        {"name": "quad24_default", "path": "steady", "mesh": "quad", "n": 24, "ny": 24, "solver": "default",
         "field": "lognormal", "bc": "fixed"},
        # 2D steady conduction with the reference's solver as it stands
        {"name": "quad256_plain", "path": "steady", "mesh": "quad", "n": 256, "ny": 256, "solver": "plain",
         "field": "lognormal", "bc": "fixed"},
        # an ordinary 3D part with the FP64 Krylov solver
        {"name": "tet24_cg", "path": "steady", "mesh": "tet", "n": 24, "solver": "plain_cg", "field": "smooth",
         "bc": "fixed"},
        # the same part with the mixed solver
        {"name": "tet24_mixed", "path": "steady", "mesh": "tet", "n": 24, "solver": "mixed", "field": "smooth",
         "bc": "fixed"},
        # the headline workload: 1.5M tets, conductivity contrast 1e3
        {"name": "tet64_mixed", "path": "steady", "mesh": "tet", "n": 64, "solver": "mixed", "field": "smooth",
         "bc": "fixed"},
        # two-phase material on a large structured mesh
        {"name": "hex100_two_phase", "path": "steady", "mesh": "hex", "n": 100, "solver": "mixed",
         "field": "two_phase", "bc": "fixed"},
        # radiative and mixed boundaries: the matrix and its hierarchy follow
        # the temperature and are rebuilt in every outer iteration
        {"name": "tet20_radiative", "path": "steady", "mesh": "tet", "n": 20, "solver": "mixed", "field": "smooth",
         "bc": "radiative"},
        # implicit time stepping
        {"name": "hex90_transient", "path": "transient", "mesh": "hex", "n": 90, "solver": "mixed",
         "field": "lognormal", "steps": 5},
        # a parameter study: uneven independent meshes in one solve
        {"name": "batch24_mixed", "path": "batch", "count": 24, "lo": 32, "hi": 256, "solver": "mixed"},
        # the linear solver alone on a system assembled elsewhere
        {"name": "csr_211x190", "path": "csr", "n": 211, "ny": 190, "solver": "bcgstab"},
        # a residual check inside a program that owns its device memory
        {"name": "residual_3m", "path": "residual", "n": 3_000_017},
        # training the learned correction
        {"name": "train_tet18", "path": "train", "n": 18, "steps": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["steady"] * 6 + ["transient", "batch", "csr", "csr", "residual", "residual", "train"])
    if path == "residual":
        return {"path": path, "n": _log_int(rng, 1000, 3_000_000)}
    if path == "train":
        return {"path": path, "n": rng.randint(8, 18), "steps": rng.randint(5, 20)}
    if path == "csr":
        return {"path": path, "n": _log_int(rng, 24, 210), "ny": _log_int(rng, 24, 190),
                "solver": rng.choice(["default", "plain_cg", "bcgstab"])}
    if path == "batch":
        return {"path": path, "count": rng.randint(4, 24), "lo": 32, "hi": rng.randint(48, 256), "solver": "mixed"}
    if path == "transient":
        return {"path": path, "mesh": "hex", "n": _log_int(rng, 16, 90), "solver": "mixed", "field": "lognormal",
                "steps": rng.randint(2, 5)}
    mesh = rng.choice(["quad", "quad", "tet", "tet", "hex"])
    solver = rng.choice(["default", "plain", "plain_cg", "mixed", "mixed", "mixed"])
    if mesh == "quad":
        c = {"n": _log_int(rng, 20, 256), "ny": _log_int(rng, 20, 256), "field": "lognormal"}
    elif mesh == "tet":
        c = {"n": _log_int(rng, 8, 40 if solver == "mixed" else 24), "field": "smooth"}
    else:
        c = {"n": _log_int(rng, 12, 80 if solver == "mixed" else 40), "field": rng.choice(["two_phase", "lognormal"])}
    radiative = mesh != "quad" and c["n"] <= 24 and solver == "mixed" and rng.random() < 0.4
    return dict({"path": path, "mesh": mesh, "solver": solver, "bc": "radiative" if radiative else "fixed"}, **c)


# ---------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=4)
def _topology(mesh, n):
    """Mesh arrays without jitter and their cell centres: they do not depend
    on the seed, and building them takes longer than the solve."""
    d = meshgen.tet_mesh(n, jitter=0.0) if mesh == "tet" else meshgen.hex_mesh(n)
    return d, meshgen.cell_centers(d)


def _mesh(case, seed):
    if case["mesh"] == "quad":
        d = meshgen.quad_mesh(case["n"], jitter=0.2, seed=seed, ny=case["ny"])
        return d, None
    d, pts = _topology(case["mesh"], case["n"])
    if case["mesh"] == "hex":
        return d, pts
    # interior nodes moved by up to 15 % of the lattice spacing
    h = 1.0 / (case["n"] - 1)
    x = d["nodes"]
    inside = np.all((x > 0.5 * h) & (x < 1.0 - 0.5 * h), axis=1)
    rng = np.random.default_rng(seed)
    nodes = x.copy()
    nodes[inside] += rng.uniform(-0.15 * h, 0.15 * h, size=(int(inside.sum()), 3))
    return dict(d, nodes=nodes), pts


def _wave(pts, seed, scale):
    """A smooth random field in [-1, 1]: 24 plane waves of random directions
    with wave numbers up to `scale`."""
    rng = np.random.default_rng(seed)
    kv = rng.normal(size=(24, 3)) * scale
    ph = rng.uniform(0, 2 * np.pi, 24)
    p = torch.from_numpy(pts)
    if torch.cuda.is_available():
        p = p.cuda()
    g = torch.zeros(len(pts), dtype=torch.float64, device=p.device)
    for j in range(24):
        g += torch.cos(p @ torch.from_numpy(kv[j]).to(p) + ph[j])
    g = (g - g.min()) / (g.max() - g.min()) * 2.0 - 1.0
    return g.cpu().numpy()


def _fields(case, pts, n, seed):
    rng = np.random.default_rng(seed + 200)
    s = rng.uniform(0.0, 1.0, n)
    kind = case["field"]
    if kind == "lognormal":
        k = rng.lognormal(0.0, 1.0, n)
    elif kind == "smooth":
        k = 10.0 ** (1.5 * _wave(pts, seed + 100, 12.0))
    else:  # 30 % of the cells conduct a hundred times better
        g = _wave(pts, seed + 100, 20.0)
        k = np.where(g > np.quantile(g, 0.7), 100.0, 1.0)
    return k, s


def _bcs(case):
    """{group id: (type, {variable: value})}"""
    if case["path"] == "transient":
        return {1: ("SpecifiedHeatFlux", {"specifiedHeatFlux": 0.0}),
                2: ("SpecifiedTemperature", {"specifiedTemperature": 400.0})}
    b = {1: ("SpecifiedTemperature", {"specifiedTemperature": 300.0}),
         2: ("SpecifiedTemperature", {"specifiedTemperature": 400.0})}
    if case.get("bc") == "radiative":
        b[3] = ("Radiative", {"farFieldTemperature": 310.0, "surfaceEmissivity": 0.7})
        b[4] = ("Mixed", {"convectiveCoefficient": 8.0, "farFieldTemperature": 320.0, "surfaceEmissivity": 0.5})
    return b


def _csr_system(case, seed):
    """Five-point diffusion with lognormal cell conductivities and a fixed
    value on one side, in delta form (negative diagonal), rows ascending."""
    nx, ny = case["n"], case["ny"]
    rng = np.random.default_rng(seed)
    k = rng.lognormal(0.0, 1.0, (ny, nx))
    n = nx * ny
    idx = np.arange(n).reshape(ny, nx)
    cx = 2.0 * k[:, :-1] * k[:, 1:] / (k[:, :-1] + k[:, 1:])
    cy = 2.0 * k[:-1] * k[1:] / (k[:-1] + k[1:])
    i = np.concatenate([idx[:, :-1].ravel(), idx[:, 1:].ravel(), idx[:-1].ravel(), idx[1:].ravel()])
    j = np.concatenate([idx[:, 1:].ravel(), idx[:, :-1].ravel(), idx[1:].ravel(), idx[:-1].ravel()])
    v = np.concatenate([cx.ravel(), cx.ravel(), cy.ravel(), cy.ravel()])
    o = np.lexsort((j, i))
    row = np.zeros(n + 1, np.int32)
    row[1:] = np.cumsum(np.bincount(i, minlength=n))
    diag = -np.bincount(i, weights=v, minlength=n)
    diag[idx[:, 0]] -= 2.0 * k[:, 0]
    return row, j[o].astype(np.int32), diag, v[o], rng.standard_normal(n)


def _residual_system(case, seed):
    """A device CSR matrix with 3 to 7 off-diagonals per row at mesh-like
    distances from it."""
    n = case["n"]
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    cnt = torch.randint(3, 8, (n,), generator=g, device=dev)
    row = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    row[1:] = torch.cumsum(cnt, 0)
    nnz = int(row[-1])
    of = torch.repeat_interleave(torch.arange(n, device=dev), cnt)
    band = max(4, int(round(n ** (2.0 / 3.0))))
    col = (of + torch.randint(-band, band + 1, (nnz,), generator=g, device=dev)).clamp_(0, n - 1).to(torch.int32)
    off = torch.rand(nnz, generator=g, device=dev, dtype=torch.float64) + 0.1
    diag = -(torch.rand(n, generator=g, device=dev, dtype=torch.float64) + 4.0)
    x = torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    b = torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    return {"row": row, "col": col, "diag": diag, "off": off, "x": x, "b": b}


def _solver(name, accel=0):
    if name == "default":
        return None  # the model's own
    amg = fvmbaseExt.AMG()
    if name == "bcgstab":
        ks = fvmbaseExt.BCGStab()
        ks.preconditioner = amg
        ks.relativeTolerance = 0.1
        ks.nMaxIterations = 200
        return ks
    inner = 0.05 if accel else 0.1
    amg.nPreSweeps = amg.nPostSweeps = 1
    amg.coarsestSize = 100
    amg.relativeTolerance = inner
    amg.nMaxIterations = 200
    if name == "plain":
        return amg
    if name == "mixed":
        amg.setupOnDevice = True
        amg.precision = fvmbaseExt.AMG.MIXED
        amg.coarseSolver = fvmbaseExt.AMG.COARSE_DIRECT
        amg.coarsestSize = 4096
        amg.coarseJacobiRows = 1 << 30
        amg.nPreSweeps, amg.nPostSweeps = 0, 2
        amg.matchPasses = 2
        amg.matchBeta = 0.5
        amg.coarsePostSweeps = 1
        amg.outerAcceleration = accel
    cg = fvmbaseExt.CG()
    cg.preconditioner = amg
    cg.relativeTolerance = inner
    cg.nMaxIterations = 200
    return cg


def _model(case, mesh_dict):
    m = fvmbaseExt.Mesh.from_dict(mesh_dict)
    tf = models.ThermalFields("therm")
    tm = models.ThermalModelA(models.GeomFields("geom"), tf, [m])
    for gid, (kind, vals) in _bcs(case).items():
        bc = tm.getBCMap()[gid]
        bc.bcType = kind
        for name, v in vals.items():
            bc.setVar(name, v)
    o = tm.getOptions()
    o.relativeTolerance = OUTER
    # mixing pays where the outer iteration carries a non-orthogonal correction
    accel = 2 if case["solver"] == "mixed" and case.get("mesh") == "tet" and case.get("bc") == "fixed" else 0
    ls = _solver(case["solver"], accel)
    if ls is not None:
        o.linearSolver = ls
    return m, tf, tm


def _batch_meshes(case, seed):
    # the sizes are the case's own, so that every seed has the same shapes
    sides = np.random.default_rng(1000 * case["count"] + case["hi"]).integers(case["lo"], case["hi"] + 1, case["count"])
    sides[0], sides[-1] = case["lo"], case["hi"]
    out = []
    for i, n in enumerate(sides):
        mesh = meshgen.quad_mesh(int(n), jitter=0.2, seed=seed + i)
        rng = np.random.default_rng(seed + 1000 + i)
        out.append((mesh, rng.lognormal(0.0, 1.0, mesh["nCells"]), rng.uniform(0.0, 1.0, mesh["nCells"])))
    return out


def prepare(case, seed):
    path = case["path"]
    st = {"case": case}
    if path == "residual":
        st.update(_residual_system(case, seed))
        st["r"] = torch.empty_like(st["x"])
        st["norm"] = torch.empty(1, dtype=torch.float64, device="cuda")
        st["lib"] = _lib.load()
        return st
    if path == "csr":
        st["system"] = _csr_system(case, seed)
        ls = _solver(case["solver"])
        if ls is None:
            ls = fvmbaseExt.AMG()
        ls.relativeTolerance = 1e-12
        ls.nMaxIterations = 500
        st["solver"] = ls
        return st
    if path == "batch":
        ms = _batch_meshes(case, seed)
        st["k"] = [k for _, k, _ in ms]
        st["s"] = [s for _, _, s in ms]
        st["batch"] = batch.BatchedThermal([m for m, _, _ in ms], {1: ("T", 300.0), 2: ("T", 400.0)},
                                           _solver(case["solver"]), relative_tolerance=OUTER)
        return st
    if path == "train":
        c = {"path": "steady", "mesh": "tet", "n": case["n"], "solver": "plain", "field": "smooth", "bc": "fixed"}
        d, pts = _mesh(c, seed)
        k, s = _fields(c, pts, d["nCells"], seed)
        m, tf, tm = _model(c, d)
        tm.init()
        tf.conductivity[m.getCells()] = k
        tf.source[m.getCells()] = s
        lc = learned.LearnedCorrection(seed=seed)
        lc.setObjective(learned.LearnedCorrection.RESIDUAL)
        lc.harvest(tm, nOuter=2, perSolve=3, relativeTolerance=1e-8, maxCycles=100)
        st["lc"], st["p0"] = lc, lc.getParams()
        return st
    d, pts = _mesh(case, seed)
    st["k"], st["s"] = _fields(case, pts, d["nCells"], seed)
    st["mesh"], st["tf"], st["tm"] = _model(case, d)
    if path == "transient":
        st["rc"] = np.random.default_rng(seed + 300).uniform(0.5, 2.0, d["nCells"])
        st["s"] = np.zeros(d["nCells"])
        o = st["tm"].getOptions()
        o.transient = True
        o["timeStep"] = DT
    return st


def run(st):
    case = st["case"]
    path = case["path"]
    if path == "residual":
        p = [ctypes.c_void_p(st[q].data_ptr()) for q in ("row", "col", "diag", "off", "x", "b", "r", "norm")]
        rc = st["lib"].fvm_csr_residual_device_noalloc(case["n"], *p,
                                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(st["lib"].fvm_last_error().decode())
        return st["r"], st["norm"]
    if path == "csr":
        x, _ = st["solver"].solve_csr(*st["system"])
        return x
    if path == "batch":
        t, rep = st["batch"].solve(st["k"], st["s"])
        return t
    if path == "train":
        st["lc"].setParams(st["p0"])
        st["lc"].train(case["steps"], lr=1e-3, seed=0)
        return st["lc"].getParams()
    cells = st["mesh"].getCells()
    tf, tm = st["tf"], st["tm"]
    tm.init()
    tf.conductivity[cells] = st["k"]
    tf.source[cells] = st["s"]
    if path == "transient":
        tf.specificHeat[cells] = st["rc"]
        for _ in range(case["steps"]):
            tm.advance(MAX_OUTER)
            tm.updateTime()
    else:
        tm.advance(MAX_OUTER)
    return tf.temperature[cells]


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _cells(case):
    """(cells, faces, dimension) of a case's mesh, about."""
    if case["path"] == "batch":
        rng = [case["lo"] + (case["hi"] - case["lo"]) * (i + 0.5) / case["count"] for i in range(case["count"])]
        n = int(sum(v * v for v in rng))
        return n, 2 * n + 4 * sum(int(v) for v in rng) // 2, 2
    n = case["n"]
    if case["path"] == "train" or case["mesh"] == "tet":
        c = 6 * (n - 1) ** 3
        return c, 2 * c + 6 * (n - 1) ** 2, 3
    if case["mesh"] == "quad":
        return n * case["ny"], 2 * n * case["ny"] + n + case["ny"], 2
    return n ** 3, 3 * n ** 3 + 3 * n ** 2, 3


def work(case):
    path = case["path"]
    if path == "residual":
        n, nnz = case["n"], 5 * case["n"]
        return {"bytes": 12.0 * nnz + (4 + 8 * 4) * n, "flops": 2.0 * nnz + 3.0 * n}
    if path == "csr":
        n = case["n"] * case["ny"]
        nnz = 4 * n
        return {"bytes": 12.0 * nnz + (4 + 8 * 3) * n, "flops": 2.0 * nnz + 2.0 * n}
    n, f, _ = _cells(case)
    if path == "train":
        # a step: forward and backward through three 64 -> 32 layers
        return {"bytes": case["steps"] * (16.0 * n + 24.0 * f), "flops": case["steps"] * 3 * 3 * 2.0 * 64 * 32 * n}
    # mesh and metrics read once, fields in, temperature out
    steps = case.get("steps", 1)
    per = f * (8 + 24 + 8) + n * (24 + 8 + 8 + 8 + 8)
    return {"bytes": float(steps * per), "flops": float(steps * (20 * f + 10 * n))}


# ---------------------------------------------------------------------------
# the same values in plain torch, 64 bits


def _geometry(d, dev):
    """Face areas, cell centroids and volumes of a mesh (the finite-volume
    scheme's own definitions), and its least-squares gradient operator."""
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    dim, n = d["dim"], d["nCells"]
    x = t(d["nodes"])
    fn = t(d["faceNodes"]).long().reshape(len(d["faceNodeCount"]), -1)
    fc = t(d["faceCells"]).long().reshape(-1, 2)
    c0, c1 = fc[:, 0], fc[:, 1]
    n_all = n + int(d["faceGroupSize"][1:].sum())
    p = x[fn]
    cross = lambda a, b: torch.linalg.cross(a, b, dim=1)  # noqa: E731
    if fn.shape[1] == 2:
        dr = p[:, 1] - p[:, 0]
        area = torch.stack([dr[:, 1], -dr[:, 0], torch.zeros_like(dr[:, 0])], 1)
    elif fn.shape[1] == 3:
        area = 0.5 * cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    else:
        area = 0.5 * cross(p[:, 2] - p[:, 0], p[:, 3] - p[:, 1])
    am = area.norm(dim=1)
    cen = p.mean(1)
    if fn.shape[1] > 3:
        en = area / am[:, None]
        num, den = torch.zeros_like(cen), torch.zeros_like(am)
        for q in range(fn.shape[1]):
            a, b = p[:, q], p[:, (q + 1) % fn.shape[1]]
            w = (0.5 * cross(a - cen, b - cen) * en).sum(1)
            num += (2.0 / 3.0) * (0.5 * (a + b) - cen) * w[:, None]
            den += w
        cen = cen + num / den[:, None]
    cc = torch.zeros(n_all, 3, dtype=torch.float64, device=dev)
    wt = torch.zeros(n_all, dtype=torch.float64, device=dev)
    for c in (c0, c1):
        cc.index_add_(0, c, cen * am[:, None])
        wt.index_add_(0, c, am)
    cc = cc / wt[:, None]
    ni = int(d["faceGroupSize"][0])
    cc[c1[ni:]] = cen[ni:]
    vol = torch.zeros(n_all, dtype=torch.float64, device=dev)
    vol.index_add_(0, c0, ((cen - cc[c0]) * area).sum(1) / dim)
    vol.index_add_(0, c1, -((cen - cc[c1]) * area).sum(1) / dim)
    vol[c1[ni:]] = vol[c0[ni:]]
    ds = cc[c1] - cc[c0]
    m = ds.norm(dim=1)
    e = ds[:, :dim] / m[:, None]
    outer = torch.zeros(n_all, dim, dim, dtype=torch.float64, device=dev)
    for c in (c0, c1):
        outer.index_add_(0, c, e[:, :, None] * e[:, None, :])
    inv = torch.zeros_like(outer)
    inv[:n] = torch.linalg.inv(outer[:n])
    return {"n": n, "n_all": n_all, "ni": ni, "c0": c0, "c1": c1, "area": area, "am": am, "vol": vol, "ds": ds,
            "m": m, "e": e, "inv": inv, "dim": dim}


def _pcg(mul, diag, b, tol, limit):
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = torch.dot(r, z)
    r0 = float(r.norm())
    for it in range(limit):
        q = mul(p)
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if it % 16 == 15 and float(r.norm()) <= tol * r0:
            break
        z = r / diag
        rn = torch.dot(r, z)
        p = z + (rn / rz) * p
        rz = rn
    return x


def _exact_thermal(case, d, k, s, rc, dev):
    g = _geometry(d, dev)
    n, c0, c1, ni = g["n"], g["c0"], g["c1"], g["ni"]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    kc = t(k)
    kf = torch.empty(len(c0), dtype=torch.float64, device=dev)
    a, b = kc[c0[:ni]], kc[c1[:ni]]
    kf[:ni] = 2.0 * a * b / (a + b)
    kf[ni:] = kc[c0[ni:]]
    dm = g["am"] ** 2 / (g["area"] * g["ds"]).sum(1)
    coef = kf * dm
    sec = kf[:, None] * (g["area"] - g["ds"] * dm[:, None])
    src = g["vol"][:n] * t(s)
    T = torch.full((g["n_all"],), 300.0, dtype=torch.float64, device=dev)
    f0, group = int(d["faceGroupSize"][0]), {}
    for q, sz in enumerate(d["faceGroupSize"][1:]):
        group[q + 1] = slice(f0, f0 + int(sz))
        f0 += int(sz)
    bcs = _bcs(case)
    sb = 5.670373e-8
    nb = len(c0) - ni
    h = torch.zeros(nb, dtype=torch.float64, device=dev)
    eps, far = torch.zeros_like(h), torch.zeros_like(h)
    fixed = torch.zeros(nb, dtype=torch.bool, device=dev)
    for gid, sl in group.items():
        kind, v = bcs.get(gid, ("SpecifiedHeatFlux", {"specifiedHeatFlux": 0.0}))
        w = slice(sl.start - ni, sl.stop - ni)
        if kind == "SpecifiedTemperature":
            fixed[w] = True
            T[c1[sl]] = v["specifiedTemperature"]
        else:
            h[w] = v.get("convectiveCoefficient", 0.0)
            far[w] = v.get("farFieldTemperature", 0.0)
            eps[w] = v.get("surfaceEmissivity", 0.0) if kind in ("Radiative", "Mixed") else 0.0
    cb, i0, i1 = coef[ni:], c0[ni:], c1[ni:]
    am = g["am"][ni:]
    ci, j0, j1 = coef[:ni], c0[:ni], c1[:ni]
    rv = t(rc) * g["vol"][:n] / DT if rc is not None else None
    orth = float((sec.norm(dim=1) / (kf * g["am"])).max()) < 1e-9

    def grad():
        dT = (T[c1] - T[c0]) / g["m"]
        v = torch.zeros(g["n_all"], g["dim"], dtype=torch.float64, device=dev)
        for c in (c0, c1):
            v.index_add_(0, c, g["e"] * dT[:, None])
        w = torch.zeros(g["n_all"], 3, dtype=torch.float64, device=dev)
        w[:, :g["dim"]] = torch.einsum("nij,nj->ni", g["inv"], v)
        w[i1] = w[i0]
        return w

    def solve(old):
        first = None
        for outer in range(120):
            flux = coef * (T[c1] - T[c0])
            if not orth:
                w = grad()
                v0, v1 = g["vol"][c0][:, None], g["vol"][c1][:, None]
                flux = flux + (((w[c0] * v0 + w[c1] * v1) / (v0 + v1)) * sec).sum(1)
            r = src.clone()
            r.index_add_(0, c0, flux)
            r.index_add_(0, j1, -flux[:ni])
            if rv is not None:
                r -= rv * (T[:n] - old)
            tb = T[i1]
            heat = (-eps * sb * (tb ** 4 - far ** 4) - h * (tb - far)) * am
            bj = heat - flux[ni:]
            ajj = -(cb + (4.0 * eps * sb * tb ** 3 + h) * am)
            free = ~fixed
            r.index_add_(0, i0[free], -cb[free] * (bj / ajj)[free])
            diag = torch.zeros(n, dtype=torch.float64, device=dev)
            diag.index_add_(0, j0, ci)
            diag.index_add_(0, j1, ci)
            diag.index_add_(0, i0, cb + torch.where(free, cb * cb / ajj, torch.zeros_like(cb)))
            if rv is not None:
                diag += rv

            def mul(p):
                q = diag * p
                q.index_add_(0, j0, -ci * p[j1])
                q.index_add_(0, j1, -ci * p[j0])
                return q

            norm = float(r.abs().sum())
            first = first or norm
            if norm <= 1e-13 * first or norm == 0.0:
                break
            dx = _pcg(mul, diag, r, 1e-6 if not orth else 1e-12, 20000)
            T[:n] += dx
            dg = -(bj + cb * dx[i0]) / ajj
            T[i1] += torch.where(free, dg, torch.zeros_like(dg))

    if rv is None:
        solve(None)
    else:
        for _ in range(case["steps"]):
            solve(T[:n].clone())
    return T.cpu().numpy()


def exact(case, seed):
    path = case["path"]
    if path == "train":
        return None
    if path == "residual":
        s = _residual_system(case, seed)
        n = case["n"]
        of = torch.repeat_interleave(torch.arange(n, device="cuda"), (s["row"][1:] - s["row"][:-1]).long())
        r = s["b"] + s["diag"] * s["x"]
        r.index_add_(0, of, s["off"] * s["x"][s["col"].long()])
        return r, r.abs().sum().reshape(1)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if path == "csr":
        row, col, diag, off, b = (torch.from_numpy(v).to(dev) for v in _csr_system(case, seed))
        n = len(b)
        of = torch.repeat_interleave(torch.arange(n, device=dev), (row[1:] - row[:-1]).long())
        col = col.long()
        return _pcg(lambda p: (-diag * p).index_add_(0, of, -off * p[col]), -diag, b, 1e-14, 20000).cpu().numpy()
    n, _, _ = _cells(case)
    if path == "batch" or (case["mesh"] != "hex" and n > 120_000):
        return None  # minutes with this solver
    d, pts = _mesh(case, seed)
    k, s = _fields(case, pts, d["nCells"], seed)
    rc = None
    if path == "transient":
        rc = np.random.default_rng(seed + 300).uniform(0.5, 2.0, d["nCells"])
        s = np.zeros(d["nCells"])
    return _exact_thermal(case, d, k, s, rc, dev)
