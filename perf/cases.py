"""The work that users of this framework have it do, case by case, through its public entry points.

Single operator calls (what an integrator calls between solves, or a Krylov method of its own calls
in its loop), the set-up of an operator from order parameters, and whole calls: FP64 and
mixed-precision solves, a batch of periodic cells and a served stream.

  apply     Elastic.Fapply                       one level, FP64 or FP32
  smooth    Elastic.Fsmooth                      two damped-Jacobi sweeps in place
  residual  Elastic.Residual                     r = b - A x and its max-norm
  post      Elastic.Stress + Elastic.Energy      the fields written after a solve
  neo       Elastic.NewtonNeoHookean + Fapply    right-hand side, tangent and a product with it
  setup     Elastic.SetModelMixture + prepareForSolve + Diagonal   what every time step begins with
  solve     Linear.solve                         to a 1e-8 relative residual
  cells     CellBatch.solve                      independent periodic cells in one batch
  serve     CellServer.submit / wait             requests of six load cases each

A level is `nx` x `ny` x `nz` cells.  Stiffness kinds: "iso" and "cubic" are fields of one tensor
per node, "grains" a Voronoi map with a table of cubic tensors, "major" the 45-slot tangent.
"""
import math

import numpy as np
import torch

from anisotropicfracture_gb300 import cells as cells_mod
from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import BCElastic, Elastic, Field, Linear, level_desc

DEV = "cuda"
F64 = torch.float64
DISP, TRAC, NEUM = 0, 1, 3
# sides touched by each of the 26 faces, edges and corners, (x, y, z) in {-1, 0, 1}, in the order
# XLO YLO ZLO XHI YHI ZHI, the edges yz, zx, xy and the corners
SIDES = ([(-1, 0, 0), (0, -1, 0), (0, 0, -1), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
         + [(0, a, b) for a in (-1, 1) for b in (-1, 1)]
         + [(b, 0, a) for a in (-1, 1) for b in (-1, 1)]
         + [(a, b, 0) for a in (-1, 1) for b in (-1, 1)]
         + [(a, b, c) for a in (-1, 1) for b in (-1, 1) for c in (-1, 1)])
# the 21 slots of a tensor with major and minor symmetry, as index pairs (i, j), (k, l)
PAIRS = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
SLOTS = [(a, b) for n, a in enumerate(PAIRS) for b in PAIRS[n:]]
SLOT_OF = {}
for _s, (_a, _b) in enumerate(SLOTS):
    for _p in {_a, _a[::-1]}:
        for _q in {_b, _b[::-1]}:
            SLOT_OF[_p + _q] = SLOT_OF[_q + _p] = _s
CELL_SOLVER = dict(max_fmg_iter=0, nu1=2, nu2=2, sweeps=2, bottom=1, bottom_max_iter=200, bottom_reltol=1e-4,
                   nuf=8, max_iter=200)


def listed():
    return [
        # a product on a small isotropic box: one Krylov step of an application's own solver, where
        # the call's latency counts
        dict(name="apply_f64_iso_small", kind="apply", dtype="f64", model="iso", nx=32, ny=32, nz=32),
        # the polycrystal's finest level, FP64: the operator at the size the headline is quoted on
        dict(name="apply_f64_grains_large", kind="apply", dtype="f64", model="grains", nx=256, ny=256, nz=256, ngrains=64),
        # an FP32 product with a tensor per node (a damaged polycrystal), 129^3 nodes
        dict(name="apply_f32_cubic", kind="apply", dtype="f32", model="cubic", nx=128, ny=128, nz=128, ngrains=32),
        # a smoother call of an application's own FP32 cycle, uneven box
        dict(name="smooth_f32_grains_uneven", kind="smooth", dtype="f32", model="grains", nx=192, ny=160, nz=224, ngrains=64),
        # the plain drop-in smoother on per-node tensors, uneven box
        dict(name="smooth_f64_cubic_uneven", kind="smooth", dtype="f64", model="cubic", nx=96, ny=80, nz=112, ngrains=16),
        # stress and energy fields after a solve, written at every plot
        dict(name="post_cubic", kind="post", dtype="f64", model="cubic", nx=128, ny=128, nz=128, ngrains=32),
        # one Newton linearisation of the finite-kinematics model and a product with its tangent
        dict(name="neo_tangent", kind="neo", dtype="f64", model="major", nx=96, ny=96, nz=96),
        # the start of a time step: stiffness and eigenstrain from three order parameters, hierarchy, diagonals
        dict(name="setup_mixture", kind="setup", dtype="f64", model="cubic", nx=128, ny=128, nz=128, nphase=3),
        # the plain FP64 solve: stiff sphere in a box, 65^3 nodes, V(2,2), CG bottom
        dict(name="solve_f64_sphere", kind="solve", dtype="f64", model="iso", nx=64, ny=64, nz=64, levels=1, bottom="cg",
             inner=1),
        # the headline: two-level polycrystal of 2 x 257^3 nodes, mixed precision
        dict(name="solve_mixed_polycrystal", kind="solve", dtype="mixed", model="grains", nx=256, ny=256, nz=256, levels=2,
             bottom="cg", inner=12, ngrains=64),
        # a batch of periodic cells of uneven edges, one strain each, mixed precision
        dict(name="cells_mixed_batch", kind="cells", dtype="mixed", ncells=128, emin=16, emax=64, loads=1),
        # homogenisation requests of six load cases each into the server
        dict(name="serve_six_loads", kind="serve", dtype="mixed", nreq=6, emin=32, emax=64, loads=6),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["apply", "apply", "smooth", "smooth", "residual", "post", "neo", "setup", "solve", "solve",
                       "cells", "serve"])
    if kind in ("apply", "smooth", "residual"):
        # even and odd cell counts, 16 to 224 per direction, not all alike
        n = _log(rng, 16, 224)
        m = lambda: max(12, min(240, round(n * rng.uniform(0.75, 1.25))))  # noqa: E731
        return dict(kind=kind, dtype="f64" if kind == "residual" else rng.choice(["f64", "f32"]),
                    model=rng.choice(["iso", "cubic", "grains"]), nx=m(), ny=m(), nz=m(), ngrains=rng.randint(4, 64))
    if kind in ("post", "neo", "setup"):
        n = _log(rng, 16, 112 if kind != "post" else 160)
        m = lambda: max(12, round(n * rng.uniform(0.8, 1.2) / 2) * 2)  # noqa: E731
        c = dict(kind=kind, dtype="f64", model="major" if kind == "neo" else "cubic", nx=m(), ny=m(), nz=m())
        c.update(dict(nphase=rng.randint(2, 5)) if kind == "setup" else dict(ngrains=rng.randint(4, 32)))
        return c
    if kind == "solve":
        # boxes that coarsen to at most 5 cells, one or two levels
        dtype = rng.choice(["f64", "mixed"])
        step = rng.choice([8, 16])
        top = 64 if dtype == "f64" else 160
        n = _log(rng, 24, top)
        m = lambda: max(16, min(top, round(n * rng.uniform(0.8, 1.25) / step) * step))  # noqa: E731
        model = rng.choice(["iso", "grains"])
        return dict(kind=kind, dtype=dtype, model=model, nx=m(), ny=m(), nz=m(), levels=1 if dtype == "f64" else rng.choice([1, 2]),
                    bottom=rng.choice(["cg", "bicgstab"]), inner=1 if dtype == "f64" else rng.choice([2, 4, 8]),
                    ngrains=rng.randint(8, 64))
    if kind == "cells":
        return dict(kind=kind, dtype=rng.choice(["mixed", "mixed", "f64"]), ncells=round(_log(rng, 1, 48)), emin=16,
                    emax=rng.choice([24, 32, 48, 64]), loads=rng.choice([1, 1, 2, 6]) if rng.random() < 0.5 else 1)
    return dict(kind=kind, dtype="mixed", nreq=rng.randint(1, 4), emin=32, emax=rng.choice([40, 48, 64]), loads=6)


# ---------------------------------------------------------------- inputs (plain numpy / torch)
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rotations(n, rng):
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    return np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
                     np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
                     np.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], -2)


def _cubic_rows(n, rng):
    """21-slot rows of n randomly rotated cubic crystals, C11 / C12 / C44 = 1.68 / 1.21 / 0.75.  C44
    sits at (i, j, i, j) alone and a slot takes the last of its index tuples, as the framework's
    cubic model (and the code it follows) has it."""
    C = np.zeros((3, 3, 3, 3))
    for i in range(3):
        for j in range(3):
            C[i, i, j, j] = 1.21
        for j in range(3):
            C[i, j, i, j] = 0.75
    for i in range(3):
        C[i, i, i, i] = 1.68
    R = _rotations(n, rng)
    full = np.einsum("npi,nsk,ijkl,nqj,ntl->npqst", R, R, C, R, R)
    out = np.zeros((n, 21))
    for p in range(3):
        for q in range(3):
            for s in range(3):
                for t in range(3):
                    out[:, SLOT_OF[p, q, s, t]] = full[:, p, q, s, t]
    return out


def _axes(c, lo=(0, 0, 0), hi=None, dx=None):
    n = (c["nx"], c["ny"], c["nz"])
    hi = n if hi is None else hi
    dx = _dx(c) if dx is None else dx
    return [torch.arange(lo[d], hi[d] + 1, device=DEV, dtype=F64) * dx[d] for d in range(3)]


def _dx(c):
    # cubic cells: the longest edge has length 1
    return (1.0 / max(c["nx"], c["ny"], c["nz"]),) * 3


def _grid(ax):
    Z, Y, X = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return X, Y, Z


def _nearest(ax, seeds):
    """Nearest seed of every node, int32."""
    sq = [[(a - float(s[d])) ** 2 for d, a in enumerate(ax)] for s in seeds]
    best = torch.full((len(ax[2]), len(ax[1]), len(ax[0])), float("inf"), device=DEV, dtype=F64)
    gid = torch.zeros(best.shape, device=DEV, dtype=torch.int32)
    for g, (x, y, z) in enumerate(sq):
        d = (x[None, None, :] + y[None, :, None]) + z[:, None, None]
        near = d < best
        gid = torch.where(near, g, gid)
        best = torch.minimum(best, d)
    return gid


def _extent(c):
    h = _dx(c)
    return np.array([c["nx"] * h[0], c["ny"] * h[1], c["nz"] * h[2]])


def _table(c, seed):
    rng = np.random.default_rng(seed)
    seeds = rng.random((c["ngrains"], 3)) * _extent(c)
    return seeds, _cubic_rows(c["ngrains"], rng)


def _sphere(ax, ext, seed):
    """(lambda, mu): a stiff diffuse sphere (E 10, matrix 1, nu 0.3) near the middle of the box."""
    rng = np.random.default_rng(seed)
    ctr = (0.5 + 0.04 * (rng.random(3) - 0.5)) * ext
    r = (0.24 + 0.02 * rng.random()) * float(min(ext))
    X, Y, Z = _grid(ax)
    rsq = (X - ctr[0]) ** 2 + (Y - ctr[1]) ** 2 + (Z - ctr[2]) ** 2
    h = float(ax[0][1] - ax[0][0])
    q = (rsq - r * r) / (r * r)
    eta = 0.5 - 0.5 * torch.erf(q / (2 * h) / torch.clamp(torch.sqrt(rsq) / (r * r), min=1e-300))
    lame = lambda E, nu: (E * nu / (1 + nu) / (1 - 2 * nu), E / 2 / (1 + nu))  # noqa: E731
    (li, mi), (lo, mo) = lame(10.0, 0.3), lame(1.0, 0.3)
    return torch.stack([(1 - eta) * lo + eta * li, (1 - eta) * mo + eta * mi])


def _damage(c, ax, seed):
    """A smooth factor in [0.7, 1.3]."""
    rng = np.random.default_rng(seed + 17)
    ph = rng.random(3) * 2 * math.pi
    X, Y, Z = _grid(ax)
    return 1 + 0.3 * torch.sin(2 * math.pi * X + ph[0]) * torch.cos(2 * math.pi * Y + ph[1]) * torch.cos(math.pi * Z + ph[2])


def _stiffness(c, seed):
    """(per-node coefficients or None, grain ids or None, table or None)"""
    ax = _axes(c)
    if c["model"] == "iso":
        return _sphere(ax, _extent(c), seed), None, None
    seeds, table = _table(c, seed)
    gid = _nearest(ax, seeds)
    if c["model"] == "grains":
        return None, gid, table
    tab = torch.from_numpy(table).to(DEV)
    dmg = _damage(c, ax, seed)
    return torch.stack([tab[:, q][gid.long()] * dmg for q in range(21)]), None, None


def _displacement(c, seed, amp=0.01, rough=0.02):
    """A displacement as a solve meets it: affine, smooth waves and a rough part."""
    rng = np.random.default_rng(seed + 3)
    X, Y, Z = _grid(_axes(c))
    u = []
    for p in range(3):
        e, ph = rng.standard_normal(3), rng.random(3) * 2 * math.pi
        w = torch.sin(2 * math.pi * X + ph[0]) * torch.sin(2 * math.pi * Y + ph[1]) * torch.cos(math.pi * Z + ph[2])
        u.append(amp * (e[0] * X + e[1] * Y + e[2] * Z + 0.3 * w))
    u = torch.stack(u)
    return u + amp * rough * torch.randn(u.shape, generator=_gen(seed + 4), device=DEV, dtype=F64)


def _bc_tables(which):
    """BC types and values per face: "pull" holds z = 0, moves z = 1 by 0.01 and leaves the sides
    free; "rollers" has symmetry planes on the low faces and x = 1 pulled by 5 per cent."""
    t = np.zeros((26, 3), dtype=np.int32)
    v = np.zeros((26, 3))
    for f, s in enumerate(SIDES):
        if which == "pull":
            t[f] = TRAC if s[2] == 0 else DISP
            if s[2] > 0:
                v[f, 2] = 0.01
        else:
            t[f] = TRAC
            for d in range(3):
                if s[d] < 0:
                    t[f, d] = DISP
            if s[0] > 0:
                t[f, 0], v[f, 0] = DISP, 0.05
    return t, v


def _bc(which):
    bc = BCElastic()
    bc.type[:], bc.val[:] = _bc_tables(which)
    return bc


def _phases(c, seed):
    """Smooth order parameters on the cells (one layer around the domain): softmax of sines."""
    rng = np.random.default_rng(seed + 5)
    h = _dx(c)
    ax = [torch.arange(-1, n + 1, device=DEV, dtype=F64) * hh + 0.5 * hh for n, hh in zip((c["nx"], c["ny"], c["nz"]), h)]
    X, Y, Z = _grid(ax)
    e = []
    for _ in range(c["nphase"]):
        ph, k = rng.random(3) * 2 * math.pi, rng.integers(1, 4, 3)
        e.append(3 * torch.sin(math.pi * k[0] * X + ph[0]) * torch.sin(math.pi * k[1] * Y + ph[1]) * torch.cos(math.pi * k[2] * Z + ph[2]))
    table = _cubic_rows(c["nphase"], rng)
    f0 = 1e-3 * rng.standard_normal((c["nphase"], 9))
    return torch.softmax(torch.stack(e), 0).contiguous(), table, f0


def _shape(c):
    return (c["nz"] + 1, c["ny"] + 1, c["nx"] + 1)


def _single_op(c, model, which="pull"):
    op = Elastic([level_desc((c["nx"], c["ny"], c["nz"]), dx=_dx(c))], model)
    op.SetBC(_bc(which))
    op.SetUniform(False)
    return op


def _prepare_field_op(c, seed):
    op = _single_op(c, models.ISOTROPIC if c["model"] == "iso" else models.MAJORMINOR)
    C, gid, table = _stiffness(c, seed)
    if gid is None:
        op.SetModel(0, Field(C.contiguous()))
    else:
        op.SetModelGrains(0, Field(gid[None].contiguous()), table)
    op.prepareForSolve()
    return op


def _prepare_solve(c, seed):
    n = (c["nx"], c["ny"], c["nz"])
    h = _dx(c)
    boxes = [dict(cells=n, lo=(0, 0, 0), hi=n, ng=0, dx=h)]
    if c["levels"] == 2:  # a patch over the central 1/8
        m = tuple(2 * v for v in n)
        lo = tuple(v // 4 * 2 for v in n)
        boxes.append(dict(cells=m, lo=lo, hi=tuple(a + v for a, v in zip(lo, n)), ng=2, dx=tuple(v / 2 for v in h)))
    op = Elastic([level_desc(b["cells"], b["lo"], b["hi"], b["dx"]) for b in boxes],
                 models.ISOTROPIC if c["model"] == "iso" else models.MAJORMINOR)
    op.SetBC(_bc("pull"))
    op.SetUniform(False)
    rhs, sol = [], []
    for a, b in enumerate(boxes):
        lo = tuple(v - b["ng"] for v in b["lo"])
        hi = tuple(v + b["ng"] for v in b["hi"])
        ax = _axes(c, lo, hi, b["dx"])
        if c["model"] == "iso":
            op.SetModel(a, Field(_sphere(ax, _extent(c), seed).contiguous(), lo))
        else:
            seeds, table = _table(c, seed)
            op.SetModelGrains(a, Field(_nearest(ax, seeds)[None].contiguous(), lo), table)
        r = torch.zeros((3, len(ax[2]), len(ax[1]), len(ax[0])), device=DEV, dtype=F64)
        op.BCInit(a, Field(r, lo))
        rhs.append(Field(r, lo))
        sol.append(Field(torch.zeros_like(r), lo))
    op.prepareForSolve()
    s = Linear(op)
    s.setMaxFmgIter(0)
    s.setBottomSolver(c["bottom"])
    s.setPreSmooth(1)
    s.setPostSmooth(1)
    s.setMaxIter(400)
    s.setPrecision("fp64" if c["dtype"] == "f64" else "mixed")
    s.opts.inner_cycles = c["inner"]
    return dict(case=c, op=op, solver=s, rhs=rhs, sol=sol)


def _cell_set(c, seed, count):
    """Edges (multiples of 8), Voronoi seeds and tables of `count` periodic cells.  The edges depend
    on the case alone: another seed is other grains on the same set of sizes."""
    sizes = np.random.default_rng(1000 * count + c["emax"])
    edges = [e for e in (16, 24, 32, 40, 48, 56, 64) if c["emin"] <= e <= c["emax"] and (c["kind"] == "serve" or e not in (40, 56))]
    out = []
    for k in range(count):
        rng = np.random.default_rng(seed * 1009 + k)
        ng = int(sizes.integers(8, 33))
        out.append((int(sizes.choice(edges)), rng.random((ng, 3)), _cubic_rows(ng, rng)))
    return out


def _strain(k):
    E = np.zeros((3, 3))
    a, b = [(0, 0), (1, 1), (2, 2), (1, 2), (2, 0), (0, 1)][k % 6]
    E[a, b] += 0.5e-3
    E[b, a] += 0.5e-3
    return E


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("apply", "smooth", "residual"):
        op = _prepare_field_op(c, seed)
        dt = F64 if c["dtype"] == "f64" else torch.float32
        x = _displacement(c, seed).to(dt)
        b = torch.randn(x.shape, generator=_gen(seed + 6), device=DEV, dtype=F64).to(dt)
        return dict(case=c, op=op, x=x, b=b, y=torch.empty_like(x))
    if kind == "post":
        op = _prepare_field_op(c, seed)
        shp = _shape(c)
        return dict(case=c, op=op, x=_displacement(c, seed), s=torch.empty((9,) + shp, device=DEV, dtype=F64),
                    w=torch.empty((1,) + shp, device=DEV, dtype=F64))
    if kind == "neo":
        op = _single_op(c, models.MAJOR, "rollers")
        u = _displacement(c, seed, amp=0.03, rough=0.002)
        v = _displacement(c, seed + 1, amp=1.0)
        b = 0.1 * torch.randn(u.shape, generator=_gen(seed + 6), device=DEV, dtype=F64)
        return dict(case=c, op=op, model=models.NeoHookean(1.0, 2.5), u=u, v=v, b=b, rhs=torch.zeros_like(u),
                    y=torch.zeros_like(u))
    if kind == "setup":
        op = _single_op(c, models.MAJORMINOR)
        eta, table, f0 = _phases(c, seed)
        shp = _shape(c)
        diag = []
        for m in range(op.NMGLevels(0)):
            lo, hi = op.storage_box(0, m)
            diag.append(torch.empty((3,) + tuple(hi[d] - lo[d] + 1 for d in (2, 1, 0)), device=DEV, dtype=F64))
        return dict(case=c, op=op, eta=eta, table=table, f0=f0, F0=torch.zeros((9,) + shp, device=DEV, dtype=F64), diag=diag)
    if kind == "solve":
        return _prepare_solve(c, seed)
    if kind == "cells":
        sets = _cell_set(c, seed, c["ncells"])
        B = cells_mod.CellBatch([(n, c["loads"]) for n, _, _ in sets])
        s = 0
        for k, (n, seeds, table) in enumerate(sets):
            B.set_grains(k, seeds, table)
            for q in range(c["loads"]):
                B.set_load(s, _strain(q))
                s += 1
        B.prepare()
        w = [torch.zeros((3,) + B.shape_of(B.solve_cell[k]), device=DEV, dtype=F64) for k in range(B.nsolves)]
        return dict(case=c, batch=B, w=w)
    S = cells_mod.CellServer(precision=1 if c["dtype"] == "mixed" else 0, inner_cycles=4, hbm_budget_bytes=8 << 30,
                             **CELL_SOLVER)
    return dict(case=c, server=S, reqs=_cell_set(c, seed, c["nreq"]), loads=[_strain(q) for q in range(c["loads"])])


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "apply":
        state["op"].Fapply(0, 0, Field(state["y"]), Field(state["x"]))
        return state["y"]
    if kind == "smooth":
        state["y"].copy_(state["x"])
        state["op"].Fsmooth(0, 0, Field(state["y"]), Field(state["b"]))
        return state["y"]
    if kind == "residual":
        n = state["op"].Residual(0, 0, Field(state["y"]), Field(state["x"]), Field(state["b"]))
        return state["y"], n
    if kind == "post":
        state["op"].Stress(0, Field(state["s"]), Field(state["x"]))
        state["op"].Energy(0, Field(state["w"]), Field(state["x"]))
        return state["s"], state["w"]
    if kind == "neo":
        op = state["op"]
        op.NewtonNeoHookean(0, Field(state["rhs"]), Field(state["u"]), Field(state["b"]), state["model"])
        op.Fapply(0, 0, Field(state["y"]), Field(state["v"]))
        return state["rhs"], state["y"]
    if kind == "setup":
        op = state["op"]
        op.SetModelMixture(0, Field(state["eta"], (-1, -1, -1)), state["table"], state["f0"], Field(state["F0"]))
        op.prepareForSolve()
        for m, d in enumerate(state["diag"]):
            op.Diagonal(0, m, Field(d))
        return [state["F0"]] + state["diag"]
    if kind == "solve":
        for f in state["sol"]:
            f.arr.zero_()
        state["solver"].solve(state["sol"], state["rhs"], 1e-8, 0.0)
        # a patch's ghost layers hold the history of the iteration, not the solution
        return [state["sol"][0].arr] + [f.arr[:, 2:-2, 2:-2, 2:-2] for f in state["sol"][1:]]
    if kind == "cells":
        B = state["batch"]
        st, _ = B.solve(precision=1 if c["dtype"] == "mixed" else 0, inner_cycles=4, **CELL_SOLVER)
        for k, w in enumerate(state["w"]):
            B.solution(k, w)
        return np.stack([s["mean_stress"] for s in st]), torch.cat([w.reshape(-1) for w in state["w"]])
    S = state["server"]
    tickets = [S.submit(n, state["loads"], seeds, table) for n, seeds, table in state["reqs"]]
    out = []
    for t in tickets:
        r = S.wait(t)
        out += [s["mean_stress"] for s in r["stats"]]
        S.release(t)
    return np.stack(out)


# ---------------------------------------------------------------- what a pass cannot do without
def _coef_bytes(c, size):
    return {"iso": 2 * size, "cubic": 21 * size, "grains": 2, "major": 45 * size}[c["model"]]


def _row_flops(c):
    # second differences of three components (27 additions), the products with the stiffness and
    # their sum: 9 coefficients a row for two Lame constants, 18 for a general tensor
    return 27 + 2 * (27 if c["model"] == "iso" else 54)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("cells", "serve"):
        count = c["ncells"] if kind == "cells" else c["nreq"]
        nn = sum(n ** 3 for n, _, _ in _cell_set(c, 0, count))
        # grain ids and one solution per load case written and read back once
        return {"bytes": nn * (2 + 24 * c["loads"]), "flops": nn * c["loads"] * 135.0}
    n = (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)
    size = 8 if c["dtype"] == "f64" else 4
    if kind == "apply":
        return {"bytes": n * (6 * size + _coef_bytes(c, size)), "flops": n * _row_flops(c)}
    if kind == "smooth":  # x, b, 1/D, coefficients in, x out; two sweeps of operations
        return {"bytes": n * (12 * size + _coef_bytes(c, size)), "flops": 2 * n * (_row_flops(c) + 9)}
    if kind == "residual":
        return {"bytes": n * (9 * size + _coef_bytes(c, size)), "flops": n * (_row_flops(c) + 3)}
    if kind == "post":  # u and coefficients in, nine stresses and the energy out
        return {"bytes": n * (24 + 168 + 80), "flops": n * (9 + 108 + 18)}
    if kind == "neo":  # u, b, v in, rhs, product and tangent out
        return {"bytes": n * (5 * 24 + 360), "flops": n * 900}
    if kind == "setup":  # order parameters in, tensors, eigenstrain and diagonals out, 8/7 for the levels
        return {"bytes": n * (8 * c["nphase"] + 72 + (168 + 48) * 8 / 7), "flops": n * (c["nphase"] * 60 + 27 * 21 / 8)}
    lev = c["levels"]  # stiffness and right-hand side in, solution out
    return {"bytes": lev * n * (48 + _coef_bytes(c, 8)), "flops": lev * n * _row_flops(c)}


# ---------------------------------------------------------------- the same in plain 64-bit torch
def _full(c, C, gid, table):
    """A function (i, j, k, l) -> field (or number) of the stiffness tensor."""
    if c["model"] == "iso":
        def get(i, j, k, l):
            v = 0.0
            if i == j and k == l:
                v = v + C[0]
            if i == k and j == l:
                v = v + C[1]
            if i == l and j == k:
                v = v + C[1]
            return v
        return get
    if gid is not None:
        tab, g = torch.from_numpy(table).to(DEV), gid.long()
        return lambda i, j, k, l: tab[:, SLOT_OF[i, j, k, l]][g]
    return lambda i, j, k, l: C[SLOT_OF[i, j, k, l]]


def _diff(f, d, h):
    """First derivative along d (0 = x): central inside, one-sided on the two end planes."""
    ax = f.dim() - 1 - d
    n = f.shape[ax]
    s = lambda a, b: f.narrow(ax, a, b - a)  # noqa: E731
    return torch.cat([(s(1, 2) - s(0, 1)) / h, (s(2, n) - s(0, n - 2)) / (2 * h), (s(n - 1, n) - s(n - 2, n - 1)) / h], ax)


def _in(f, o=(0, 0, 0)):
    """The interior of f, shifted by o = (x, y, z)."""
    nz, ny, nx = f.shape
    return f[1 + o[2]:nz - 1 + o[2], 1 + o[1]:ny - 1 + o[1], 1 + o[0]:nx - 1 + o[0]]


def _second(f, a, b, h):
    e = lambda d, s: tuple(s if k == d else 0 for k in range(3))  # noqa: E731
    if a == b:
        return (_in(f, e(a, 1)) - 2 * _in(f) + _in(f, e(a, -1))) / h[a] ** 2
    t = lambda s, r: tuple(x + y for x, y in zip(e(a, s), e(b, r)))  # noqa: E731
    return (_in(f, t(1, 1)) + _in(f, t(-1, -1)) - _in(f, t(1, -1)) - _in(f, t(-1, 1))) / (4 * h[a] * h[b])


def _faces(shape):
    """(flat indices of the boundary nodes, their face number, their normal)"""
    nz, ny, nx = shape
    side = lambda n: torch.tensor([-1] + [0] * (n - 2) + [1], device=DEV)  # noqa: E731
    sx, sy, sz = (v.expand(shape).reshape(-1) for v in (side(nx)[None, None, :], side(ny)[None, :, None], side(nz)[:, None, None]))
    code = (sx + 1) * 9 + (sy + 1) * 3 + sz + 1
    at = torch.nonzero(code != 13)[:, 0]
    look = torch.zeros(27, dtype=torch.long, device=DEV)
    for f, s in enumerate(SIDES):
        look[(s[0] + 1) * 9 + (s[1] + 1) * 3 + s[2] + 1] = f
    s = torch.stack([sx[at], sy[at], sz[at]]).to(F64)
    w = torch.tensor([0, 1.0, 0.70710678118, 0.57735026919], device=DEV, dtype=F64)[s.abs().sum(0).long()]
    return at, look[code[at]], s * w


def _boundary_rows(types, u, g, sig):
    """The boundary rows of one operator application: displacement, traction or normal gradient."""
    at, face, nrm = _faces(u.shape[1:])
    t = torch.from_numpy(types).to(DEV)[face]
    out = []
    for r in range(3):
        tr = sum(sig(r, d).reshape(-1)[at] * nrm[d] for d in range(3))
        gr = sum(g[r][d].reshape(-1)[at] * nrm[d] for d in range(3))
        out.append(torch.where(t[:, r] == DISP, u[r].reshape(-1)[at], torch.where(t[:, r] == TRAC, tr, gr)))
    return at, out


def _apply64(get, u, h, types):
    g = [[_diff(u[k], l, h[l]) for l in range(3)] for k in range(3)]
    f = torch.zeros_like(u)
    for k in range(3):
        for l in range(3):
            gi = _in(g[k][l])
            for j in range(3):
                bkl = _second(u[k], l, j, h)
                o = tuple(1 if d == j else 0 for d in range(3))
                m = tuple(-v for v in o)
                for i in range(3):
                    C = get(i, j, k, l)
                    if not torch.is_tensor(C):
                        continue
                    _in(f[i]).add_(_in(C) * bkl + (_in(C, o) - _in(C, m)) / (2 * h[j]) * gi)

    def sig(r, d):
        return sum(get(r, d, k, l) * g[k][l] for k in range(3) for l in range(3))

    at, rows = _boundary_rows(types, u, g, sig)
    for r in range(3):
        f[r].view(-1)[at] = rows[r]
    return f


def _diag64(get, shape, h, types):
    D = torch.zeros((3,) + tuple(shape), device=DEV, dtype=F64)
    at, face, nrm = _faces(shape)
    t = torch.from_numpy(types).to(DEV)[face]
    sgn = torch.sign(nrm)
    for p in range(3):
        _in(D[p]).add_(sum(-2 / h[d] ** 2 * _in(get(p, d, p, d) + torch.zeros(shape, device=DEV, dtype=F64)) for d in range(3)))
        tr = torch.zeros(len(at), device=DEV, dtype=F64)
        for j in range(3):
            for l in range(3):
                C = get(p, j, p, l)
                if torch.is_tensor(C):
                    tr += C.reshape(-1)[at] * (sgn[l] / h[l]) * nrm[j]
        gr = sum(sgn[l] / h[l] * nrm[l] for l in range(3))
        D[p].view(-1)[at] = torch.where(t[:, p] == DISP, torch.ones_like(tr), torch.where(t[:, p] == TRAC, tr, gr))
    return D


def _restrict64(f):
    """Full weighting onto every second node, plain injection in a direction on its end planes."""
    for d in (2, 1, 0):
        n = f.shape[d]
        s = lambda a: f.narrow(d, a, n - 2)  # noqa: E731
        w = 0.25 * s(0) + 0.5 * s(1) + 0.25 * s(2)
        f = torch.cat([f.narrow(d, 0, 1), w, f.narrow(d, n - 1, 1)], d)
        f = f.index_select(d, torch.arange(0, n, 2, device=DEV))
    return f


def _neo64(c, u, b, v, mu, kappa, types, h):
    """Right-hand side b - div DW and the tangent's product with v at F = I + grad u."""
    eye = [[1.0 if p == d else 0.0 for d in range(3)] for p in range(3)]
    g = [[_diff(u[p], d, h[d]) for d in range(3)] for p in range(3)]
    F = [[g[p][d] + eye[p][d] for d in range(3)] for p in range(3)]
    A = torch.stack([torch.stack(r, -1) for r in F], -2)
    J = (F[0][0] * (F[1][1] * F[2][2] - F[1][2] * F[2][1]) - F[0][1] * (F[1][0] * F[2][2] - F[1][2] * F[2][0])
         + F[0][2] * (F[1][0] * F[2][1] - F[1][1] * F[2][0]))
    cr = [torch.linalg.cross(A[..., (i + 1) % 3, :], A[..., (i + 2) % 3, :]) for i in range(3)]
    G = [[cr[i][..., j] / J for j in range(3)] for i in range(3)]
    J23 = torch.abs(J) ** (2.0 / 3.0)
    tr = sum(F[i][j] ** 2 for i in range(3) for j in range(3))
    dw = [[mu * (F[i][j] / J23 - tr * G[i][j] / (3 * J23)) + kappa * (J - 1) * J * G[i][j] for j in range(3)] for i in range(3)]

    def get(i, j, k, l):
        t1 = (-2.0 / 3.0) * (F[i][j] * G[k][l] + G[i][j] * F[k][l]) + (2.0 / 9.0) * tr * G[i][j] * G[k][l]
        t1 = t1 + (1.0 / 3.0) * tr * G[i][l] * G[k][j] + (1.0 if (i == k and j == l) else 0.0)
        t2 = (2 * J - 1) * G[i][j] * G[k][l] + (1 - J) * G[i][l] * G[k][j]
        return mu / J23 * t1 + kappa * J * t2

    rhs = b.clone()
    for p in range(3):
        _in(rhs[p]).sub_(sum((_in(dw[p][d], tuple(1 if q == d else 0 for q in range(3)))
                              - _in(dw[p][d], tuple(-1 if q == d else 0 for q in range(3)))) / (2 * h[d]) for d in range(3)))
    at, rows = _boundary_rows(types, u, g, lambda r, d: dw[r][d])
    for r in range(3):
        rhs[r].view(-1)[at] = b[r].reshape(-1)[at] - rows[r]
    return rhs, _apply64(get, v, h, types)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind not in ("apply", "smooth", "residual", "post", "neo", "setup"):
        return None  # iterates of a solver that stops at a tolerance
    h = _dx(c)
    if kind == "neo":
        u = _displacement(c, seed, amp=0.03, rough=0.002)
        v = _displacement(c, seed + 1, amp=1.0)
        b = 0.1 * torch.randn(u.shape, generator=_gen(seed + 6), device=DEV, dtype=F64)
        return _neo64(c, u, b, v, 1.0, 2.5, _bc_tables("rollers")[0], h)
    types = _bc_tables("pull")[0]
    if kind == "setup":
        eta, table, f0 = _phases(c, seed)
        m = 0.25 * (eta[:, 1:, 1:, 1:] + eta[:, 1:, :-1, 1:] + eta[:, 1:, 1:, :-1] + eta[:, 1:, :-1, :-1])
        w = m / m.sum(0)
        C = torch.stack([sum(float(table[n, q]) * w[n] for n in range(len(w))) for q in range(21)])
        out = [torch.stack([sum(float(f0[n, q]) * w[n] for n in range(len(w))) for q in range(9)])]
        n = [c["nx"], c["ny"], c["nz"]]
        while True:
            out.append(_diag64(lambda i, j, k, l: C[SLOT_OF[i, j, k, l]], C.shape[1:], h, types))
            if any(v % 2 or v < 4 for v in n):
                return out
            C = torch.stack([_restrict64(C[q]) for q in range(21)])
            n, h = [v // 2 for v in n], tuple(2 * v for v in h)
    get = _full(c, *_stiffness(c, seed))
    x = _displacement(c, seed)
    if kind == "post":
        g = [[_diff(x[k], l, h[l]) for l in range(3)] for k in range(3)]
        s = [[sum(get(i, j, k, l) * g[k][l] for k in range(3) for l in range(3)) for j in range(3)] for i in range(3)]
        return (torch.stack([s[i][j] for i in range(3) for j in range(3)]),
                sum(s[i][j] * g[i][j] for i in range(3) for j in range(3))[None])
    dt = F64 if c["dtype"] == "f64" else torch.float32
    x = x.to(dt).to(F64)
    if kind == "apply":
        return _apply64(get, x, h, types)
    b = torch.randn(x.shape, generator=_gen(seed + 6), device=DEV, dtype=F64).to(dt).to(F64)
    if kind == "residual":
        r = b - _apply64(get, x, h, types)
        return r, r.abs().max()
    D = _diag64(get, x.shape[1:], h, types)
    for _ in range(2):
        x = x + (2.0 / 3.0) * (b - _apply64(get, x, h, types)) / D
    return x
