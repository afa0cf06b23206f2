"""What the performance of this framework is measured on.

Every case is a piece of work that a finite-element program hands to the
framework, through the entry points it would use: par_loops over triangles,
tetrahedra and extruded prisms, sparsity patterns, matrix assembly and
products, adjoints, batches of meshes and the vector operations of a Krylov
solver.  ``listed()`` fixes twelve of them, ``draw(rng)`` spreads more over
the same ranges.

    prepare(case, seed)   the meshes, Dats, loops and matrices a program keeps
    run(state)            one pass, returning whole outputs
    work(case)            compulsory bytes and FP operations of one pass
    exact(case, seed)     the outputs in 64-bit torch, without this package
"""
import ctypes
import math

import numpy as np
import torch

from pyop2_gb300 import _lib, device, op2
from pyop2_gb300 import workloads as W
from pyop2_gb300.adjoint import AdjointParLoop
from pyop2_gb300.batch import BatchedParLoop
from pyop2_gb300.meshes import p2_square

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest call: one 2D Laplacian action with its area Global on a
        # 64 x 64 square (8,192 triangles), as a time step on a small mesh
        # repeats it.  Launch and host latency count.
        dict(name="tri_action_64", kind="tri_action", n=64),
        # The headline loop: a matrix-free P1 Laplacian action on 12.6 M
        # tetrahedra (an operator application inside a large solve).
        dict(name="tet_action_128", kind="tet_action", n=128, permute=False),
        # Moving data between cells and vertices with little arithmetic: cell
        # means of a vertex field, the cell values added back to the vertices,
        # and sum / min / max of the cell values (projections, diagnostics).
        dict(name="project_tet_128", kind="project", n=128, permute=False, dtype="float64"),
        # The same on an extruded mesh in single precision, with the fluxes
        # through the top of the columns (atmosphere and ocean models).
        dict(name="column_256x64_f32", kind="column", n=256, cells=64, dtype="float32"),
        # Set-up of a matrix on a new mesh: the CSR pattern of P1 tetrahedra.
        dict(name="pattern_tet_128", kind="pattern_tet", n=128, permute=False),
        # Re-assembly of the P1 stiffness matrix on that pattern, as every
        # Newton or time step does it.
        dict(name="assemble_tet_100", kind="assemble_tet", n=100, permute=False),
        # Products with the assembled matrix and its transpose (a Krylov
        # iteration, an adjoint solve).
        dict(name="mult_tet_128", kind="mult_tet", n=128, permute=False),
        # Elasticity on extruded prisms: assembly of the 3x3-block matrix and
        # one product with it.
        dict(name="prism_matrix_64x32", kind="prism_matrix", n=64, cells=32),
        # The matrix-free form for eight right-hand sides, forward and adjoint
        # (sensitivities with respect to displacement and material).
        dict(name="prism_action_64x32", kind="prism_action", n=64, cells=32),
        # A nonlinear residual and its gradients through torch.autograd, as an
        # inverse problem calls it in every optimisation step.
        dict(name="adjoint_tet_64", kind="adjoint", n=64),
        # P2 operators on many meshes of uneven size, recorded once and
        # replayed in one launch (ensembles, patches).
        dict(name="batch_p2_32", kind="batch", meshes=32, lo=1e3, hi=1e6),
        # Two conjugate-gradient iterations on 1.57 M tetrahedra with the
        # matrix-free operator: actions, axpys, inner products and copies of
        # vertex Dats.
        dict(name="cg_tet_64", kind="cg", n=64, permute=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tri_action", "tet_action", "project", "column", "pattern_tet",
                       "pattern_prism", "assemble_tet", "mult_tet", "prism_matrix",
                       "prism_action", "adjoint", "batch", "cg"])
    c = dict(kind=kind)
    if kind == "tri_action":
        c["n"] = _log_int(rng, 5, 1000)
    elif kind in ("tet_action", "project", "pattern_tet", "mult_tet"):
        c["n"] = _log_int(rng, 4, 127)
        c["permute"] = rng.random() < 0.4
        if kind == "project":
            c["dtype"] = rng.choice(["float64", "float32"])
    elif kind in ("assemble_tet", "cg"):
        c["n"] = _log_int(rng, 4, 99 if kind == "assemble_tet" else 63)
        c["permute"] = rng.random() < 0.4
    elif kind == "column":
        c["n"] = _log_int(rng, 6, 250)
        c["cells"] = rng.randint(2, 64)
        c["dtype"] = rng.choice(["float64", "float32"])
    elif kind in ("pattern_prism", "prism_matrix", "prism_action"):
        c["n"] = _log_int(rng, 4, 63)
        c["cells"] = rng.randint(3, 32)
    elif kind == "adjoint":
        c["n"] = _log_int(rng, 4, 63)
    else:
        c.update(meshes=rng.randint(3, 32), lo=1e3, hi=10 ** rng.uniform(4, 6))
    return c


# ------------------------------------------------------------------ the meshes
def _tris(n, rng):
    """n x n squares split in two, interior vertices moved by up to 0.2 h."""
    c = np.arange(n + 1) / n
    X = np.stack([np.tile(c, n + 1), np.repeat(c, n + 1)], axis=1)
    inner = ((X > 0) & (X < 1)).all(axis=1)
    X += inner[:, None] * rng.uniform(-0.2 / n, 0.2 / n, X.shape)
    i = np.arange(n, dtype=np.int32)
    q = ((n + 1) * i[:, None] + i[None, :]).reshape(-1, 1, 1)
    corner = np.array([[0, 1, n + 2], [0, n + 2, n + 1]], dtype=np.int32)
    return X, (q + corner[None]).reshape(-1, 3)


def _tets(n, permute, rng):
    """n^3 cubes split into six tetrahedra each, interior vertices moved by up
    to 0.1 h; vertices in lexicographic or random order."""
    m = n + 1
    c = np.arange(m) / n
    X = np.empty((m, m, m, 3))
    X[..., 0] = c[None, None, :]
    X[..., 1] = c[None, :, None]
    X[..., 2] = c[:, None, None]
    if n > 1:
        X[1:-1, 1:-1, 1:-1] += rng.uniform(-0.1 / n, 0.1 / n, (n - 1, n - 1, n - 1, 3))
    X = X.reshape(-1, 3)
    s = (1, m, m * m)
    corner = np.array([[0, s[a], s[a] + s[b], 1 + m + m * m]
                       for a in range(3) for b in range(3) if a != b], dtype=np.int32)
    i = np.arange(n, dtype=np.int32)
    q = m * m * i[:, None, None] + m * i[None, :, None] + i[None, None, :]
    cells = (q.reshape(-1, 1, 1) + corner[None]).reshape(-1, 4)
    if permute:
        new = rng.permutation(m * m * m).astype(np.int32)
        cells = new[cells]
        old = np.empty_like(new)
        old[new] = np.arange(len(new), dtype=np.int32)
        X = X[old]
    return X, cells


def _prisms(n, cells, rng):
    """Columns of `cells` prisms over _tris(n); node = base vertex * (cells + 1)
    + level.  Returns node coordinates and the bottom cells' nodes."""
    B, tri = _tris(n, rng)
    lev = cells + 1
    X = np.empty((len(B), lev, 3))
    X[..., :2] = B[:, None, :]
    X[..., 2] = np.arange(lev) / cells
    base = np.concatenate([tri * lev, tri * lev + 1], axis=1).astype(np.int32)
    return X.reshape(-1, 3), base


def _renumbered(cells, nverts, rng, levels=1):
    """The mesh with its (base) vertices shuffled inside windows of 32, as a
    bandwidth-reducing numbering leaves them: each seed has its own pattern."""
    new = np.argsort(np.arange(nverts) // 32 + rng.random(nverts)).astype(np.int32)
    return new[cells // levels] * np.int32(levels) + cells % levels


def _sizes(case):
    """Cell counts of a batch: log-uniform in [lo, hi], fixed by the case."""
    k = case["meshes"]
    t = (np.arange(k) * 0.6180339887498949) % 1.0       # evenly spread, fixed order
    cells = case["lo"] * (case["hi"] / case["lo"]) ** t
    return [max(1, int(round(math.sqrt(c / 2)))) for c in cells]


# ------------------------------------------------------------------ the inputs
def _inputs(case, seed):
    """Host arrays of a case, from the seed alone."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "tri_action":
        X, cells = _tris(case["n"], rng)
        return dict(X=X, cells=cells, x=rng.uniform(-1, 1, len(X)))
    if kind in ("tet_action", "project", "pattern_tet", "assemble_tet", "mult_tet", "cg",
                "adjoint"):
        X, cells = _tets(case["n"], case.get("permute", False), rng)
        if kind == "pattern_tet":
            cells = _renumbered(cells, len(X), rng)
        d = dict(X=X, cells=cells)
        if kind == "adjoint":
            d["u"] = rng.uniform(-1, 1, len(X))
            d["kappa"] = rng.lognormal(0.0, 0.5, len(cells))
            d["lam"] = rng.uniform(-1, 1, len(X))
        elif kind == "project":
            d["x"] = rng.uniform(-1, 1, len(X)).astype(case["dtype"])
        elif kind in ("tet_action", "mult_tet", "cg"):
            d["x"] = rng.uniform(-1, 1, len(X))
        return d
    if kind == "batch":
        out = []
        for n in _sizes(case):
            X, cells, dofs, nd = p2_square(n, jitter=0.2, seed=int(rng.integers(1 << 30)))
            out.append(dict(X=X, cells=cells, dofs=dofs, x=rng.uniform(-1, 1, nd)))
        return out
    X, base = _prisms(case["n"], case["cells"], rng)
    if kind == "pattern_prism":
        lev = case["cells"] + 1
        base = _renumbered(base, len(X) // lev, rng, lev)
    d = dict(X=X, base=base)
    nc = len(base) * case["cells"]
    if kind == "column":
        d["x"] = rng.uniform(-1, 1, len(X)).astype(case["dtype"])
    elif kind == "prism_matrix":
        d["lame"] = rng.lognormal(0.0, 0.3, (nc, 2))
        d["x"] = rng.uniform(-1, 1, (len(X), 3))
    elif kind == "prism_action":
        d["lame"] = rng.lognormal(0.0, 0.3, (nc, 2))
        d["u"] = rng.uniform(-1, 1, (len(X), W.PRISM_NRHS, 3))
        d["w"] = rng.uniform(-1, 1, (len(X), W.PRISM_NRHS, 3))
    return d


# ------------------------------------------------------------------ local kernels
def _project_kernels(t, arity):
    return (op2.Kernel("static void cell_mean(%s *m, const %s *x)\n{ %s s = 0;\n"
                       "  for (int i = 0; i < %d; ++i) s += x[i];\n  m[0] = s * (%s)%r; }"
                       % (t, t, t, arity, t, 1.0 / arity), "cell_mean"),
            op2.Kernel("static void cell_to_vertex(%s *y, const %s *m)\n"
                       "{ for (int i = 0; i < %d; ++i) y[i] += m[0]; }" % (t, t, arity),
                       "cell_to_vertex"),
            op2.Kernel("static void cell_stats(const %s *m, %s *s, %s *lo, %s *hi)\n"
                       "{ s[0] += m[0] * m[0]; if (m[0] < lo[0]) lo[0] = m[0];\n"
                       "  if (m[0] > hi[0]) hi[0] = m[0]; }" % (t, t, t, t), "cell_stats"))


def _c(dtype):
    return {"float64": "double", "float32": "float"}[dtype]


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    device.require()
    return _PREPARE[case["kind"]](case, _inputs(case, seed))


def _flat(d):
    """Sets, map and coordinates of a flat simplicial mesh."""
    X, cells = d["X"], d["cells"]
    verts, cset = op2.Set(len(X)), op2.Set(len(cells))
    return dict(verts=verts, cells=cset, c2v=op2.Map(cset, verts, cells.shape[1], cells),
                X=op2.Dat(verts ** X.shape[1], X))


def _extruded(case, d):
    base, nn = d["base"], len(d["X"])
    bset, nodes = op2.Set(len(base)), op2.Set(nn)
    cells = op2.ExtrudedSet(bset, case["cells"] + 1)
    prisms = op2.Set(len(base) * case["cells"])
    c2n = op2.Map(cells, nodes, 6, base, offset=np.ones(6, dtype=np.int32))
    c2c = op2.Map(cells, prisms, 1,
                  (np.arange(len(base)) * case["cells"]).astype(np.int32).reshape(-1, 1),
                  offset=np.ones(1, dtype=np.int32))
    return dict(cells=cells, nodes=nodes, prisms=prisms, c2n=c2n, c2c=c2c)


def _prep_tri(case, d):
    s = _flat(d)
    s.update(x=op2.Dat(s["verts"], d["x"]), y=op2.Dat(s["verts"]), area=op2.Global(1, 0.0),
             k=op2.Kernel(W.P1_2D_LAPLACE, "p1_laplace_2d"), go=_run_tri)
    return s


def _run_tri(s):
    y, area, c2v = s["y"], s["area"], s["c2v"]
    y.zero()
    area.zero()
    op2.par_loop(s["k"], s["cells"], y(op2.INC, c2v), s["X"](op2.READ, c2v),
                 s["x"](op2.READ, c2v), area(op2.INC))
    return y.tensor, area.tensor


def _prep_tet(case, d):
    s = _flat(d)
    s.update(x=op2.Dat(s["verts"], d["x"]), y=op2.Dat(s["verts"]),
             k=op2.Kernel(W.P1_3D_LAPLACE_ACTION, "p1_laplace_3d"), go=_run_tet)
    return s


def _run_tet(s):
    y, c2v = s["y"], s["c2v"]
    y.zero()
    op2.par_loop(s["k"], s["cells"], y(op2.INC, c2v), s["X"](op2.READ, c2v),
                 s["x"](op2.READ, c2v))
    return y.tensor


def _prep_project(case, d):
    s = _flat(d)
    t = np.dtype(case["dtype"])
    s.update(x=op2.Dat(s["verts"], d["x"], t), m=op2.Dat(s["cells"], dtype=t),
             y=op2.Dat(s["verts"], dtype=t), sum=op2.Global(1, 0.0, t),
             lo=op2.Global(1, 0.0, t), hi=op2.Global(1, 0.0, t),
             k=_project_kernels(_c(case["dtype"]), 4), go=_run_project)
    return s


def _run_project(s):
    x, m, y, cells, c2v = s["x"], s["m"], s["y"], s["cells"], s["c2v"]
    mean, back, stats = s["k"]
    op2.par_loop(mean, cells, m(op2.WRITE), x(op2.READ, c2v))
    y.zero()
    op2.par_loop(back, cells, y(op2.INC, c2v), m(op2.READ))
    for g in (s["sum"], s["lo"], s["hi"]):
        g.zero()
    op2.par_loop(stats, cells, m(op2.READ), s["sum"](op2.INC), s["lo"](op2.MIN),
                 s["hi"](op2.MAX))
    return m.tensor, y.tensor, s["sum"].tensor, s["lo"].tensor, s["hi"].tensor


def _prep_column(case, d):
    s = _extruded(case, d)
    t = np.dtype(case["dtype"])
    c = _c(case["dtype"])
    mean, back, _ = _project_kernels(c, 6)
    top = op2.Kernel("static void top_flux(%s *f, const %s *x)\n"
                     "{ f[0] += x[3] + x[4] + x[5]; }" % (c, c), "top_flux")
    s.update(x=op2.Dat(s["nodes"], d["x"], t), m=op2.Dat(s["prisms"], dtype=t),
             y=op2.Dat(s["nodes"], dtype=t), flux=op2.Global(1, 0.0, t),
             k=(mean, back, top), go=_run_column)
    return s


def _run_column(s):
    x, m, y, cells, c2n, c2c = s["x"], s["m"], s["y"], s["cells"], s["c2n"], s["c2c"]
    mean, back, top = s["k"]
    op2.par_loop(mean, cells, m(op2.WRITE, c2c), x(op2.READ, c2n))
    y.zero()
    op2.par_loop(back, cells, y(op2.INC, c2n), m(op2.READ, c2c))
    s["flux"].zero()
    op2.par_loop(top, cells, s["flux"](op2.INC), x(op2.READ, c2n), iteration_region=op2.ON_TOP)
    return m.tensor, y.tensor, s["flux"].tensor


def _pattern_desc(values, nrows, cells=0):
    """The C ABI's description of the pattern of one map with itself and the
    diagonal, the map on the device; cells > 0: columns of that many cells."""
    pair = (_lib.SparsityPair * 1)()
    dmap = torch.as_tensor(values, device=DEV)
    off = np.ones(values.shape[1], dtype=np.int32)
    layers = torch.tensor([[0, cells + 1]], dtype=torch.int32, device=DEV)
    D, P = _lib.SparsityDesc(), pair[0]
    for side in "rc":
        setattr(P, side + "map", dmap.data_ptr())
        setattr(P, side + "arity", values.shape[1])
        if cells:
            setattr(P, side + "offset", off.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
    P.nent, P.region = len(values), int(op2.ALL)
    D.nrows = D.ncols = nrows
    D.set_diag, D.npairs, D.pairs = 1, 1, pair
    D.constant_layers, D.layer_slots = 1, 1
    if cells:
        # slots as op2.ExtrudedSet.layer_slots() counts them: the layers
        D.extruded, D.layer_slots, D.layers = 1, cells + 1, layers.data_ptr()
    return dict(desc=D, keep=(pair, dmap, off, layers), nrows=nrows, go=_run_pattern)


def _run_pattern(s):
    """op2g_sparsity_workspace / _count / _fill, the entry points that stand in
    for the reference's build_sparsity (op2.Sparsity calls the same three and
    then keeps the pattern for good)."""
    D, st = ctypes.byref(s["desc"]), device.stream_handle()
    nbytes, nnz = ctypes.c_size_t(), ctypes.c_int64()
    _lib.call("op2g_sparsity_workspace", D, ctypes.byref(nbytes))
    ws = torch.empty(nbytes.value, dtype=torch.uint8, device=DEV)
    rowptr = torch.empty(s["nrows"] + 1, dtype=torch.int64, device=DEV)
    _lib.call("op2g_sparsity_count", D, ws.data_ptr(), nbytes.value, rowptr.data_ptr(),
              ctypes.byref(nnz), st)
    colidx = torch.empty(nnz.value, dtype=torch.int32, device=DEV)
    _lib.call("op2g_sparsity_fill", D, ws.data_ptr(), nbytes.value, rowptr.data_ptr(),
              colidx.data_ptr(), st)
    return rowptr, colidx


def _prep_pattern_tet(case, d):
    return _pattern_desc(d["cells"], len(d["X"]))


def _prep_pattern_prism(case, d):
    return _pattern_desc(d["base"], len(d["X"]), case["cells"])


def _stiffness(s):
    sp = op2.Sparsity((s["verts"] ** 1, s["verts"] ** 1), [(s["c2v"], s["c2v"], None)])
    return op2.Mat(sp), op2.Kernel(W.P1_3D_LAPLACE_MATRIX, "p1_laplace_3d_mat")


def _prep_assemble(case, d):
    s = _flat(d)
    s["A"], s["k"] = _stiffness(s)
    s["go"] = _run_assemble
    return s


def _run_assemble(s):
    A, c2v = s["A"], s["c2v"]
    A.zero()
    op2.par_loop(s["k"], s["cells"], A(op2.INC, (c2v, c2v)), s["X"](op2.READ, c2v))
    A.assemble()
    return A.tensor


def _prep_mult(case, d):
    s = _prep_assemble(case, d)
    _run_assemble(s)
    s.update(x=op2.Dat(s["verts"], d["x"]), y=op2.Dat(s["verts"]), z=op2.Dat(s["verts"]),
             go=_run_mult)
    return s


def _run_mult(s):
    s["A"].mult(s["x"], s["y"])
    s["A"].mult(s["x"], s["z"], transpose=True)
    return s["y"].tensor, s["z"].tensor


def _prep_prism_matrix(case, d):
    s = _extruded(case, d)
    n3 = s["nodes"] ** 3
    s.update(A=op2.Mat(op2.Sparsity((n3, n3), [(s["c2n"], s["c2n"], None)])),
             X=op2.Dat(n3, d["X"]), L=op2.Dat(s["prisms"] ** 2, d["lame"]),
             x=op2.Dat(n3, d["x"]), y=op2.Dat(n3),
             k=op2.Kernel(W.PRISM_ELASTICITY_MATRIX, "prism_elasticity_mat"),
             go=_run_prism_matrix)
    return s


def _run_prism_matrix(s):
    A, c2n = s["A"], s["c2n"]
    A.zero()
    op2.par_loop(s["k"], s["cells"], A(op2.INC, (c2n, c2n)), s["X"](op2.READ, c2n),
                 s["L"](op2.READ, s["c2c"]))
    A.assemble()
    A.mult(s["x"], s["y"])
    return A.tensor, s["y"].tensor


def _prep_prism_action(case, d):
    s = _extruded(case, d)
    ds = op2.DataSet(s["nodes"], (W.PRISM_NRHS, 3))
    s.update(X=op2.Dat(s["nodes"] ** 3, d["X"]), L=op2.Dat(s["prisms"] ** 2, d["lame"]),
             u=op2.Dat(ds, d["u"]), w=op2.Dat(ds, d["w"]), y=op2.Dat(ds), du=op2.Dat(ds),
             dL=op2.Dat(s["prisms"] ** 2),
             k=(op2.Kernel(W.PRISM_ELASTICITY_ACTION, "prism_elasticity"),
                op2.Kernel(W.PRISM_ELASTICITY_VJP, "prism_elasticity_vjp")),
             go=_run_prism_action)
    return s


def _run_prism_action(s):
    cells, c2n, c2c, X, L, u = s["cells"], s["c2n"], s["c2c"], s["X"], s["L"], s["u"]
    s["y"].zero()
    op2.par_loop(s["k"][0], cells, s["y"](op2.INC, c2n), X(op2.READ, c2n), u(op2.READ, c2n),
                 L(op2.READ, c2c))
    s["du"].zero()
    op2.par_loop(s["k"][1], cells, s["w"](op2.READ, c2n), X(op2.READ, c2n), u(op2.READ, c2n),
                 L(op2.READ, c2c), s["du"](op2.INC, c2n), s["dL"](op2.WRITE, c2c))
    return s["y"].tensor, s["du"].tensor, s["dL"].tensor


def _prep_adjoint(case, d):
    s = _flat(d)
    v1 = s["verts"] ** 1
    loop = AdjointParLoop(s["cells"], op2.Kernel(W.NL_RESIDUAL, "nl_residual"),
                          op2.Kernel(W.NL_RESIDUAL_VJP, "nl_residual_vjp"),
                          (v1, s["c2v"]), [(v1, s["c2v"]), (s["cells"] ** 1, None)],
                          constants=[(s["X"], s["c2v"])])
    t = {k: torch.tensor(d[k], device=DEV) for k in ("u", "kappa", "lam")}
    s.update(loop=loop, u=t["u"].requires_grad_(), kappa=t["kappa"].requires_grad_(),
             lam=t["lam"], go=_run_adjoint)
    return s


def _run_adjoint(s):
    F = s["loop"](s["u"], s["kappa"])
    du, dk = torch.autograd.grad(F, (s["u"], s["kappa"]), s["lam"])
    return F.detach(), du, dk


def _prep_batch(case, meshes):
    k = op2.Kernel(W.P2_MASS_LAPLACE, "p2_mass_laplace")
    total = sum(len(d["x"]) for d in meshes)
    ytot = torch.zeros(total, dtype=torch.float64, device=DEV)
    loops, gs, at = [], [], 0
    for d in meshes:
        m = _flat(d)
        dofs = op2.Set(len(d["x"]))
        c2d = op2.Map(m["cells"], dofs, 6, d["dofs"])
        y = op2.Dat.from_tensor(dofs ** 1, ytot[at:at + len(d["x"])])
        at += len(d["x"])
        g = op2.Global(1, 0.0)
        gs.append(g)
        loops.append(op2.ParLoop(k, m["cells"], y(op2.INC, c2d), m["X"](op2.READ, m["c2v"]),
                                 op2.Dat(dofs, d["x"])(op2.READ, c2d), g(op2.INC)))
    b = BatchedParLoop(loops)
    b.capture()
    return dict(batch=b, y=ytot, g=gs, go=_run_batch)


def _run_batch(s):
    s["y"].zero_()
    for g in s["g"]:
        g.zero()
    s["batch"].replay()
    return [s["y"]] + [g.tensor for g in s["g"]]


CG_STEPS = 2


def _prep_cg(case, d):
    s = _prep_tet(case, d)
    v = s["verts"]
    # the Laplacian plus a lumped mass term keeps the operator definite
    s.update(b=s["x"], mass=op2.Dat(v, np.full(len(d["X"]), 1.0 / len(d["X"]))),
             x=op2.Dat(v), r=op2.Dat(v), p=op2.Dat(v), q=op2.Dat(v), go=_run_cg)
    return s


def _run_cg(s):
    x, r, p, q, c2v = s["x"], s["r"], s["p"], s["q"], s["c2v"]
    x.zero()
    s["b"].copy(r)
    r.copy(p)
    rr = r.inner(r)
    for _ in range(CG_STEPS):
        q.zero()
        op2.par_loop(s["k"], s["cells"], q(op2.INC, c2v), s["X"](op2.READ, c2v),
                     p(op2.READ, c2v))
        q += s["mass"] * p
        alpha = float(rr / p.inner(q))
        x += p * alpha
        r -= q * alpha
        new = r.inner(r)
        p *= float(new / rr)
        p += r
        rr = new
    return x.tensor, r.tensor, np.array([r.norm])


_PREPARE = {"tri_action": _prep_tri, "tet_action": _prep_tet, "project": _prep_project,
            "column": _prep_column, "pattern_tet": _prep_pattern_tet,
            "pattern_prism": _prep_pattern_prism, "assemble_tet": _prep_assemble,
            "mult_tet": _prep_mult, "prism_matrix": _prep_prism_matrix,
            "prism_action": _prep_prism_action, "adjoint": _prep_adjoint, "batch": _prep_batch,
            "cg": _prep_cg}


def run(state):
    return state["go"](state)


# ------------------------------------------------------------------ work
def _tet_nnz(n):
    """Distinct neighbours of the split cubes' vertices, themselves included:
    the vertices plus twice the edges (axes, face diagonals, body diagonals)."""
    m = n + 1
    return m ** 3 + 2 * (3 * n * m * m + 3 * n * n * m + n ** 3)


def _prism_blocks(n, cells):
    lev = cells + 1
    base = (n + 1) ** 2 + 2 * (2 * n * (n + 1) + n * n)
    return base * (lev + 2 * cells)


def work(case):
    """Compulsory bytes (each input read once, each output written once) and
    floating-point operations (FMA = 2) of one pass."""
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for n in _sizes(case):
            C, V, D = 2 * n * n, (n + 1) ** 2, (2 * n + 1) ** 2
            b += C * 36 + V * 16 + D * 16
            f += C * W.P2_FLOPS
        return dict(bytes=b, flops=f)
    n = case["n"]
    if kind == "tri_action":
        C, V = 2 * n * n, (n + 1) ** 2
        return dict(bytes=C * 12 + V * 32 + 8, flops=C * W.P1_2D_FLOPS)
    if kind in ("column", "pattern_prism", "prism_matrix", "prism_action"):
        B, N = 2 * n * n, (n + 1) ** 2 * (case["cells"] + 1)
        C = B * case["cells"]
        maps = B * 28
        nb = _prism_blocks(n, case["cells"])
        if kind == "column":
            e = np.dtype(case["dtype"]).itemsize
            return dict(bytes=2 * maps + (2 * C + 2 * N + (n + 1) ** 2) * e,
                        flops=13 * C + 3 * B)
        if kind == "pattern_prism":
            return dict(bytes=B * 24 + N * 8 + nb * 4, flops=0)
        if kind == "prism_matrix":
            return dict(bytes=maps + N * 24 + C * 16 + nb * 4 + nb * 72
                        + nb * 76 + N * 56, flops=C * 6300 + nb * 18)
        r = W.PRISM_NRHS
        return dict(bytes=2 * maps + 2 * (N * 24 + C * 16) + N * r * 24 * 5 + C * 16,
                    flops=C * r * (W.PRISM_ACTION_FLOPS_PER_RHS + 1300))
    C, V = 6 * n ** 3, (n + 1) ** 3
    nnz = _tet_nnz(n)
    if kind == "tet_action":
        return dict(bytes=C * 16 + V * 40, flops=C * W.P1_3D_FLOPS)
    if kind == "project":
        e = np.dtype(case["dtype"]).itemsize
        return dict(bytes=2 * (C * 16) + (3 * C + 2 * V) * e, flops=12 * C)
    if kind == "pattern_tet":
        return dict(bytes=C * 16 + V * 8 + nnz * 4, flops=0)
    if kind == "assemble_tet":
        return dict(bytes=C * 16 + V * 32 + nnz * 12, flops=C * W.P1_3D_MATRIX_FLOPS)
    if kind == "mult_tet":
        return dict(bytes=2 * (nnz * 12 + V * 24), flops=4 * nnz)
    if kind == "adjoint":
        return dict(bytes=C * 16 + V * 40 + C * 8 + C * 16 + V * 48 + C * 16,
                    flops=C * (W.NL_RESIDUAL_FLOPS + W.NL_RESIDUAL_VJP_FLOPS))
    return dict(bytes=V * 24 + CG_STEPS * (C * 16 + V * 40 + V * 8 * 22),
                flops=CG_STEPS * (C * W.P1_3D_FLOPS + V * 14))


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """What ``run`` returns, computed in 64 bits by plain torch."""
    f = _EXACT.get(case["kind"])
    if f is None:
        return None
    with torch.no_grad():
        return f(case, _inputs(case, seed))


def _t(a):
    t = torch.as_tensor(np.ascontiguousarray(a), device=DEV)
    return t if t.dtype in (torch.int32, torch.int64) else t.double()


def _tet_geometry(X, c):
    """Columns G_0..G_3 (gradients of the hat functions times det) and det."""
    p = X[c]
    a, b, d = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], p[:, 3] - p[:, 0]
    g1, g2, g3 = torch.linalg.cross(b, d), torch.linalg.cross(d, a), torch.linalg.cross(a, b)
    det = (a * g1).sum(1)
    return torch.stack([-(g1 + g2 + g3), g1, g2, g3], 1), det


def _tet_apply(X, c, x):
    G, det = _tet_geometry(X, c)
    v = (G * x[c].unsqueeze(2)).sum(1)
    e = (G * v.unsqueeze(1)).sum(2) / (6 * det.abs()).unsqueeze(1)
    return torch.zeros_like(x).index_add_(0, c.reshape(-1), e.reshape(-1))


def _exact_tri(case, d):
    X, c, x = _t(d["X"]), _t(d["cells"]).long(), _t(d["x"])
    p = X[c]
    e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    det = e1[:, 0] * e2[:, 1] - e2[:, 0] * e1[:, 1]
    area = det.abs() / 2
    g1 = torch.stack([e2[:, 1], -e2[:, 0]], 1) / det[:, None]
    g2 = torch.stack([-e1[:, 1], e1[:, 0]], 1) / det[:, None]
    G = torch.stack([-(g1 + g2), g1, g2], 1)
    v = (G * x[c].unsqueeze(2)).sum(1)
    e = area[:, None] * (G * v.unsqueeze(1)).sum(2)
    y = torch.zeros_like(x).index_add_(0, c.reshape(-1), e.reshape(-1))
    return y, area.sum().reshape(1)


def _exact_tet(case, d):
    return _tet_apply(_t(d["X"]), _t(d["cells"]).long(), _t(d["x"]))


def _exact_project(case, d):
    c, x = _t(d["cells"]).long(), _t(d["x"])
    m = x[c].mean(1)
    y = torch.zeros_like(x).index_add_(0, c.reshape(-1), m.repeat_interleave(4))
    z = torch.zeros(1, dtype=torch.float64, device=DEV)
    return (m, y, (m * m).sum().reshape(1), torch.minimum(m.min(), z), torch.maximum(m.max(), z))


def _prism_nodes(case, d):
    """[columns * cells, 6] nodes, cells of a column in order."""
    b = _t(d["base"]).long()
    k = torch.arange(case["cells"], device=DEV)
    return (b[:, None, :] + k[None, :, None]).reshape(-1, 6)


def _exact_column(case, d):
    c, x = _prism_nodes(case, d), _t(d["x"])
    m = x[c].mean(1)
    y = torch.zeros_like(x).index_add_(0, c.reshape(-1), m.repeat_interleave(6))
    top = _t(d["base"]).long()[:, 3:] + (case["cells"] - 1)
    return m, y, x[top].sum().reshape(1)


def _tet_csr(case, d):
    """Sorted (row, column) keys and values of the assembled stiffness."""
    X, c = _t(d["X"]), _t(d["cells"]).long()
    G, det = _tet_geometry(X, c)
    e = torch.bmm(G, G.transpose(1, 2)) / (6 * det.abs())[:, None, None]
    V = len(X)
    key = (c[:, :, None] * V + c[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    return uniq, torch.zeros(len(uniq), dtype=torch.float64, device=DEV).index_add_(
        0, inv, e.reshape(-1)), V


def _exact_assemble(case, d):
    return _tet_csr(case, d)[1]


def _exact_mult(case, d):
    y = _exact_tet(case, d)
    return y, y.clone()


def _prism_points(case, d):
    """Gradients of the six nodal functions at the six quadrature points of
    every prism, [cells, point, node, 3], and the points' weights."""
    p = _t(d["X"])[_prism_nodes(case, d)]
    e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    det = e1[:, 0] * e2[:, 1] - e2[:, 0] * e1[:, 1]
    h = p[:, 3, 2] - p[:, 0, 2]
    g1 = torch.stack([e2[:, 1], -e2[:, 0]], 1) / det[:, None]
    g2 = torch.stack([-e1[:, 1], e1[:, 0]], 1) / det[:, None]
    g = torch.stack([-(g1 + g2), g1, g2], 1)
    G = torch.zeros(len(p), 6, 6, 3, dtype=torch.float64, device=DEV)
    tl = (torch.full((3, 3), 1 / 6, dtype=torch.float64, device=DEV)
          + 0.5 * torch.eye(3, dtype=torch.float64, device=DEV))
    for z, zz in enumerate((0.5 - 0.5 / math.sqrt(3), 0.5 + 0.5 / math.sqrt(3))):
        for q in range(3):
            k = 3 * z + q
            G[:, k, :3, :2] = g * (1 - zz)
            G[:, k, 3:, :2] = g * zz
            G[:, k, :3, 2] = -tl[q] / h[:, None]
            G[:, k, 3:, 2] = tl[q] / h[:, None]
    return G, (det * h).abs() / 12


def _exact_prism_matrix(case, d):
    G, wq = _prism_points(case, d)
    lame, nodes = _t(d["lame"]), _prism_nodes(case, d)
    wl, wm = (wq * lame[:, 0]), (wq * lame[:, 1])
    GG = torch.einsum("nqic,nqjd->nijcd", G, G)
    tr = GG.diagonal(dim1=3, dim2=4).sum(-1)
    K = (wl[:, None, None, None, None] * GG
         + wm[:, None, None, None, None] * (GG.transpose(3, 4)
                                            + tr[..., None, None]
                                            * torch.eye(3, dtype=torch.float64, device=DEV)))
    V = len(d["X"])
    key = (nodes[:, :, None] * V + nodes[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    A = torch.zeros(len(uniq), 3, 3, dtype=torch.float64, device=DEV).index_add_(
        0, inv, K.reshape(-1, 3, 3))
    x = _t(d["x"])
    y = torch.zeros_like(x).index_add_(0, uniq // V,
                                       (A * x[uniq % V].unsqueeze(1)).sum(2))
    return A.reshape(-1), y


def _exact_prism_action(case, d):
    G, wq = _prism_points(case, d)
    lame, nodes = _t(d["lame"]), _prism_nodes(case, d)
    u, w = _t(d["u"]), _t(d["w"])
    lam, mu = lame[:, 0], lame[:, 1]
    y, du = torch.zeros_like(u), torch.zeros_like(u)
    dl, dm = torch.zeros_like(lam), torch.zeros_like(lam)

    def eps(f, r):
        return torch.einsum("nqid,nic->nqcd", G, f[nodes, r])

    def force(e):
        tr = e.diagonal(dim1=2, dim2=3).sum(-1)
        s = mu[:, None, None, None] * (e + e.transpose(2, 3)) + \
            (lam[:, None] * tr)[..., None, None] * torch.eye(3, dtype=torch.float64, device=DEV)
        return torch.einsum("nqid,nqcd->nic", G, s) * wq[:, None, None], tr

    for r in range(u.shape[1]):
        eu, ew = eps(u, r), eps(w, r)
        fu, tu = force(eu)
        fw, tw = force(ew)
        for out, f in ((y, fu), (du, fw)):
            out[:, r].index_add_(0, nodes.reshape(-1), f.reshape(-1, 3))
        dl += wq * (tu * tw).sum(1)
        dm += wq * 0.5 * ((eu + eu.transpose(2, 3)) * (ew + ew.transpose(2, 3))).sum((1, 2, 3))
    return y, du, torch.stack([dl, dm], 1)


def _exact_adjoint(case, d):
    X, c = _t(d["X"]), _t(d["cells"]).long()
    u, kappa, lam = _t(d["u"]), _t(d["kappa"]), _t(d["lam"])
    G, det = _tet_geometry(X, c)
    s, uc, lc = 1 / (6 * det.abs()), u[c], lam[c]
    S = uc.sum(1)
    q1 = 1 + 0.05 * ((uc * uc).sum(1) + S * S)
    v = (G * uc.unsqueeze(2)).sum(1)
    vl = (G * lc.unsqueeze(2)).sum(1)
    Gv, Gl = (G * v.unsqueeze(1)).sum(2), (G * vl.unsqueeze(1)).sum(2)
    gg = (v * vl).sum(1)
    Fe = (kappa * q1 * s)[:, None] * Gv - (det.abs() / 24)[:, None]
    de = (kappa * s)[:, None] * (0.1 * gg[:, None] * (uc + S[:, None]) + q1[:, None] * Gl)
    z = torch.zeros_like(u)
    return (z.clone().index_add_(0, c.reshape(-1), Fe.reshape(-1)),
            z.clone().index_add_(0, c.reshape(-1), de.reshape(-1)), q1 * gg * s)


def _p2_matrices():
    """Mass matrix and the three stiffness blocks of the P2 reference triangle
    (vertices, then the edges opposite to them), by a product Gauss rule."""
    g, wg = np.polynomial.legendre.leggauss(5)
    g, wg = (g + 1) / 2, wg / 2
    s, t = (a.ravel() for a in np.meshgrid(g, g, indexing="ij"))
    wq = np.outer(wg, wg).ravel() * (1 - s)
    L = np.stack([1 - s - t * (1 - s), s, t * (1 - s)])
    dL = np.array([[-1.0, -1.0], [1.0, 0.0], [0.0, 1.0]])
    phi, dphi = [], []
    for a in range(3):
        phi.append(L[a] * (2 * L[a] - 1))
        dphi.append((4 * L[a] - 1)[:, None] * dL[a])
    for a, b in ((1, 2), (0, 2), (0, 1)):
        phi.append(4 * L[a] * L[b])
        dphi.append(4 * (L[a][:, None] * dL[b] + L[b][:, None] * dL[a]))
    phi, dphi = np.stack(phi), np.stack(dphi)
    K = np.einsum("q,iqa,jqb->abij", wq, dphi, dphi)
    return [np.einsum("q,iq,jq->ij", wq, phi, phi), K[0, 0], K[0, 1] + K[1, 0], K[1, 1]]


def _exact_batch(case, meshes):
    R = [_t(m) for m in _p2_matrices()]
    ys, gs = [], []
    for d in meshes:
        p, c, x = _t(d["X"])[_t(d["cells"]).long()], _t(d["dofs"]).long(), _t(d["x"])
        e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        det = (e1[:, 0] * e2[:, 1] - e2[:, 0] * e1[:, 1]).abs()
        w = (det, (e2 * e2).sum(1) / det, -(e1 * e2).sum(1) / det, (e1 * e1).sum(1) / det)
        e = sum(wi[:, None] * (x[c] @ Ri.T) for wi, Ri in zip(w, R))
        ys.append(torch.zeros_like(x).index_add_(0, c.reshape(-1), e.reshape(-1)))
        gs.append((e * e).sum().reshape(1))
    return [torch.cat(ys)] + gs


def _exact_cg(case, d):
    X, c, b = _t(d["X"]), _t(d["cells"]).long(), _t(d["x"])
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), torch.dot(r, r)
    for _ in range(CG_STEPS):
        q = _tet_apply(X, c, p) + p / len(b)
        alpha = rr / torch.dot(p, q)
        x = x + alpha * p
        r = r - alpha * q
        new = torch.dot(r, r)
        p = (new / rr) * p + r
        rr = new
    return x, r, torch.sqrt(torch.dot(r, r)).reshape(1)


_EXACT = {"tri_action": _exact_tri, "tet_action": _exact_tet, "project": _exact_project,
          "column": _exact_column, "assemble_tet": _exact_assemble, "mult_tet": _exact_mult,
          "prism_matrix": _exact_prism_matrix, "prism_action": _exact_prism_action,
          "adjoint": _exact_adjoint, "batch": _exact_batch, "cg": _exact_cg}
