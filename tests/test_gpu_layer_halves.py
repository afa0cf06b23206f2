"""Light extruded loops over enough cells that a thread takes two layers of a
column: columns of even and odd length around the shortest that do, cell counts
on both sides of the line, cells and interior facets, subsets, negative map
entries, increments, reductions and writes.  Whole numbers, so that every order
of the sums is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = {"float64": "double", "float32": "float", "int64": "long long"}
LINE = 400_000      # cells from which two layers go together


def mesh(op2, n, cells, negative, rng):
    levels = cells + 1
    v = rng.integers(0, n // 2 + 2, (n, 3)) * levels
    m = np.concatenate([v, v + 1], axis=1)
    if negative:
        m[rng.random(m.shape) < 0.05] = -1
    base, nodes = op2.Set(n), op2.Set((n // 2 + 2) * levels)
    ext = op2.ExtrudedSet(base, levels)
    return ext, nodes, m.astype(np.int32), op2.Map(ext, nodes, 6, m.astype(np.int32),
                                                   offset=np.ones(6, dtype=np.int32))


def packs(m, rows, x, facets, cells):
    """Per layer: the target indices and the x values of an iteration."""
    for l in range(cells - 1 if facets else cells):
        v = m[rows]
        idx = np.where(v >= 0, v + l, -1)
        if facets:
            idx = np.concatenate([idx, np.where(v >= 0, v + l + 1, -1)], axis=1)
        yield l, idx, np.where(idx >= 0, x[idx], 0)


@pytest.mark.parametrize("dtype", ["float64", "float32", "int64"])
@pytest.mark.parametrize("cells,facets,negative", [
    (31, False, False), (32, False, False), (33, False, True), (47, False, False),
    (64, False, True), (33, True, False), (34, True, True)])
@pytest.mark.parametrize("above", [False, True])
def test_against_numpy(gpu_op2, dtype, cells, facets, negative, above):
    op2 = gpu_op2
    rng = np.random.default_rng(cells)
    per = cells - 1 if facets else cells
    n = LINE // per + (1 if above else -1)
    ext, nodes, m, mp = mesh(op2, n, cells, negative, rng)
    t = C[dtype]
    xv = rng.integers(-2, 3, nodes.size).astype(dtype)
    x, y, g = op2.Dat(nodes, xv, dtype), op2.Dat(nodes, dtype=dtype), op2.Global(1, 0, dtype)
    ne = 12 if facets else 6
    k = op2.Kernel("static void inc(%s *y, const %s *x, %s *g, int layer) { for (int i = 0; i < %d; ++i) "
                   "{ y[i] += x[i] * (i + 1) + layer; g[0] += x[i]; } }" % (t, t, t, ne), "inc")
    region = op2.ON_INTERIOR_FACETS if facets else op2.ALL
    for it, rows in ((ext, np.arange(n)), (op2.Subset(ext, np.arange(1, n)), np.arange(1, n))):
        y.zero()
        g.zero()
        op2.par_loop(k, it, y(op2.INC, mp), x(op2.READ, mp), g(op2.INC), iteration_region=region,
                     pass_layer_arg=True)
        ref, total = np.zeros(nodes.size, dtype=np.int64), 0
        for l, idx, v in packs(m, rows, xv.astype(np.int64), facets, cells):
            w = v * (np.arange(ne) + 1) + l
            ok = idx >= 0
            ref += np.bincount(idx[ok], weights=w[ok], minlength=nodes.size).astype(np.int64)
            total += int(v.sum())
        assert np.array_equal(y.data_ro, ref.astype(dtype))
        assert int(g.data_ro[0]) == total


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("cells", [32, 37])
def test_writes(gpu_op2, dtype, cells):
    """A cell field written from the column's nodes."""
    op2 = gpu_op2
    rng = np.random.default_rng(3)
    n = LINE // cells + 1
    ext, nodes, m, mp = mesh(op2, n, cells, False, rng)
    prisms = op2.Set(n * cells)
    c2c = op2.Map(ext, prisms, 1, (np.arange(n) * cells).reshape(-1, 1).astype(np.int32),
                  offset=np.ones(1, dtype=np.int32))
    xv = rng.integers(-9, 10, nodes.size).astype(dtype)
    x, c = op2.Dat(nodes, xv, dtype), op2.Dat(prisms, np.full(n * cells, 77), dtype)
    t = C[dtype]
    k = op2.Kernel("static void w(%s *c, const %s *x, int layer) { c[0] = layer; for (int i = 0; i < 6; ++i) "
                   "c[0] += (i + 1) * x[i]; }" % (t, t), "w")
    op2.par_loop(k, ext, c(op2.WRITE, c2c), x(op2.READ, mp), pass_layer_arg=True)
    ref = np.empty((n, cells))
    for l, _, v in packs(m, np.arange(n), xv.astype(np.float64), False, cells):
        ref[:, l] = l + v @ (np.arange(6) + 1)
    assert np.array_equal(c.data_ro, ref.reshape(-1).astype(dtype))
