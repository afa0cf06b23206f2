"""Light extruded loops: neighbouring layers' increments combined in a warp
(8-byte types), the (entity, layer) stepped along the sweep and one sign test
per iteration.  Maps whose entries pair up, pair up on some columns only, or
do not; negative entries; layer counts around a warp; regions, subsets and
periodic columns; whole numbers, so that every order of the sums is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = {"float64": "double", "float32": "float", "int64": "long long"}


def columns(rng, n, levels, kind):
    """[n, 6] base-layer nodes of columns over n + 2 base vertices."""
    base = np.stack([np.arange(n), np.arange(n) + 1, rng.permutation(n) + 2], axis=1) * levels
    m = np.concatenate([base, base + 1], axis=1)
    if kind == "some":                       # every third column in another order
        m[::3] = m[::3][:, [3, 1, 2, 0, 4, 5]]
    elif kind == "none":
        m = m[:, ::-1].copy()
    elif kind == "negative":
        m[rng.random(m.shape) < 0.2] = -1
    return m.astype(np.int32)


def expected(m, cells, rows, x, size, lay0, lay1):
    y = np.zeros(size, dtype=x.dtype)
    for l in range(lay0, lay1):
        v = m[rows]
        idx = v + l
        contrib = x[rows][:, None] * (np.arange(6) + 1) + l
        np.add.at(y, idx[v >= 0], contrib[v >= 0].astype(x.dtype))
    return y


@pytest.mark.parametrize("dtype", ["float64", "float32", "int64"])
@pytest.mark.parametrize("kind", ["pairs", "some", "none", "negative"])
@pytest.mark.parametrize("n,cells", [(1, 1), (3, 31), (7, 32), (40, 33), (501, 2), (9_001, 70)])
def test_increments(gpu_op2, dtype, kind, n, cells):
    op2 = gpu_op2
    rng = np.random.default_rng(n + cells)
    levels = cells + 1
    m = columns(rng, n, levels, kind)
    size = (n + 2) * levels
    bset, nodes = op2.Set(n), op2.Set(size)
    ext = op2.ExtrudedSet(bset, levels)
    mp = op2.Map(ext, nodes, 6, m, offset=np.ones(6, dtype=np.int32))
    xv = rng.integers(-3, 4, n).astype(dtype)
    x = op2.Dat(bset, xv, dtype)
    t = C[dtype]
    k = op2.Kernel("static void inc(%s *y, const %s *x, int layer) { for (int i = 0; i < 6; ++i) "
                   "y[i] += x[0] * (i + 1) + layer; }" % (t, t), "inc")
    ranges = {op2.ALL: (0, cells), op2.ON_BOTTOM: (0, 1), op2.ON_TOP: (cells - 1, cells)}
    sub = np.arange(0, n, 2)
    for region, (l0, l1) in ranges.items():
        for it, rows in ((ext, np.arange(n)), (op2.Subset(ext, sub), sub)):
            y = op2.Dat(nodes, dtype=dtype)
            op2.par_loop(k, it, y(op2.INC, mp), x(op2.READ), iteration_region=region,
                         pass_layer_arg=True)
            ref = expected(m, cells, rows, xv, size, l0, l1)
            assert np.array_equal(y.data_ro, ref), region


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("kind", ["pairs", "negative"])
def test_gathers(gpu_op2, dtype, kind):
    op2 = gpu_op2
    rng = np.random.default_rng(5)
    n, cells = 4_003, 37
    levels = cells + 1
    m = columns(rng, n, levels, kind)
    bset, nodes, prisms = op2.Set(n), op2.Set((n + 2) * levels), op2.Set(n * cells)
    ext = op2.ExtrudedSet(bset, levels)
    mp = op2.Map(ext, nodes, 6, m, offset=np.ones(6, dtype=np.int32))
    c2c = op2.Map(ext, prisms, 1, (np.arange(n) * cells).astype(np.int32).reshape(-1, 1),
                  offset=np.ones(1, dtype=np.int32))
    xv = rng.integers(-9, 10, nodes.size).astype(dtype)
    x, o = op2.Dat(nodes, xv, dtype), op2.Dat(prisms, dtype=dtype)
    t = C[dtype]
    k = op2.Kernel("static void g(%s *o, const %s *x) { o[0] = x[0] + 2 * x[1] - x[2] + 3 * x[3] "
                   "+ x[4] - 2 * x[5]; }" % (t, t), "g")
    op2.par_loop(k, ext, o(op2.WRITE, c2c), x(op2.READ, mp))
    w = np.array([1, 2, -1, 3, 1, -2], dtype=dtype)
    idx = m[:, None, :] + np.arange(cells)[None, :, None]
    vals = np.where(m[:, None, :] >= 0, xv[np.where(m[:, None, :] >= 0, idx, 0)], 0)
    assert np.array_equal(o.data_ro, (vals * w).sum(-1).astype(dtype).reshape(-1))
