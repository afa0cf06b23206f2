"""Increments of neighbouring cells combined in a warp before they reach
memory: targets shared by none, two, four or all lanes, cells that name a
target twice, negative entries, ragged ends, subsets, several components and
types, kernels on both sides of the rule for doubles.  Whole numbers, so every
order of the sums is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = {"float64": "double", "float32": "float", "int32": "int", "int64": "long long"}
BODY = {"plain": "y[i * %(D)d + j] += x[0];",              # moves data: combined
        "product": "y[i * %(D)d + j] += x[0] * (i + 2);"}   # doubles: not combined


def targets(rng, n, arity, size, shared):
    if shared == "all":
        return np.full((n, arity), size // 2, dtype=np.int32)
    m = rng.integers(0, size, (n, arity)).astype(np.int32)
    if shared in (2, 3, 4, 6):       # runs of cells share their even entries
        m[:, ::2] = m[np.arange(n) // shared * shared][:, ::2]
    if shared == "twice":
        m[:, -1] = m[:, 0]
    if shared == "negative":
        m[rng.random(m.shape) < 0.3] = -1
    return m


@pytest.mark.parametrize("dtype", ["float64", "float32", "int32", "int64"])
@pytest.mark.parametrize("shared", ["none", 2, 3, 4, 6, "all", "twice", "negative"])
@pytest.mark.parametrize("n,arity,dim", [(1, 1, 1), (31, 4, 1), (33, 3, 2), (4_097, 4, 4),
                                         (4_097, 4, 5), (200_003, 4, 1)])
def test_increments(gpu_op2, dtype, shared, n, arity, dim):
    op2 = gpu_op2
    rng = np.random.default_rng(n + dim)
    size = max(3, n // 5)
    m = targets(rng, n, arity, size, shared)
    cells, verts = op2.Set(n), op2.Set(size)
    mp = op2.Map(cells, verts, arity, m)
    xv = rng.integers(-3, 4, n).astype(dtype)
    x = op2.Dat(cells, xv, dtype)
    t = C[dtype]
    sub = np.arange(0, n, 3)
    for kind, body in BODY.items():
        src = ("static void inc(%s *y, const %s *x) { for (int i = 0; i < %d; ++i) for (int j = 0; "
               "j < %d; ++j) %s }" % (t, t, arity, dim, body % {"D": dim}))
        k = op2.Kernel(src, "inc")
        scale = np.arange(arity) + 2 if kind == "product" else np.ones(arity, dtype=int)
        for it, rows in ((cells, np.arange(n)), (op2.Subset(cells, sub), sub)):
            y = op2.Dat(verts ** dim, dtype=dtype)
            op2.par_loop(k, it, y(op2.INC, mp), x(op2.READ))
            ref = np.zeros(size, dtype=np.int64)
            v = m[rows]
            np.add.at(ref, v[v >= 0], (xv[rows][:, None] * scale).astype(np.int64)[v >= 0])
            got = y.data_ro.reshape(size, dim)
            assert np.array_equal(got, np.repeat(ref[:, None], dim, axis=1).astype(dtype))
