"""Launch shapes of register-heavy wrappers and of Mat insertion: sizes around
the change between the balanced entry, CTAs of 64 threads and one CTA per
block, flat and extruded, through a Subset, against an explicit grid (which
takes none of these) and, for whole numbers, exactly."""
import numpy as np
import pytest

from pyop2_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# 60 independent accumulators per cell keep more than 64 registers in use
HEAVY = """
static void heavy(double *y, const double *x)
{
  double a[60];
  for (int i = 0; i < 60; ++i) a[i] = x[i % 4] + i;
  for (int r = 0; r < 3; ++r)
    for (int i = 0; i < 60; ++i) a[i] = a[i] + a[(i + 7) % 60] - a[(i + 11) % 60];
  double s = 0.0;
  for (int i = 0; i < 60; ++i) s += a[i] * (i % 5 - 2);
  for (int i = 0; i < 4; ++i) y[i] += s + i;
}
"""


@pytest.mark.parametrize("cells", [1, 63, 65, 38_911, 38_913, 77_825, 89_000, 155_647, 155_649,
                                   311_297, 700_001])
@pytest.mark.parametrize("subset", [False, True])
def test_heavy_flat_loop(gpu_op2, cells, subset):
    """Whole-number arithmetic, so every order of the sums is exact."""
    op2 = gpu_op2
    rng = np.random.default_rng(cells)
    verts = op2.Set(max(4, cells // 3))
    cset = op2.Set(cells)
    m = op2.Map(cset, verts, 4, rng.integers(0, verts.size, (cells, 4)))
    x = op2.Dat(verts, rng.integers(-3, 4, verts.size).astype(float))
    it = op2.Subset(cset, np.arange(0, cells, 2)) if subset else cset
    k = op2.Kernel(HEAVY, "heavy")
    out = []
    for grid in (0, 11):
        y = op2.Dat(verts)
        lp = op2.ParLoop(k, it, y(op2.INC, m), x(op2.READ, m))
        lp.build(0, 256, 0, grid)
        lp.compute()
        out.append(y.data_ro.copy())
    assert np.any(out[0])
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("n,cells", [(7, 5), (30, 20), (40, 32), (63, 10), (50, 33)])
def test_prism_assembly_and_action(gpu_op2, n, cells):
    op2 = gpu_op2
    p = W.build_prisms(op2, n=n, layers=cells + 1, seed=n)
    nodes, c2n, c2c = p["nodes"], p["c2n"], p["c2c"]
    ds = op2.DataSet(nodes, (p["nrhs"], 3))
    u = op2.Dat(ds, p["u"])
    sp = op2.Sparsity((nodes ** 3, nodes ** 3), [(c2n, c2n, None)])
    res = []
    for grid in (0, 152 * 7):
        y, A = op2.Dat(ds), op2.Mat(sp)
        act = op2.ParLoop(op2.Kernel(W.PRISM_ELASTICITY_ACTION, "prism_elasticity"), p["cells"],
                          y(op2.INC, c2n), p["X"](op2.READ, c2n), u(op2.READ, c2n),
                          p["L"](op2.READ, c2c))
        asm = op2.ParLoop(op2.Kernel(W.PRISM_ELASTICITY_MATRIX, "prism_elasticity_mat"),
                          p["cells"], A(op2.INC, (c2n, c2n)), p["X"](op2.READ, c2n),
                          p["L"](op2.READ, c2c))
        for lp in (act, asm):
            lp.build(0, 256, 0, grid)
            lp.compute()
        A.assemble()
        res.append((y.data_ro.copy(), A.tensor.cpu().numpy()))
    for a, b in zip(*res):
        # the same terms in another order: at most 24 prisms meet in a node
        # pair, so 64 roundings of the largest partial sum bound the difference
        assert np.max(np.abs(a - b)) <= 64 * 2.0 ** -52 * np.max(np.abs(b))
