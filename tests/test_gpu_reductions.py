"""Global reductions: pure reduction loops (several iterations loaded together,
one resident wave) and loops that also move data, from one entity to several
sweep steps of every thread, per-warp and per-CTA atomics, more components than
the CTA reduction takes, several CTA sizes.  Whole numbers, so sums are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = {"float64": "double", "float32": "float", "int32": "int", "int64": "long long"}
WAVE = 152 * 2048


@pytest.mark.parametrize("n", [0, 1, 31, 257, 9_999, 65_537, 8 * WAVE - 1, 8 * WAVE + 1, 3_000_001])
@pytest.mark.parametrize("dtype", ["float64", "float32", "int32", "int64"])
@pytest.mark.parametrize("dim", [1, 3])
def test_sum_min_max(gpu_op2, n, dtype, dim):
    op2 = gpu_op2
    rng = np.random.default_rng(n + dim)
    v = rng.integers(-2, 3, (n, dim))
    v[n // 2:n // 2 + 1, 0] = 41
    v[-1:, dim - 1] = -43
    s = op2.Set(n)
    d = op2.Dat(s ** dim, v, dtype)
    t = C[dtype]
    k = op2.Kernel("static void red(const %s *a, %s *s, %s *lo, %s *hi) { for (int i = 0; i < %d; "
                   "++i) { s[0] += a[i]; if (a[i] < lo[0]) lo[0] = a[i]; if (a[i] > hi[0]) "
                   "hi[0] = a[i]; } }" % (t, t, t, t, dim), "red")
    tot, lo, hi = (op2.Global(1, x, dtype) for x in (5, 0, 1))
    for block in (256, 32, 64):
        lp = op2.ParLoop(k, s, d(op2.READ), tot(op2.INC), lo(op2.MIN), hi(op2.MAX))
        lp.build(0, block, 0, 0)
        lp.compute()
    assert tot.data_ro[0] == 5 + 3 * v.sum()
    assert lo.data_ro[0] == (min(0, v.min()) if n else 0)
    assert hi.data_ro[0] == (max(1, v.max()) if n else 1)


@pytest.mark.parametrize("n", [100, 700_001])
@pytest.mark.parametrize("comps", [1, 16, 17])
def test_components_and_written_data(gpu_op2, n, comps):
    """A loop that writes a Dat and reduces `comps` components (16 is the
    largest CTA reduction), and the same over a Subset."""
    op2 = gpu_op2
    s = op2.Set(n)
    v = np.arange(n) % 7 - 3.0
    d, o = op2.Dat(s, v), op2.Dat(s)
    k = op2.Kernel("static void red(double *o, const double *a, double *g) { o[0] = 2 * a[0]; "
                   "for (int i = 0; i < %d; ++i) g[i] += a[0] * (i - 4); }" % comps, "red")
    for it, pick in ((s, np.arange(n)), (op2.Subset(s, np.arange(0, n, 3)), np.arange(0, n, 3))):
        g = op2.Global(comps, np.zeros(comps))
        op2.par_loop(k, it, o(op2.WRITE), d(op2.READ), g(op2.INC))
        assert np.array_equal(g.data_ro, v[pick].sum() * (np.arange(comps) - 4.0))
        assert np.array_equal(o.data_ro[pick], 2 * v[pick])


def test_infinities_and_nan(gpu_op2):
    """Compares with NaN are false: a NaN entry changes neither extreme."""
    op2 = gpu_op2
    v = np.array([np.nan, -np.inf, 3.0, np.inf, np.nan] * 50_000)
    s = op2.Set(len(v))
    d = op2.Dat(s, v)
    k = op2.Kernel("static void ext(const double *a, double *lo, double *hi) { if (a[0] < lo[0]) "
                   "lo[0] = a[0]; if (a[0] > hi[0]) hi[0] = a[0]; }", "ext")
    lo, hi = op2.Global(1, 0.0), op2.Global(1, np.finfo(np.float64).min)
    op2.par_loop(k, s, d(op2.READ), lo(op2.MIN), hi(op2.MAX))
    assert lo.data_ro[0] == -np.inf and hi.data_ro[0] == np.inf
