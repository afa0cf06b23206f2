"""The forms of the sparsity build's row kernel against numpy: a warp per row
with 1 to 8 candidates per lane, a lane per row (large meshes), rows with more
distinct columns than a lane's table takes, rows with more candidates than
either form takes, and what the transpose list holds (flat, constant layers,
codes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LARGE = 152 * 20 * 32 + 77      # rows from which a lane takes a row, and a ragged batch


def pattern(pairs, nrows, ncols, diag):
    """(rowptr, colidx) of the (rows [n, a], cols [n, b]) pairs."""
    keys = [np.arange(min(nrows, ncols), dtype=np.int64) * (ncols + 1)] if diag else []
    for r, c in pairs:
        r, c = r[:, :, None].astype(np.int64), c[:, None, :].astype(np.int64)
        keep = np.broadcast_to((r >= 0) & (c >= 0), (len(r), r.shape[1], c.shape[2]))
        keys.append((r * ncols + c)[keep])
    k = np.unique(np.concatenate(keys))
    return np.concatenate([[0], np.cumsum(np.bincount(k // ncols, minlength=nrows))]), k % ncols


def check(sp, ref):
    rp, ci = sp.csr()
    assert np.array_equal(rp, ref[0])
    assert np.array_equal(ci, ref[1])


def near(rng, n, arity, size, window):
    """Map values within `window` of a base that sweeps the target set."""
    base = (np.arange(n, dtype=np.int64) * size // n)[:, None]
    return np.clip(base + rng.integers(-window, window + 1, (n, arity)), 0, size - 1).astype(np.int32)


# rows, cells per row, arity, window: candidates per row about cells * arity^2,
# distinct columns up to 4 * window + 1
@pytest.mark.parametrize("rows,cells,arity,window", [
    (1, 1, 1, 0), (33, 1, 3, 3), (500, 3, 4, 4), (700, 6, 4, 8), (900, 2, 7, 9),
    (1200, 7, 4, 40), (3000, 3, 8, 60), (300, 5, 9, 100),
    (LARGE, 2, 4, 2), (LARGE, 2, 4, 5), (LARGE, 2, 3, 7), (LARGE, 3, 4, 30), (LARGE, 1, 8, 12)])
@pytest.mark.parametrize("hub", [False, True])
def test_one_flat_map(gpu_op2, rows, cells, arity, window, hub):
    op2 = gpu_op2
    rng = np.random.default_rng(rows + arity)
    n = max(1, rows * cells // arity) if rows > 1 else 1
    m = near(rng, n, arity, rows, window)
    m[rng.random(m.shape) < 0.01] = -1
    if hub:                      # a row that many cells name: more than 256 candidates
        m[:: max(1, n // 300), 0] = rows // 2
    cset, vset = op2.Set(n), op2.Set(rows)
    mp = op2.Map(cset, vset, arity, m)
    sp = op2.Sparsity((vset ** 1, vset ** 1), [(mp, mp, None)])
    check(sp, pattern([(m, m)], rows, rows, True))


@pytest.mark.parametrize("rows,cols", [(400, 90), (LARGE, 5000), (90, LARGE)])
def test_two_maps(gpu_op2, rows, cols):
    """Row and column maps differ (rectangular; no diagonal, or a square pair
    whose diagonal is no candidate), arities 3 and 5."""
    op2 = gpu_op2
    rng = np.random.default_rng(rows)
    n = rows
    r, c = near(rng, n, 3, rows, 3), near(rng, n, 5, cols, 3)
    cset, rset, kset = op2.Set(n), op2.Set(rows), op2.Set(cols)
    rm, cm = op2.Map(cset, rset, 3, r), op2.Map(cset, kset, 5, c)
    check(op2.Sparsity((rset ** 1, kset ** 1), [(rm, cm, None)]), pattern([(r, c)], rows, cols, False))
    c2 = near(rng, n, 5, rows, 3)
    cm2 = op2.Map(cset, rset, 5, c2)
    check(op2.Sparsity((rset ** 1, rset ** 1), [(rm, cm2, None)]), pattern([(r, c2)], rows, rows, True))
    # two pairs with a common number of columns, and with different ones
    check(op2.Sparsity((rset ** 1, rset ** 1), [(rm, rm, None), (cm2, rm, None)]),
          pattern([(r, r), (c2, r)], rows, rows, True))
    check(op2.Sparsity((rset ** 1, rset ** 1), [(rm, rm, None), (cm2, cm2, None)]),
          pattern([(r, r), (c2, c2)], rows, rows, True))


@pytest.mark.parametrize("columns,levels", [(40, 5), (LARGE // 16 + 3, 16)])
@pytest.mark.parametrize("layers", ["constant", "raised", "ragged"])
def test_extruded(gpu_op2, columns, levels, layers):
    op2 = gpu_op2
    rng = np.random.default_rng(columns)
    base = near(rng, columns, 3, columns, 2)
    m = np.concatenate([base * levels, base * levels + 1], axis=1).astype(np.int32)
    lay = np.zeros((columns, 2), dtype=np.int32)
    if layers == "ragged":
        lay[:, 1] = rng.integers(2, levels + 1, columns)
    else:
        lay[:, 1] = levels
    arg = levels if layers == "constant" else lay
    cells = op2.ExtrudedSet(op2.Set(columns), arg)
    nodes = op2.Set(columns * levels)
    mp = op2.Map(cells, nodes, 6, m, offset=np.ones(6, dtype=np.int32))
    sp = op2.Sparsity((nodes ** 1, nodes ** 1), [(mp, mp, None)])
    full = []
    for k in range(levels - 1):
        rows = m[lay[:, 1] - 1 > k] + k
        full.append((rows, rows))
    check(sp, pattern(full, columns * levels, columns * levels, True))


@pytest.mark.parametrize("rows", [300, LARGE])
def test_composed(gpu_op2, rows):
    """A composed map gives the pattern of its composition."""
    op2 = gpu_op2
    rng = np.random.default_rng(rows)
    n = rows // 2
    m = near(rng, n, 4, rows, 4)
    pick = rng.permutation(n).astype(np.int32)[: n - 5]
    cset, vset, sub = op2.Set(n), op2.Set(rows), op2.Set(len(pick))
    outer, inner = op2.Map(cset, vset, 4, m), op2.Map(sub, cset, 1, pick)
    comp = op2.ComposedMap(outer, inner)
    sp = op2.Sparsity((vset ** 1, vset ** 1), [(comp, comp, None)])
    check(sp, pattern([(m[pick], m[pick])], rows, rows, True))
