"""CSR products through bulk copies (op2g_mat_spmv_sized) against the lane
kernel bit for bit (the same sums in the same order) and against numpy: row
counts around a batch of 32, ragged and empty rows, batches too long for the
buffer, last batches whose rounded copies would leave the arrays, value arrays
that are not aligned, infinite x entries, and sizes the rule leaves to the lane
kernel."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 330_000          # enough batches for every warp of 152 SMs to have two


def matrix(rng, nrows, kind):
    n = {"even": np.full(nrows, 15), "short": np.full(nrows, 2),
         "ragged": rng.integers(0, 21, nrows), "empty": np.zeros(nrows, dtype=int),
         "long": rng.integers(5, 9, nrows)}[kind]
    if kind == "long":
        n[rng.integers(0, nrows, 40)] = 1500
        n[-1] = 900
    if kind == "empty":
        n[::37] = 3
    rp = np.concatenate([[0], np.cumsum(n)])
    ci = rng.integers(0, nrows, rp[-1]).astype(np.int32)
    return rp.astype(np.int64), ci, rng.integers(-4, 5, rp[-1]).astype(float)


def product(nblocks, rp, ci, v, x, ncols, transpose):
    import torch
    from pyop2_gb300 import _lib, device
    b = _lib.BCSR()
    b.nrows, b.ncols, b.rdim, b.cdim = len(rp) - 1, ncols, 1, 1
    b.rowptr, b.colidx, b.values = rp.data_ptr(), ci.data_ptr(), v.data_ptr()
    y = torch.zeros(ncols if transpose else b.nrows, dtype=torch.float64, device="cuda")
    _lib.call("op2g_mat_spmv_sized", ctypes.byref(b), nblocks, x.data_ptr(), y.data_ptr(),
              int(transpose), device.stream_handle())
    return y


@pytest.mark.parametrize("kind", ["even", "short", "ragged", "empty", "long"])
@pytest.mark.parametrize("nrows", [ROWS, ROWS + 1, ROWS + 31, 4_000])
@pytest.mark.parametrize("offset", [0, 1])
def test_csr(gpu_op2, kind, nrows, offset):
    import torch
    rng = np.random.default_rng(nrows)
    rp, ci, v = matrix(rng, nrows, kind)
    x = rng.integers(-9, 10, nrows).astype(float)
    dev = [torch.as_tensor(a, device="cuda") for a in (rp, ci)]
    dv = torch.as_tensor(np.concatenate([v[:offset], v]), device="cuda")[offset:]
    dx = torch.as_tensor(x, device="cuda")
    got = product(len(ci), dev[0], dev[1], dv, dx, nrows, False)
    lane = product(-1, dev[0], dev[1], dv, dx, nrows, False)
    assert torch.equal(got, lane)
    rows = np.repeat(np.arange(nrows), np.diff(rp))
    ref = np.bincount(rows, v * x[ci], nrows)          # whole numbers: exact
    assert np.array_equal(got.cpu().numpy(), ref)
    t = product(len(ci), dev[0], dev[1], dv, dx, nrows, True)
    assert np.array_equal(t.cpu().numpy(), np.bincount(ci, v * x[rows], nrows))


def test_infinite_entry_reaches_its_rows_only(gpu_op2):
    import torch
    rng = np.random.default_rng(1)
    rp, ci, v = matrix(rng, ROWS, "ragged")
    v[v == 0] = 1.0
    x = np.zeros(ROWS)
    x[7] = np.inf
    d = [torch.as_tensor(a, device="cuda") for a in (rp, ci, v, x)]
    y = product(len(ci), d[0], d[1], d[2], d[3], ROWS, False).cpu().numpy()
    rows = np.repeat(np.arange(ROWS), np.diff(rp))
    hit = np.unique(rows[ci == 7])
    assert len(hit) and not np.isfinite(y[hit]).any()
    assert np.isfinite(np.delete(y, hit)).all()
