"""The vector kernels behind Dat arithmetic (op2g_vec_op, op2g_vec_dot): every
element type, lengths around a 16-byte pack and a grid, aligned and offset
arrays, operands that alias, ghosts, threads on streams of their own, and the
operands that take the par_loop instead."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = ["float64", "float32", "int32", "int64", "uint32", "uint64"]
LENGTHS = [0, 1, 2, 3, 5, 255, 4097, 152 * 512 * 2 + 3, 1_500_001]


def dat(op2, s, v, offset):
    """A Dat over v whose array starts `offset` elements into an allocation
    (offset 1 is not 16-byte aligned; torch has no 32/64-bit unsigned here)."""
    if not offset or v.dtype.name.startswith("u"):
        return op2.Dat(s, v, v.dtype)
    import torch
    base = torch.from_numpy(np.concatenate([v[:1], v])).cuda()
    return op2.Dat.from_tensor(s ** 1, base[1:])


def assert_sum(got, A, B):
    """Exact but for float32, whose whole numbers end at 2^24: there the bound
    of test_inner_of_reals."""
    if A.dtype == np.float32:
        ref = np.dot(A.astype(np.float64), B.astype(np.float64))
        assert abs(float(got) - ref) <= 64 * 2.0 ** -24 * abs(ref)
    else:
        assert got == (A * B).sum(dtype=A.dtype)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", LENGTHS)
def test_operations(gpu_op2, dtype, offset, n):
    op2 = gpu_op2
    rng = np.random.default_rng(n)
    s = op2.Set(n)
    A = rng.integers(1, 50, n).astype(dtype)
    B = rng.integers(1, 9, n).astype(dtype)
    if n == 0:
        offset = 0
    a, b = dat(op2, s, A, offset), op2.Dat(s, B, dtype)
    div = np.divide if dtype.startswith("f") else np.floor_divide
    three = A.dtype.type(3)
    for got, want in ((a + b, A + B), (a - b, A - B), (a * b, A * B), (a / b, div(A, B)),
                      (a + 3, A + three), (a - 3, A - three), (a * 3.9, None), (a / 3, div(A, three)),
                      (-a, -A), (a + a, A + A), (a / a, div(A, A))):
        if want is None:     # a scalar is converted to the Dat's type first
            want = A * A.dtype.type(3.9)
        assert got.dtype == A.dtype
        assert np.array_equal(got.data_ro, want)
    assert_sum(a.inner(b), A, B)
    assert_sum(a.inner(a), A, A)
    a += b
    a *= a
    a -= 2
    b /= b
    W = (A + B) * (A + B) - A.dtype.type(2)
    assert np.array_equal(a.data_ro, W)
    assert np.array_equal(b.data_ro, np.ones_like(B))
    assert_sum(a.inner(b), W, np.ones_like(W))


def test_inner_of_reals(gpu_op2):
    """Against a sum in extended precision: n products and as many additions
    in any order are off by at most n eps sum |a b|; a tree is far below."""
    op2 = gpu_op2
    rng = np.random.default_rng(0)
    for dtype, eps in (("float64", 2.0 ** -53), ("float32", 2.0 ** -24)):
        A, B = (rng.uniform(-1, 1, 777_777).astype(dtype) for _ in range(2))
        s = op2.Set(len(A))
        a, b = op2.Dat(s, A, dtype), op2.Dat(s, B, dtype)
        ref = np.sum(A.astype(np.longdouble) * B.astype(np.longdouble))
        bound = 64 * eps * float(np.sum(np.abs(A.astype(np.float64) * B)))
        got = a.inner(b)
        assert got.dtype == A.dtype and abs(float(got - ref)) <= bound
        assert got == a.inner(b)
        assert abs(a.norm - np.sqrt(float(np.sum(A.astype(np.float64) ** 2)))) <= 64 * eps * a.norm


def test_ghosts_and_multi_dim(gpu_op2):
    op2 = gpu_op2
    s = op2.Set((3, 7, 9))
    A = np.arange(1.0, 28.0).reshape(9, 3)
    a, b = op2.Dat(s ** 3, A), op2.Dat(s ** 3, 2 * A)
    r = a + b
    assert np.array_equal(r.data_ro_with_halos[:7], 3 * A[:7]) and not r.data_ro_with_halos[7:].any()
    a *= b
    assert np.array_equal(a.data_ro_with_halos[:7], 2 * A[:7] ** 2)
    assert np.array_equal(a.data_ro_with_halos[7:], A[7:])
    assert b.inner(b) == (4 * A[:7] ** 2).sum()
    v = a.dat_version
    a += 1.0
    assert a.dat_version == v + 1 and not a.halo_valid


def test_operands_that_take_the_loop(gpu_op2):
    op2 = gpu_op2
    s, t = op2.Set(6), op2.Set(6)
    a, f = op2.Dat(s, np.arange(6.0)), op2.Dat(s, np.arange(6), np.float32)
    i = op2.Dat(s, np.arange(6), np.int16)
    assert np.array_equal((a + f).data_ro, 2 * np.arange(6.0))
    assert np.array_equal((i + i).data_ro, 2 * np.arange(6))
    with pytest.raises(Exception):
        i.inner(i)          # no 16-bit Global reductions
    with pytest.raises(op2.MapValueError if hasattr(op2, "MapValueError") else Exception):
        a + op2.Dat(t, np.arange(6.0))
    with a.frozen_halo(op2.READ):
        with pytest.raises(RuntimeError):
            a += 1.0
    with pytest.raises(Exception):
        a + np.arange(3.0)
    a += 1.0
    assert np.array_equal(a.data_ro, np.arange(6.0) + 1)


def test_threads(gpu_op2):
    """Products and sums of several threads, each on a stream of its own."""
    import threading
    import torch
    op2 = gpu_op2
    n = 200_003
    out = {}

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            s = op2.Set(n)
            a = op2.Dat(s, np.full(n, float(k)))
            got = []
            for _ in range(20):
                b = a * 2.0
                b += a
                got.append(float(b.inner(a)))
            out[k] = got
    ts = [threading.Thread(target=work, args=(k,)) for k in range(1, 5)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k in range(1, 5):
        assert out[k] == [3.0 * k * k * n] * 20
