"""GPU: the DENSE op in digits on the FP16 tensor cores (PGX_DENSE_TC) against long double products.

Bound, derived: rows and lines are rounded at 2^-63 of their power-of-two scale (at most twice the largest
value), the digit pairs left out (i + j <= 5) sum to at most 7 products of 2^14 256^5 2^-124 a column, and
the result is rounded once: |error| <= cols (2^-61 + 2^-64) max|row| max|line| + 2^-53 |y|, cols columns all of one sign.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import pypde_gb300
    return pypde_gb300


def apply(A, x, axis, tb=8, nthreads=128, more=()):
    """LOAD, DENSE, ``more``, STORE of the columns of x (lines along ``axis``) through pgx_run."""
    import ctypes
    import torch
    from pypde_gb300 import _lib
    from pypde_gb300.navier.fused import dense_dev
    (rows, cols), lines = A.shape, x.shape[1]
    table = dense_dev(A)
    dev = [torch.as_tensor(np.ascontiguousarray(v if axis == 0 else v.T), device="cuda") for v in (x, np.full((rows, lines), 7.0))]
    P, inst = _lib.PgxProgram(), _lib.PgxInstance()
    P.axis, P.lines_len, P.tb, P.lcap, P.nslots, P.fft_n, P.nthreads = axis, 0, tb, (max(rows, cols) + 1) | 1, 1, 0, nthreads
    ops = [("LOAD", dict(a=0, arr=0, len=1)), ("DENSE", dict(a=0, mat=0, len=2, k=_lib.DENSE_TC)), *more,
           ("STORE", dict(a=0, arr=1))]
    P.nops = len(ops)
    for i, (code, f) in enumerate(ops):
        P.ops[i] = _lib.op(code, **f)
    for i, t in enumerate(dev):
        a = inst.arr[i]
        a.ptr, a.s0, a.s1, a.n0, a.n1 = t.data_ptr(), t.stride(0), t.stride(1), t.shape[0], t.shape[1]
    inst.len[0], inst.len[1], inst.len[2], inst.mat[0] = lines, cols, rows, table.data_ptr()
    _lib.check(_lib.lib().pgx_run(ctypes.byref(P), ctypes.byref(inst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "pgx_run")
    torch.cuda.synchronize()
    y = dev[1].cpu().numpy()
    return y if axis == 0 else y.T


def check(A, x, y):
    ref = A.astype(np.longdouble) @ x.astype(np.longdouble)
    size = np.abs(A).max(axis=1, keepdims=True).astype(np.longdouble) * np.abs(x).max(axis=0, keepdims=True)
    bound = A.shape[1] * (2.0 ** -61 + 2.0 ** -64) * size + 2.0 ** -53 * np.abs(ref) + 5e-324
    assert np.all(np.abs(y - ref) <= bound), float(np.max(np.abs(y - ref) / bound))


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("rows,cols,lines", [(1, 1, 1), (2, 5, 3), (15, 17, 8), (16, 16, 9), (17, 33, 1), (48, 50, 50),
                                             (127, 129, 20), (128, 128, 64), (130, 145, 7), (255, 257, 33),
                                             (511, 513, 40), (300, 1025, 5)])
def test_shapes(pg, rows, cols, lines, axis):
    """Edges of the 16 x 16 blocks, of the eight lines and of the 128 columns between two roundings, rows split
    over CTAs; all-ones operands, whose digit sums are the largest, and columns and lines of any size."""
    rng = np.random.default_rng(rows * 1000 + cols)
    A = rng.standard_normal((rows, cols)) * 10.0 ** rng.integers(-8, 8, (rows, 1))
    x = rng.uniform(-1, 1, (cols, lines)) * 10.0 ** rng.integers(-8, 8, (1, lines))
    check(A, x, apply(A, x, axis))
    check(A, x, apply(A, x, axis, tb=3, nthreads=256))
    # not split over CTAs: another op behind it (a length that stays)
    check(A, x, apply(A, x, axis, tb=12, nthreads=64, more=[("SETLEN", dict(a=0, len=2))]))
    A, x = np.full((rows, cols), -(1.0 - 2.0 ** -9)), np.full((cols, lines), 1.0 - 2.0 ** -7)
    check(A, x, apply(A, x, axis))
    A = A * rng.uniform(0.5, 1.0, A.shape)
    x = x * np.exp(-10.0 * np.arange(cols) / cols)[:, None]
    check(A, x, apply(A, x, axis))


@pytest.mark.parametrize("rows,cols,lines", [(511, 513, 511), (100, 129, 500), (63, 65, 300)])
def test_public_operator_on_both_sides_of_the_rule(pg, rows, cols, lines):
    """MatrixApply takes the digits from 456 lines on and FP64 chains below."""
    import torch
    from pypde_gb300.bases import MatrixApply
    rng = np.random.default_rng(rows)
    A, x = rng.standard_normal((rows, cols)), rng.uniform(-1, 1, (cols, lines))
    y = MatrixApply(A).apply(torch.as_tensor(x, device="cuda"), 0).cpu().numpy()
    ref = A.astype(np.longdouble) @ x.astype(np.longdouble)
    assert np.all(np.abs(y - ref) <= cols * 2.0 ** -53 * (np.abs(A) @ np.abs(x)))


def test_values_at_the_limits(pg):
    """Zero, subnormal and huge lines; a NaN or an infinity in a line or a row gives what the plain products give
    there and nothing elsewhere."""
    rng = np.random.default_rng(0)
    A = rng.uniform(-1, 1, (40, 50))
    x = rng.uniform(-1, 1, (50, 12))
    x[:, 0] = 0.0
    x[:, 1] *= 2.0 ** -1065
    x[:, 2] *= 2.0 ** 1015
    clean = [k for k in range(12) if k not in (4, 5)]
    x[3, 4], x[7, 5] = np.nan, np.inf
    y = apply(A, x, 0)
    assert not y[:, 0].any() and np.isnan(y[:, 4]).all()
    assert np.array_equal(y[:, 5], np.copysign(np.inf, A[:, 7]))
    check(A, x[:, clean], y[:, clean])
    A[5, 6] = np.inf
    y = apply(A, x[:, clean], 0)
    assert np.isnan(y[5, 0]) and np.isinf(y[5, 1:]).all() and np.isfinite(np.delete(y, 5, axis=0)).all()
