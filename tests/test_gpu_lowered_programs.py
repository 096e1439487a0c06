"""GPU: programs whose neighbouring ops a launch merges, or between which it drops the barrier, against NumPy.

The merged forms do the operations of the separate ones in the same order, so results agree to the rounding
of the derivative's partial sums: at most n additions of n values, 2^-53 n^2 relative to the largest.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from pypde_gb300 import _lib
    return torch, _lib


def run(env, ops, arrays, lens, axis, tb, nthreads, sten):
    """pgx_run of ``ops`` (code, {fields}) on arrays stored with lines along ``axis``; returns them."""
    torch, _lib = env
    L = _lib.lib()
    dev = [torch.as_tensor(np.ascontiguousarray(a.T if axis == 0 else a), device="cuda") for a in arrays]
    table = torch.as_tensor(sten, device="cuda")
    P, inst = _lib.PgxProgram(), _lib.PgxInstance()
    P.axis, P.lines_len, P.tb, P.lcap, P.nslots, P.fft_n, P.nthreads = axis, 0, tb, (max(lens[1:]) + 3) | 1, 3, 0, nthreads
    P.nops = len(ops)
    for i, (code, f) in enumerate(ops):
        P.ops[i] = _lib.op(code, **f)
    for i, t in enumerate(dev):
        A = inst.arr[i]
        A.ptr, A.s0, A.s1, A.n0, A.n1 = t.data_ptr(), t.stride(0), t.stride(1), t.shape[0], t.shape[1]
    for i, n in enumerate(lens):
        inst.len[i] = n
    inst.mat[0] = table.data_ptr()
    inst.par[0] = 0.375
    _lib.check(L.pgx_run(ctypes.byref(P), ctypes.byref(inst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "pgx_run")
    torch.cuda.synchronize()
    return [t.cpu().numpy().T if axis == 0 else t.cpu().numpy() for t in dev]


def stencil(v, sten):
    u = np.zeros((v.shape[0], v.shape[1] + 2))
    u[:, :-2] += v
    u[:, 2:] += sten[:v.shape[1]] * v
    return u


def diff(c):
    n = c.shape[1]
    d = np.zeros_like(c)
    for j in range(n - 2, -1, -1):
        d[:, j] = (d[:, j + 2] if j + 2 < n else 0.0) + 2.0 * (j + 1) * c[:, j + 1]
    d[:, 0] *= 0.5
    return d


@pytest.mark.parametrize("axis,tb,nthreads", [(1, 1, 32), (0, 1, 256), (1, 2, 64), (0, 3, 128), (1, 8, 128)])
@pytest.mark.parametrize("n,lines", [(3, 1), (4, 5), (17, 7), (64, 3), (65, 9), (130, 4)])
def test_merged_ops_and_dropped_barriers(env, n, lines, axis, tb, nthreads):
    rng = np.random.default_rng(n)
    sten = -rng.uniform(0.5, 1.0, n + 4)
    x, z = rng.uniform(-1, 1, (lines, n)), np.full((lines, n + 2), 7.0)
    lens = [lines, n, n + 2, n - 2]
    tol = 2.0 ** -53 * (n + 2) ** 2 * 4.0

    def near(got, want):
        assert np.max(np.abs(got - want)) <= tol * max(np.max(np.abs(want)), 1.0)

    # LOAD STENCIL | COPY DIFF SCALE | two STOREs
    ops = [("LOAD", dict(a=0, arr=0, len=1)), ("STENCIL", dict(a=0, mat=0)), ("COPY", dict(a=1, b=0)),
           ("DIFF", dict(a=1, k=1)), ("SCALE", dict(a=1, par=0)), ("STORE", dict(a=0, arr=1)), ("STORE", dict(a=1, arr=2))]
    got = run(env, ops, [x, z, z], lens, axis, tb, nthreads, sten)
    u = stencil(x, sten)
    near(got[1], u)
    near(got[2], 0.375 * diff(u))
    # a factor keeps LOAD and STENCIL apart, two derivatives COPY and DIFF; DIFF SCALE in place
    ops = [("LOAD", dict(a=0, arr=0, len=1, alpha=-2.0)), ("STENCIL", dict(a=0, mat=0)), ("COPY", dict(a=1, b=0)),
           ("DIFF", dict(a=1, k=2)), ("DIFF", dict(a=0, k=1)), ("SCALE", dict(a=0, alpha=0.5)),
           ("STORE", dict(a=0, arr=1)), ("STORE", dict(a=1, arr=2))]
    got = run(env, ops, [x, z, z], lens, axis, tb, nthreads, sten)
    near(got[1], -diff(u))
    near(got[2] / (n + 2) ** 2, -2.0 * diff(diff(u)) / (n + 2) ** 2)
    # a length cut and grown again leaves zeros; an array stored and loaded back; a slot never loaded is zero
    ops = [("LOAD", dict(a=0, arr=0, len=1)), ("SETLEN", dict(a=0, len=3)), ("SETLEN", dict(a=0, len=2)),
           ("STORE", dict(a=0, arr=1)), ("LOAD", dict(a=1, arr=1, len=2)), ("SCALE", dict(a=1, alpha=3.0)),
           ("STORE", dict(a=1, arr=1)), ("LOAD", dict(a=1, arr=1, len=2)), ("AXPY", dict(a=2, b=1, alpha=1.0)),
           ("AXPY", dict(a=2, b=0, alpha=-1.0)), ("STORE", dict(a=2, arr=2))]
    got = run(env, ops, [x, z, z], lens, axis, tb, nthreads, sten)
    cut = np.zeros((lines, n + 2))
    cut[:, :n - 2] = x[:, :n - 2]
    near(got[1], 3.0 * cut)
    near(got[2], 2.0 * cut)
