"""The warp scan with its maps from the table (PGX_CHAIN_SCAN) against the scan that composes them on the way: the
same maps meet the same states in the same order, so the values are the same bits."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _factors(rng, n, systems):
    t = rng.uniform(-0.6, 0.6, (systems, 4, n))
    t[:, 1] = 1.0 / rng.uniform(1.0, 3.0, (systems, n))
    t[:, 0, :2] = 0.0
    t[:, 2, n - 2:] = 0.0
    t[:, 3, max(n - 4, 0):] = 0.0
    return t.ravel()


def _run(code, n, lines, table, x, flags, slots, threads):
    from pypde_gb300 import _lib
    L = _lib.lib()
    P, I = _lib.PgxProgram(), _lib.PgxInstance()
    P.axis, P.lines_len, P.nslots, P.tb, P.lcap, P.nthreads = 1, 0, slots, 3, (n + 1) | 1, threads
    I.len[0], I.len[1] = lines, n
    y = torch.empty_like(x)
    ops = []
    for s in range(slots):
        I.mat[s] = table.data_ptr()
        for k, t in ((2 * s, x[s]), (2 * s + 1, y[s])):
            a = I.arr[k]
            a.ptr, a.s0, a.s1, a.n0, a.n1 = t.data_ptr(), n, 1, lines, n
        ops.append(_lib.op("LOAD", a=s, arr=2 * s, len=1))
    ops.append(_lib.op(code, a=0, b=slots, mat=0, k=flags))
    ops += [_lib.op("STORE", a=s, arr=2 * s + 1) for s in range(slots)]
    P.nops = len(ops)
    for i, o in enumerate(ops):
        P.ops[i] = o
    _lib.check(L.pgx_run(ctypes.byref(P), ctypes.byref(I), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return y


# one unknown a lane or none, ragged segments, the longest line; one slot and several
@pytest.mark.parametrize("n", [4, 5, 7, 31, 32, 33, 63, 64, 65, 66, 127, 129, 255, 511, 1000, 2104])
@pytest.mark.parametrize("lines", [1, 7])
@pytest.mark.parametrize("code", ["FDMA", "FDMA_T", "POISSON", "POISSON_T"])
def test_maps_from_the_table_give_the_same_bits(n, lines, code):
    from pypde_gb300 import _lib
    from pypde_gb300.navier.fused import chain_dev
    rng = np.random.default_rng(n + lines)
    table = chain_dev(_factors(rng, n, lines if code.startswith("POIS") else 1), n)
    slots = 1 if code.startswith("POIS") or n > 1000 else 2
    x = torch.as_tensor(rng.uniform(-1, 1, (slots, lines, n)), dtype=F64, device="cuda")
    for threads in (32, 224):
        a = _run(code, n, lines, table, x, _lib.CHAIN_WARP, slots, threads)
        b = _run(code, n, lines, table, x, _lib.CHAIN_WARP | _lib.CHAIN_SCAN, slots, threads)
        assert torch.isfinite(a).all() and torch.equal(a, b)
