"""GPU: the fixed-point DCT-I against a long double transform, at the lengths, tiles and values where it
can go wrong.

Bound, derived: a line is scaled so that its absolute sum is at least 2^57 units (numbers below the
normal range count as 2^-1023).  Each stage of the FFT rounds within 2 units, which the later ones
amplify by the root of their lengths' product: at most about 2 sqrt(N) units for a spectrum point, and
the odd outputs sum the errors of at most N/2 increments about their mean, sqrt(N) of them in size, twice
that at the worst of N outputs.  So every output is within 4 N 2^-57 sum|x| and its own rounding,
2^-53 |y|.  Beside a line whose points are all of one size, a line goes down by that line's log2(N)
bits: N max|x| in place of its sum.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = ("RAW", "FWD", "BWD", "FWD_T", "BWD_T")


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from pypde_gb300 import _lib
    return torch, _lib


def scales(mode, n):
    """(pre, post) of a mode around the raw transform."""
    N, k = n - 1, np.arange(n)
    end = (k == 0) | (k == N)
    sg = np.where(k % 2, -1.0, 1.0)
    one = np.ones(n)
    return {"RAW": (one, one), "FWD": (one, sg * np.where(end, 0.5, 1.0) / N), "BWD": (sg * np.where(end, 1.0, 0.5), one),
            "FWD_T": (sg * 0.5 / N, np.where(end, 1.0, 2.0)), "BWD_T": (np.where(end, 1.0, 0.5), sg)}[mode]


def reference(x, mode):
    """Lines of x along axis 1, in long double."""
    n = x.shape[1]
    pre, post = (np.asarray(v, dtype=np.longdouble) for v in scales(mode, n))
    v = x.astype(np.longdouble) * pre
    j = np.arange(n)
    ang = ((np.outer(j, j) % (2 * (n - 1))).astype(np.longdouble)) / (n - 1)
    C = np.cos(ang * np.longdouble("3.14159265358979323846264338327950288")) * 2
    C[:, 0] = 1
    C[:, -1] = np.where(j % 2, -1, 1)
    y = np.stack([(C * line).sum(axis=1) for line in v])
    return y * post, np.abs(v).sum(axis=1, keepdims=True) * np.abs(post), (n - 1) * np.abs(v).max(axis=1, keepdims=True) * np.abs(post)


def run(env, x, mode, tb, nthreads, flags=0, slots=1):
    """LOAD, DCT, STORE of the lines of x (the C ABI); ``slots`` arrays through one multi-slot op."""
    torch, _lib = env
    L = _lib.lib()
    xs = [torch.as_tensor(np.roll(x, s, axis=0).copy(), device="cuda") for s in range(slots)]
    ys = [torch.full_like(t, 7.0) for t in xs]
    nl, n = x.shape
    tab = ctypes.c_void_p()
    _lib.check(L.pgx_dct_table(n, ctypes.byref(tab)), "dct table")
    P, inst = _lib.PgxProgram(), _lib.PgxInstance()
    P.axis, P.lines_len, P.tb, P.lcap, P.nslots, P.fft_n, P.nthreads = 1, 1, tb, (n + 1) | 1, slots, n, nthreads
    ops = [_lib.op("LOAD", a=s, arr=2 * s, len=0) for s in range(slots)]
    ops.append(_lib.op("DCT", a=0, b=slots, mat=0, k=getattr(_lib, "DCT_" + mode) | flags))
    ops += [_lib.op("STORE", a=s, arr=2 * s + 1) for s in range(slots)]
    P.nops = len(ops)
    for i, o in enumerate(ops):
        P.ops[i] = o
    for s in range(slots):
        for a, t in ((2 * s, xs[s]), (2 * s + 1, ys[s])):
            inst.arr[a].ptr, inst.arr[a].s0, inst.arr[a].s1 = t.data_ptr(), n, 1
            inst.arr[a].n0, inst.arr[a].n1 = nl, n
    inst.len[0], inst.len[1], inst.mat[0] = n, nl, tab.value
    _lib.check(L.pgx_run(ctypes.byref(P), ctypes.byref(inst), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
               "pgx_run")
    torch.cuda.synchronize()
    return [np.roll(y.cpu().numpy(), -s, axis=0) for s, y in enumerate(ys)]


def check(x, mode, got, mixed=False):
    ref, size, most = reference(x, mode)
    n = x.shape[1]
    size = most if mixed else size
    size = np.maximum(size, (n - 1) * 2.0 ** -1023)
    bound = 4 * (n - 1.0) * 2.0 ** -57 * size + 2.0 ** -53 * np.abs(ref) + 5e-324
    for y in got:
        assert np.all(np.abs(y - ref) <= bound), float(np.max(np.abs(y - ref) / bound))


KINDS = ("noise", "decay", "spike", "mixed")


def lines(n, nl, kind):
    """Noise, decaying spectra, single large points, or all three beside each other; any size per line."""
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (nl, n))
    decay, spike = {"noise": (0, 0), "decay": (1, 0), "spike": (0, 1), "mixed": (3, 3)}[kind]
    if decay:
        x[1 % decay::decay] *= np.exp(-20.0 * np.arange(n) / n)
    if spike:
        x[2 % spike::spike] *= 1e-6
        x[2 % spike::spike, n // 3] = 1.0
    return x * 10.0 ** rng.integers(-12, 12, (nl, 1))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n", [3, 5, 7, 13, 17, 25, 33, 37, 49, 55, 65, 97, 129, 145, 163, 193, 257, 385])
def test_lengths_and_modes(env, n, mode):
    """Every build (2^a and 3 2^a points) and the general stages, in the warp-local form, the CTA-wide form
    with an odd tile, and three slots at once."""
    for kind in KINDS:
        x = lines(n, 11, kind)
        check(x, mode, run(env, x, mode, 4, 32), kind == "mixed")
        check(x, mode, run(env, x, mode, 3, 128), kind == "mixed")
        check(x, mode, run(env, x, mode, 2, 64, slots=3), kind == "mixed")


@pytest.mark.parametrize("tb,nthreads", [(2, 64), (4, 32), (2, 256)])
@pytest.mark.parametrize("n", [17, 49, 97, 193, 385, 513, 769])
def test_in_the_slot(env, n, tb, nthreads):
    """The result in the slot after an odd number of stages, in the spare after an even one (385, 769)."""
    _, _lib = env
    for kind in KINDS:
        x = lines(n, 7, kind)
        check(x, "BWD", run(env, x, "BWD", tb, nthreads, flags=_lib.DCT_SLOT), kind == "mixed")


@pytest.mark.parametrize("n", [513, 769, 1025, 1537, 2049])
def test_long_lines(env, n):
    for mode, kind in (("FWD", "noise"), ("BWD", "decay"), ("FWD", "mixed")):
        x = lines(n, 5, kind)
        check(x, mode, run(env, x, mode, 2, 256), kind == "mixed")
        check(x, mode, run(env, x, mode, 1, 128))


@pytest.mark.parametrize("n", [17, 97, 193, 513])
def test_values_at_the_limits(env, n):
    """Lines at both ends of the exponent range, subnormal, zero and constant ones; a NaN or an infinity
    makes its own line NaN and no other."""
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, (12, n))
    x[0] *= 2.0 ** 1000
    x[1] *= 2.0 ** -1000
    x[2] *= 2.0 ** -1060
    x[3] = 0.0
    x[4] = 1.0
    x[5] = 2.0 ** 1023
    x[6, 3], x[7, n - 1], x[8, 0] = np.nan, np.inf, -np.inf
    x[9] = 0.0
    x[9, n // 2] = 5e-324
    got = run(env, x, "RAW", 4, 64)[0]
    assert np.isnan(got[6:9]).all() and not np.isnan(np.delete(got, [6, 7, 8], axis=0)).any()
    assert not got[3].any()
    assert got[5, 0] == np.inf and np.all(np.abs(got[5, 1:]) < 2.0 ** 1023)  # the sum overflows, the rest cancels
    ok = [0, 1, 2, 4, 9, 10, 11]
    check(x[ok], "RAW", [got[ok]], mixed=True)
