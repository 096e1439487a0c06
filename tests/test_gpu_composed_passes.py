"""The one-pass compositions (stencil with transform or derivative, forward and transposed) against the same maps
taken as two passes through the library's own entry points.

Both run the same operators on the same data, so they differ by rounding only: each transform's own error is below
4e-15 of the largest value of its line times log2 N, and the derivative's and the mass solve's operators are the same
ops.  The tolerance is 1e-13 of the largest output (a derivative's rows grow like N^2 and share one norm)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _base(key, N, **kw):
    from pypde_gb300 import Base
    return Base(N, key, **kw)


def _lines(n, lines, layout, seed):
    """A line array of one of the layouts that the calls take: row-major, transposed, every second column of a
    wider one, or one line."""
    rng = np.random.default_rng(seed)
    if layout == "one":
        return torch.as_tensor(rng.uniform(-1, 1, n), dtype=F64, device="cuda")
    if layout == "transposed":
        return torch.as_tensor(rng.uniform(-1, 1, (lines, n)), dtype=F64, device="cuda").t()
    if layout == "strided":
        return torch.as_tensor(rng.uniform(-1, 1, (n, 2 * lines + 1)), dtype=F64, device="cuda")[:, 1::2]
    return torch.as_tensor(rng.uniform(-1, 1, (n, lines)), dtype=F64, device="cuda")


def _near(a, b):
    assert a.shape == b.shape and a.dtype == b.dtype
    assert (a - b).abs().max() <= 1e-13 * max(1e-300, float(b.abs().max()))


def _both_ways(one, two, x, seed):
    """Values and vector-Jacobian products of the one-pass and the two-pass form."""
    got = []
    for fn in (one, two):
        v = x.detach().requires_grad_(True)
        y = fn(v)
        w = torch.as_tensor(np.random.default_rng(seed).uniform(-1, 1, tuple(y.shape)), dtype=F64, device="cuda")
        got.append((fn(x), y, torch.autograd.grad(y, v, w)[0]))
    for a, b in zip(*got):
        _near(a.detach(), b.detach())


# the dense form (N <= 33 and few lines; lengths with other factors than 2 and 3 at any size), the FFT in the slot
# and (N - 1 odd, or twice an odd power of three) out of it, more lines than SMs, than warps for their chains, and
# the many-line dense form
SIZES = [(5, 1), (6, 7), (17, 33), (33, 9), (34, 40), (50, 48), (65, 2), (97, 65), (129, 511), (193, 300), (132, 460),
         (33, 1300), (1025, 5), (1535, 3), (28, 30), (55, 20), (163, 31), (244, 12), (129, 5000), (2049, 3)]


@pytest.mark.parametrize("key", ["CD", "CN"])
@pytest.mark.parametrize("N,lines", SIZES)
@pytest.mark.parametrize("layout", ["rows", "transposed", "strided", "one"])
def test_composed_maps(key, N, lines, layout):
    b = _base(key, N)
    v = _lines(N - 2, lines, layout, N)
    _both_ways(b.backward_fft, lambda x: b.family.backward_fft(b.to_chebyshev(x)), v, 1)
    for d in (1, 2):
        _both_ways(lambda x: b.derivative(x, d), lambda x: b.family.derivative(b.to_chebyshev(x), d), v, 2)
    f = _lines(N, lines, layout, N + 1)
    _both_ways(b.forward_fft, lambda x: b.from_chebyshev(b.family.forward_fft(x)), f, 3)
    short = f[:N - 1]
    _both_ways(b.forward_fft, lambda x: b.from_chebyshev(b.family.forward_fft(x)), short, 4)


@pytest.mark.parametrize("N,lines", [(17, 20), (33, 33), (50, 75), (129, 193), (89, 500)])
def test_values_on_a_longer_grid(N, lines):
    from pypde_gb300.field import _values
    b = _base("CN", N, dealias=3 / 2)
    v = _lines(N - 2, lines, "transposed", N)
    _both_ways(lambda x: _values(b, b.dealias, x), lambda x: b.dealias.family._dct(b.to_chebyshev(x), 2), v, 5)


def test_what_was_refused_is_refused():
    b = _base("CD", 33)
    with pytest.raises(AssertionError):
        b.backward_fft(torch.zeros(32, 4, dtype=F64, device="cuda"))
    with pytest.raises(AssertionError):
        b.derivative(torch.zeros(33, 4, dtype=F64, device="cuda"), 1)
    with pytest.raises(ValueError):
        b.forward_fft(torch.zeros(34, 4, dtype=F64, device="cuda"))
    with pytest.raises(NotImplementedError):
        b.backward_fft(torch.zeros(31, 4, 2, dtype=F64, device="cuda"))
    with pytest.raises(RuntimeError):  # no lines: an empty tensor has no address
        b.backward_fft(torch.zeros(31, 0, dtype=F64, device="cuda"))
    with pytest.raises(RuntimeError):
        b.family.backward_fft(b.to_chebyshev(torch.zeros(31, 0, dtype=F64, device="cuda")))


def test_a_base_with_its_own_stencil_keeps_it():
    from pypde_gb300.bases import ChebDirichlet

    class Doubled(ChebDirichlet):
        def to_chebyshev(self, vhat):
            return 2.0 * ChebDirichlet.to_chebyshev(self, vhat)

    v = _lines(31, 9, "rows", 1)
    _near(Doubled(33).backward_fft(v), 2.0 * _base("CD", 33).backward_fft(v))
