"""Transforms of many lines against the same lines a few at a time: the tile (lines and threads a CTA) is chosen by
the number of lines, and no line's result depends on it beyond rounding.

Every transform is within 4e-15 log2 N of the largest value of its output, so two of them agree to 1e-13."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# pairs of lines, tiles of 4 .. 16 lines that are all resident, launches that fill the GPU several times over; the
# transform in the slot and (N - 1 odd, twice an odd power of three, or several factors) out of it; ragged last tiles
@pytest.mark.parametrize("n,lines", [(34, 5), (49, 3649), (65, 5001), (65, 20003), (129, 10007), (163, 4999), (244, 3651),
                                     (513, 3003), (769, 9001), (1025, 4001), (1537, 2051), (2049, 701), (2049, 2501)])
@pytest.mark.parametrize("axis", [0, 1])
def test_lines_do_not_depend_on_the_tile(n, lines, axis):
    from pypde_gb300 import Base
    b = Base(n, "CH")
    g = torch.Generator(device="cuda").manual_seed(n + lines)
    f = torch.rand((n, lines) if axis == 0 else (lines, n), dtype=torch.float64, device="cuda", generator=g) - 0.5
    if axis:
        f = f.t()
    for fn in (b.forward_fft, b.backward_fft):
        y = fn(f)
        for at in (0, 300 * (lines // 600), max(0, lines - 77)):
            part = fn(f[:, at:at + 300])
            assert (y[:, at:at + 300] - part).abs().max() <= 1e-13 * part.abs().max()
