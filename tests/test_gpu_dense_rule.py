"""Dense operators through the C calls on both sides of the rule that sends them to the tensor cores: thin ones,
few lines, ragged rows and columns, against NumPy.

Either form's error is below 2e-15 of |A| |x| a row (FP64 chains of up to 400 products; the digits are closer), so the
tolerance is 1e-14 of its largest value."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(2, 257), (257, 2), (31, 400), (32, 400), (65, 65), (131, 133), (207, 209), (209, 208),
                                       (255, 257), (400, 385)])
@pytest.mark.parametrize("lines", [1, 8, 33, 153, 305, 457])
@pytest.mark.parametrize("axis", [0, 1])
def test_dense_operator(rows, cols, lines, axis):
    from pypde_gb300.bases import MatrixApply
    rng = np.random.default_rng(rows + cols + lines)
    A, x = rng.standard_normal((rows, cols)), rng.standard_normal((cols, lines))
    b = torch.as_tensor(x if axis == 0 else np.ascontiguousarray(x.T), device="cuda")
    y = MatrixApply(A).apply(b, axis).cpu().numpy()
    y = y if axis == 0 else y.T
    assert np.abs(y - A @ x).max() <= 1e-14 * (np.abs(A) @ np.abs(x)).max()
