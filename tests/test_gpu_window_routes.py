"""Boxes and segments on images so narrow that a window is wider than the image."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _vertical(a, hy, dilate):
    """Extremum over 2 hy + 1 rows; a window that is clipped also holds the type's lowest (highest) finite value."""
    info = np.finfo(a.dtype) if a.dtype.kind == "f" else np.iinfo(a.dtype)
    p = np.pad(a, ((hy, hy), (0, 0)), constant_values=info.min if dilate else info.max)
    op = np.maximum if dilate else np.minimum
    return op.reduce([p[t:t + a.shape[0]] for t in range(2 * hy + 1)])


@pytest.mark.parametrize("dt", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("hy,hx", [(0, 2), (0, 6), (5, 2), (3, 7), (12, 1), (31, 30)])
@pytest.mark.parametrize("rows", [16, 100, 1000])
def test_one_column(dt, hy, hx, rows):
    # a row window clipped to the pixel itself adds nothing: infinities stay where no row is clipped
    from poutre2_gb300 import llm
    rng = np.random.default_rng(rows + hy)
    a = rng.integers(0, 200, (rows, 1)).astype(dt)
    if dt == np.float32:
        a[rng.random(a.shape) < 0.9] = -np.inf
        a[rows // 3:rows // 3 * 2] = np.inf
    x = torch.from_numpy(a).cuda()
    out = torch.empty_like(x)
    for dilate in (True, False):
        (llm.DilateSE if dilate else llm.ErodeSE)(x, llm.se_rect(hy, hx), out)
        np.testing.assert_array_equal(out.cpu().numpy(), _vertical(a, hy, dilate))
