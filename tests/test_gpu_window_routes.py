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


def _extremum(a, offsets, dilate):
    info = np.finfo(a.dtype) if a.dtype.kind == "f" else np.iinfo(a.dtype)
    ry, rx = (max(abs(o[i]) for o in offsets) for i in (0, 1))
    p = np.pad(a, ((ry, ry), (rx, rx)), constant_values=info.min if dilate else info.max)
    out = None
    for dy, dx in offsets:
        v = p[ry + dy:ry + dy + a.shape[0], rx + dx:rx + dx + a.shape[1]]
        out = v.copy() if out is None else (np.maximum if dilate else np.minimum)(out, v, out=out)
    return out


def _check(a, se, passes, dilate):
    from poutre2_gb300 import llm
    x = torch.from_numpy(a).cuda()
    out = torch.empty_like(x)
    (llm.DilateSE if dilate else llm.ErodeSE)(x, se, out)
    want = a
    for offsets in passes:
        want = _extremum(want, offsets, dilate)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("dt", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("shape", [(60000, 8), (60000, 7), (3000, 8), (20000, 64), (20000, 130), (1239, 48)])
def test_boxes_on_narrow_images(dt, shape):
    from poutre2_gb300 import llm
    a = np.random.default_rng(1).integers(0, 250, shape).astype(dt)
    for hy, hx in ((2, 2), (10, 3), (2, 9)):
        rows, cols = [(t, 0) for t in range(-hy, hy + 1)], [(0, t) for t in range(-hx, hx + 1)]
        _check(a, llm.se_rect(hy, hx), (cols, rows), hy != 2)


@pytest.mark.parametrize("dt", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("shape", [(30000, 144), (30000, 21), (18000, 6), (3000, 21), (900, 2900), (1520, 5856), (300, 400)])
def test_segments_on_narrow_and_wide_images(dt, shape):
    from poutre2_gb300 import llm
    a = np.random.default_rng(2).integers(0, 250, shape).astype(dt)
    for dy, dx, half in ((1, 0, 9), (1, 0, 20), (1, 1, 5), (0, 1, 4)):
        _check(a, llm.se_line(dy, dx, half), ([(t * dy, t * dx) for t in range(-half, half + 1)],), half != 9)
