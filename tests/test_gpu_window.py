"""The window kernel (boxes and segments of any half length, any row length and alignment) against the oracle,
bit-exact: half lengths around the powers of two its windows are built from, widths around its tiles
(120 words of 4, 2 or 1 pixels), heights around its 64-row tiles, misaligned buffers, infinities."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

DTYPES = [np.uint8, np.uint16, np.int32, np.float32]


def _image(shape, dt, seed):
    rng = np.random.default_rng(seed)
    if np.dtype(dt).kind == "f":
        a = rng.standard_normal(shape).astype(dt)
        a[rng.random(shape) < 0.01] = -np.inf
        a[rng.random(shape) < 0.01] = np.inf
        return a
    info = np.iinfo(dt)
    return rng.integers(info.min, info.max, shape, dtype=dt, endpoint=True)


def _device(a, offset):
    """The image in a buffer that starts `offset` pixels past an aligned address."""
    buf = torch.empty(a.size + offset, dtype=torch.from_numpy(a).dtype, device="cuda")
    x = buf[offset:].view(a.shape)
    x.copy_(torch.from_numpy(a))
    return x


def _window(a, offsets, dilate):
    """Clipped window extremum by a list of offsets; like the kernels, a window that is clipped also holds the
    type's lowest (highest) finite value."""
    lo = np.finfo(a.dtype).min if a.dtype.kind == "f" else np.iinfo(a.dtype).min
    hi = np.finfo(a.dtype).max if a.dtype.kind == "f" else np.iinfo(a.dtype).max
    ry, rx = max(abs(o[0]) for o in offsets), max(abs(o[1]) for o in offsets)
    p = np.pad(a, ((ry, ry), (rx, rx)), constant_values=lo if dilate else hi)
    out = None
    for dy, dx in offsets:
        v = p[ry + dy:ry + dy + a.shape[0], rx + dx:rx + dx + a.shape[1]]
        out = v.copy() if out is None else (np.maximum if dilate else np.minimum)(out, v)
    return out


def _box(a, hy, hx, dilate):
    return _window(_window(a, [(0, t) for t in range(-hx, hx + 1)], dilate), [(t, 0) for t in range(-hy, hy + 1)], dilate)


def _run(a, se, dilate, offset=0):
    from poutre2_gb300 import llm
    x = _device(a, offset)
    out = _device(np.zeros_like(a), offset)
    (llm.DilateSE if dilate else llm.ErodeSE)(x, se, out)
    return out.cpu().numpy()


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("hy,hx", [(1, 2), (2, 1), (3, 5), (4, 4), (6, 0), (0, 6), (8, 9), (10, 10), (12, 3), (16, 17),
                                   (30, 29), (0, 32), (32, 0), (33, 2), (63, 1), (1, 31)])
def test_boxes(dt, hy, hx):
    from poutre2_gb300 import llm
    for shape in ((16, 3), (65, 121), (64, 241), (131, 487), (70, 1000)):
        a = _image(shape, dt, hy * 64 + hx)
        for dilate in (True, False):
            np.testing.assert_array_equal(_run(a, llm.se_rect(hy, hx), dilate), _box(a, hy, hx, dilate), err_msg=f"{shape}")


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("dy,dx", [(1, 0), (-1, 1), (1, 1)])
@pytest.mark.parametrize("half", [2, 4, 5, 8, 9, 13, 20, 31, 40, 63])
def test_segments(dt, dy, dx, half):
    from poutre2_gb300 import llm
    offsets = [(t * dy, t * dx) for t in range(-half, half + 1)]
    for shape in ((17, 5), (64, 119), (67, 483), (200, 301)):
        a = _image(shape, dt, half)
        for dilate in (True, False):
            np.testing.assert_array_equal(_run(a, llm.se_line(dy, dx, half), dilate), _window(a, offsets, dilate),
                                          err_msg=f"{shape}")


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_misaligned_buffers(dt, offset):
    from poutre2_gb300 import llm
    for shape in ((40, 480), (33, 479), (33, 482)):
        a = _image(shape, dt, offset)
        np.testing.assert_array_equal(_run(a, llm.se_rect(5, 6), True, offset), _box(a, 5, 6, True))
        np.testing.assert_array_equal(_run(a, llm.se_line(1, -1, 6), False, offset),
                                      _window(a, [(t, -t) for t in range(-6, 7)], False))


@pytest.mark.parametrize("dt", [np.uint8, np.int32, np.float32])
def test_against_the_oracle(dt):
    from poutre2_gb300 import llm
    rng = np.random.default_rng(9)
    a = rng.integers(0, 200, (150, 333)).astype(dt)
    np.testing.assert_array_equal(_run(a, llm.se_rect(9, 9), True), oracle.dilate(a, "SESquare2D", 9))
    np.testing.assert_array_equal(_run(a, llm.se_rect(9, 9), False), oracle.erode_dilate_static(a, "SESquare2D", 9, False))
