"""Neighbour lists through their chords (runs of offsets along a row) against the oracle, bit-exact: disks, lists
without the centre, chords longer than a pass takes, far and repeated offsets, volumes; widths around the tiles
(480 u8, 240 u16, 120 f32 pixels) and heights around their 24, 32 or 8 rows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

DTYPES = [np.uint8, np.uint16, np.int32, np.float32]


def _disk(r):
    return [(y, x) for y in range(-r, r + 1) for x in range(-r, r + 1) if y * y + x * x <= r * r + r]


LISTS = {
    "disk2": _disk(2), "disk5": _disk(5), "disk9": _disk(9),
    "ring": [o for o in _disk(6) if o not in _disk(4)],
    "one-sided": [(y, x) for y in range(0, 4) for x in range(-9, 1 - 2 * y)],
    "long row": [(0, x) for x in range(-70, 71)] + [(1, x) for x in range(-5, 90)],
    "tall": [(y, x) for y in (-60, -59, 0, 60) for x in range(-3, 4)],
    "far": [(0, x) for x in range(400, 420)] + [(-300, x) for x in range(-2, 3)] + [(20, x) for x in range(-1200, -1180)],
    "repeated": _disk(3) + _disk(3) + [(0, 0)],
}


def _check(a, offsets):
    from poutre2_gb300 import llm
    from poutre2_gb300.se import NeighborList
    x, nl = torch.from_numpy(a).cuda(), NeighborList(offsets)
    for dilate in (True, False):
        out = torch.empty_like(x)
        (llm.Dilate if dilate else llm.Erode)(x, nl, out)
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.erode_dilate_nl(a, offsets, dilate), err_msg=f"{a.shape}")


def _image(shape, dt, rng):
    if np.dtype(dt).kind == "f":
        return rng.standard_normal(shape).astype(dt)
    info = np.iinfo(dt)
    return rng.integers(info.min, info.max, shape, dtype=dt, endpoint=True)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("name", sorted(LISTS))
def test_images(dt, name):
    rng = np.random.default_rng(len(name))
    for shape in ((16, 1), (33, 121), (31, 239), (65, 483)):
        _check(_image(shape, dt, rng), LISTS[name])


@pytest.mark.parametrize("dt", [np.uint8, np.float32])
def test_larger_image(dt):
    _check(_image((700, 1501), dt, np.random.default_rng(1)), _disk(4))  # 24- and 32-row tiles


@pytest.mark.parametrize("dt", DTYPES)
def test_volumes(dt):
    rng = np.random.default_rng(7)
    ball = [(z, y, x) for z in range(-3, 4) for y in range(-3, 4) for x in range(-3, 4) if z * z + y * y + x * x <= 12]
    for shape in ((1, 16, 9), (5, 17, 130), (9, 40, 61)):
        _check(_image(shape, dt, rng), ball)
        _check(_image(shape, dt, rng), [(2, 0, x) for x in range(-4, 5)] + [(-1, y, x) for y in (-2, 2) for x in range(0, 6)])


def test_a_list_of_scattered_offsets_is_gathered():
    # no two offsets in a row: the chords would cost more than the offsets
    rng = np.random.default_rng(2)
    offs = [(int(y), int(x)) for y, x in rng.integers(-20, 21, (40, 2))]
    for dt in DTYPES:
        _check(_image((50, 77), dt, rng), offs)
