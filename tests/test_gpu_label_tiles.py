"""Labelling across the tiles of its shared-memory pass (128 x 64 pixels, wider for images of a few rows),
the 32-pixel runs and the segments of the numbering (1024 words of 32 pixels), against the oracle.  Whole
numbers: equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _serpentine(shape):
    """One component that crosses every tile border many times: rows joined at alternating ends."""
    a = np.zeros(shape, np.uint8)
    a[::2] = 1
    a[1::4, -1] = 1
    a[3::4, 0] = 1
    return a


def _patterns(shape, rng):
    yield "ones", np.ones(shape, np.uint8)
    yield "serpentine", _serpentine(shape)
    yield "serpentine down", np.ascontiguousarray(_serpentine(shape[::-1]).T)
    for density in (0.4, 0.6, 0.9):
        yield f"noise {density}", (rng.random(shape) < density).astype(np.uint8)
    yield "diagonals", (np.add.outer(np.arange(shape[0]), np.arange(shape[1])) % 3 == 0).astype(np.uint8)


def _check(a, se, flat):
    from poutre2_gb300 import label
    from poutre2_gb300.se import Common_NL_SE
    out = torch.empty(a.shape, dtype=torch.int64, device="cuda")
    f = label.label_flat_zones if flat else label.label_binary
    n = f(torch.from_numpy(a).cuda(), Common_NL_SE[se], out)
    exp, m = oracle.label(a, se, flat)
    assert n == m
    np.testing.assert_array_equal(out.cpu().numpy(), exp)


@pytest.mark.parametrize("shape", [(1, 8193), (2, 4097), (5, 2047), (33, 64), (63, 129), (64, 128), (65, 127), (97, 31), (300, 1), (191, 513)])
@pytest.mark.parametrize("se", ["SESquare2D", "SECross2D", "SESegmentY2D"])
def test_tiles_2d(shape, se):
    rng = np.random.default_rng(shape[0] * 8191 + shape[1])
    for name, a in _patterns(shape, rng):
        for flat in (False, True):
            _check(a, se, flat)
    _check(rng.integers(-3, 4, shape).astype(np.int32), se, False)  # a negative pixel joins no later one


@pytest.mark.parametrize("n", [1, 31, 33, 8191, 8193, 70001])
def test_tiles_1d(n):
    rng = np.random.default_rng(n)
    for density in (0.5, 0.999, 1.1):
        a = (rng.random(n) < density).astype(np.uint16)
        _check(a, "SESegmentX1D", False)
        _check(a, "SESegmentX1D", True)


@pytest.mark.parametrize("shape", [(3, 33, 65), (9, 64, 64), (40, 2, 130), (5, 70, 31)])
@pytest.mark.parametrize("se", ["SECross3D", "SESegmentX3D", "SESegmentY3D", "SESegmentZ3D"])
def test_tiles_3d(shape, se):
    rng = np.random.default_rng(sum(shape))
    for density in (0.3, 0.7, 1.1):
        a = (rng.random(shape) < density).astype(np.uint8)
        _check(a, se, False)
        _check(a, se, True)


def test_many_segments():
    # 9.4 Mpixel, 288 segments of the numbering; output on an odd 8-byte word
    from poutre2_gb300 import label
    from poutre2_gb300.se import Common_NL_SE
    a = (np.random.default_rng(3).random((3000, 3137)) < 0.45).astype(np.uint8)
    exp, m = oracle.label(a, "SESquare2D", False)
    buf = torch.empty(a.size + 1, dtype=torch.int64, device="cuda")
    out = buf[1:].view(a.shape)
    assert label.label_binary(torch.from_numpy(a).cuda(), Common_NL_SE.SESquare2D, out) == m
    np.testing.assert_array_equal(out.cpu().numpy(), exp)


def test_doubled_segments():
    # rows of one pixel take a bitmap word each: 2.2 M words are more than 2048 segments of 1024
    from poutre2_gb300 import label
    from poutre2_gb300.se import Common_NL_SE
    a = (np.random.default_rng(4).random((2_200_003, 1)) < 0.7).astype(np.uint8)
    exp, m = oracle.label(a, "SECross2D", False)
    out = torch.empty(a.shape, dtype=torch.int64, device="cuda")
    assert label.label_binary(torch.from_numpy(a).cuda(), Common_NL_SE.SECross2D, out) == m
    np.testing.assert_array_equal(out.cpu().numpy(), exp)
