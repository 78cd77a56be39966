"""Labelling of narrow images (tiles of 32 x 256 pixels, a single column as a row) and of thin volumes (several slices a
tile): around the sides of those tiles and the number of slices that fit, against the oracle.  Whole numbers: equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _check(a, se, flat):
    from poutre2_gb300 import label
    from poutre2_gb300.se import Common_NL_SE
    out = torch.empty(a.shape, dtype=torch.int64, device="cuda")
    f = label.label_flat_zones if flat else label.label_binary
    n = f(torch.from_numpy(a).cuda(), Common_NL_SE[se], out)
    exp, m = oracle.label(a, se, flat)
    assert n == m
    np.testing.assert_array_equal(out.cpu().numpy(), exp)


def _images(shape):
    rng = np.random.default_rng(sum(shape))
    yield np.ones(shape, np.uint8)
    for density in (0.3, 0.6, 0.9):
        yield (rng.random(shape) < density).astype(np.uint8)
    yield rng.integers(0, 3, shape).astype(np.uint16)
    yield (np.indices(shape).sum(0) % 5 < 2).astype(np.uint8)
    yield rng.integers(0, 256, shape).astype(np.uint8)  # nearly every pixel its own flat zone: dense bitmap words


@pytest.mark.parametrize("shape", [(1, 1), (255, 1), (257, 1), (1000, 3), (256, 31), (513, 32), (257, 33), (128, 64), (129, 63), (300, 65)])
@pytest.mark.parametrize("se", ["SESquare2D", "SECross2D", "SESegmentX2D", "SESegmentY2D"])
def test_narrow_images(shape, se):
    for a in _images(shape):
        for flat in (False, True):
            _check(a, se, flat)


@pytest.mark.parametrize("shape", [(1, 1, 1), (300, 1, 1), (70, 3, 5), (33, 8, 8), (32, 8, 32), (9, 31, 33), (5, 128, 17), (4, 255, 3),
                                   (3, 257, 32), (7, 21, 64), (5, 64, 65), (3, 65, 130), (2, 33, 200), (40, 2, 1000), (400, 8, 8), (700, 5, 33), (350, 1, 40), (310, 70, 2)])
@pytest.mark.parametrize("se", ["SECross3D", "SESegmentX3D", "SESegmentY3D", "SESegmentZ3D"])
def test_thin_volumes(shape, se):
    for a in _images(shape):
        for flat in (False, True):
            _check(a, se, flat)
    _check(np.random.default_rng(1).integers(-3, 4, shape).astype(np.int32), se, False)  # a negative pixel joins no later one
