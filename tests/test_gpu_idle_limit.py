"""The bounded wait of a resident tile (brick) that has nothing to do counts from the last progress anywhere: a path that
winds through the whole image or volume for many times the limit is followed to its end."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture()
def limit():
    from poutre2_gb300 import _lib
    L = _lib.load()
    yield lambda ns: L.pg_debug_set_limits(0, ns)
    assert L.pg_debug_set_limits(0, 0) == 0


def _path(shape, dt):
    """A corridor of value 100 along every second row, joined at alternating ends (and from slice to slice)."""
    f = np.zeros(shape, dt)
    flat = f.reshape((-1,) + shape[-2:])
    for z in range(0, flat.shape[0], 2):
        rows = range(0, shape[-2], 2)
        for i, r in enumerate(rows):
            flat[z, r] = 100
            if i + 1 < len(rows):
                flat[z, r + 1, -1 if i % 2 == 0 else 0] = 100
        if z + 2 < flat.shape[0]:  # from this slice's last corridor end, or its first one, to the next slice
            r = rows[-1] if z % 4 == 0 else 0
            flat[z + 1, r, (-1 if len(rows) % 2 else 0) if z % 4 == 0 else 0] = 100
    return f


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("shape", [(2200, 2200), (64, 96, 256)])
def test_a_path_longer_than_the_limit(limit, shape, dt):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    f = _path(shape, dt)
    m = np.zeros_like(f)
    m[(0,) * len(shape)] = 100
    x, k = torch.from_numpy(m).cuda(), torch.from_numpy(f).cuda()
    out = torch.empty_like(k)
    se = Common_NL_SE.SECross2D if len(shape) == 2 else Common_NL_SE.SECross3D

    def run():
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        geo.Reconstruction(geo.reconstruction_type.dilate, x, k, se, out)  # raises if the kernel gave up
        b.record()
        b.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), f)
        return a.elapsed_time(b)

    ms = run()
    assert limit(int(ms * 1e6 / 10)) == 0
    run()
