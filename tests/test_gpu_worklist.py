"""The tile worklist beyond what the resident kernels hold: 1- and 2-byte images of a few tiles more than 32 an SM (markers,
erosions, effective masks and clips of the levelings, rows of no whole words), and the give-up paths of the worklist and
of the resident volumes."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

NOT_CONVERGED = 9


def _plateaus(shape, dt, seed):
    rng = np.random.default_rng(seed)
    a = np.kron(rng.integers(0, 40, ((shape[0] + 10) // 11, (shape[1] + 12) // 13)), np.ones((11, 13), np.int64))
    a = a[:shape[0], :shape[1]] * 5 + rng.integers(0, 5, shape)
    return np.ascontiguousarray(a * (1 if dt == np.uint8 else 250)).astype(dt)


def _dev(a, offset):
    t = torch.from_numpy(a)
    x = torch.empty(a.size + offset, dtype=t.dtype, device="cuda")[offset:].view(a.shape)
    x.copy_(t)
    return x


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("se,offset", [("SESquare2D", 1), ("SECross2D", 0)])
def test_just_beyond_the_resident_tiles(dt, se, offset):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shape = (32 * sms // 2 + 3, 64 * 32 - 5)  # 64 tiles a row, one tile row more than 32 an SM
    assert -(-shape[0] // 32) * 64 > 32 * sms
    f, m = _plateaus(shape, dt, 1), _plateaus(shape, dt, 2)
    x, k = _dev(f, offset), _dev(m, offset)
    out = _dev(np.zeros_like(f), offset)
    s = Common_NL_SE[se]
    geo.low_leveling(x, k, s, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.low_leveling(f, m, se))
    geo.high_leveling(x, k, s, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.high_leveling(f, m, se))
    for kind, dilate in ((geo.reconstruction_type.dilate, True), (geo.reconstruction_type.erode, False)):
        geo.Reconstruction(kind, k, x, s, out)
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.reconstruct(m, f, se, dilate))


@pytest.fixture()
def L():
    from poutre2_gb300 import _lib
    lib = _lib.load()
    yield lib
    assert lib.pg_debug_set_limits(0, 0) == 0


def _corridor(shape, dt):
    """One corridor through the whole image or volume, marked at its first pixel."""
    f = np.zeros(shape, dt)
    flat = f.reshape((-1,) + shape[-2:])
    for z in range(0, flat.shape[0], 2):
        flat[z, ::4] = 100
        flat[z, 1::8, -1] = flat[z, 2::8, -1] = flat[z, 3::8, -1] = 100
        flat[z, 5::8, 0] = flat[z, 6::8, 0] = flat[z, 7::8, 0] = 100
        if z + 1 < flat.shape[0]:
            flat[z + 1, 0, 0] = 100
    m = np.zeros_like(f)
    m[(0,) * len(shape)] = 100
    return m, f


@pytest.mark.parametrize("limits", [(1, 0), (0, 1)], ids=["visits", "wait"])
@pytest.mark.parametrize("shape,dt", [((512, 512), np.float32), ((24, 96, 128), np.uint8), ((24, 96, 128), np.uint16)])
def test_gives_up_then_the_next_call_succeeds(L, limits, shape, dt):
    from poutre2_gb300.image import descriptor
    mk, f = _corridor(shape, dt)
    m, k = torch.from_numpy(mk).cuda(), torch.from_numpy(f).cuda()
    out = torch.empty_like(k)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    d = [descriptor(t) for t in (m, k, out)]
    se = 2 if len(shape) == 2 else 9

    def run():
        assert L.pg_reconstruction(1, ctypes.byref(d[0]), ctypes.byref(d[1]), se, ctypes.byref(d[2]), s) == 0
        return L.pg_check_device(s)

    assert L.pg_debug_set_limits(*limits) == 0
    assert run() == NOT_CONVERGED
    assert L.pg_debug_set_limits(0, 0) == 0
    assert run() == 0
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.reconstruct(mk, f, "SESquare2D" if se == 2 else "SECross3D", True))
