"""Reconstruction of images whose 32 x 32 tiles stay on the GPU from start to end (1- and 2-byte pixels, up to
4864 tiles on 152 SMs) and of those just beyond, against the oracle; whole numbers, equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 33), (31, 32), (32, 31), (33, 65), (64, 96), (65, 63), (200, 301), (97, 1030)]


def _image(shape, dt, seed):
    """Grey plateaus of many sizes: paths wind through several tiles."""
    rng = np.random.default_rng(seed)
    a = np.kron(rng.integers(0, 40, ((shape[0] + 4) // 5, (shape[1] + 6) // 7)), np.ones((5, 7), np.int64))
    a = a[:shape[0], :shape[1]] * 5 + rng.integers(0, 5, shape)
    return np.ascontiguousarray(a * (1 if dt == np.uint8 else 250)).astype(dt)


def _dev(a, offset=0):
    t = torch.from_numpy(a)
    buf = torch.empty(a.size + offset, dtype=t.dtype, device="cuda")
    x = buf[offset:].view(a.shape)
    x.copy_(t)
    return x


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("se", ["SESquare2D", "SECross2D"])
def test_operations(dt, se):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    s, h = Common_NL_SE[se], 30 if dt == np.uint8 else 7000
    for shape in SIZES:
        f = _image(shape, dt, shape[1])
        x = _dev(f)
        out = torch.empty_like(x)
        for name in ("h_maxima", "h_minima", "h_convex", "h_concave", "dynamic_pseudo_opening", "dynamic_pseudo_closing"):
            getattr(geo, name)(x, h, s, out)
            np.testing.assert_array_equal(out.cpu().numpy(), getattr(oracle, name)(f, h, se), err_msg=f"{name} {shape}")
        b = torch.empty(shape, dtype=torch.uint8, device="cuda")
        geo.h_maxima_binary(x, h, s, b)
        np.testing.assert_array_equal(b.cpu().numpy(), oracle.h_maxima_binary(f, h, se), err_msg=f"binary {shape}")
        m = f[::-1, ::-1].copy()
        geo.leveling(x, _dev(m), s, out)
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.leveling(f, m, se), err_msg=f"leveling {shape}")


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_reconstruction_of_misaligned_buffers(dt, offset):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    for shape in ((64, 64), (70, 129), (33, 98)):
        f = _image(shape, dt, 11)
        for kind, marker in ((geo.reconstruction_type.dilate, f // 2), (geo.reconstruction_type.erode, f + (np.iinfo(dt).max - f) // 2)):
            x, k = _dev(marker.astype(dt), offset), _dev(f, offset)
            out = _dev(np.zeros_like(f), offset)
            geo.Reconstruction(kind, x, k, Common_NL_SE.SESquare2D, out)
            exp = oracle.reconstruct(marker.astype(dt), f, "SESquare2D", kind == geo.reconstruction_type.dilate)
            np.testing.assert_array_equal(out.cpu().numpy(), exp, err_msg=f"{shape} {kind}")


@pytest.mark.parametrize("rows", [2432, 2433])
def test_around_the_most_tiles(rows):
    # 76 x 64 = 4864 tiles stay on 152 SMs of 32 warps; one row more is 4928
    from poutre2_gb300 import geo, synthetic
    from poutre2_gb300.se import Common_NL_SE
    f = synthetic.smoothed_noise_u8((rows, 2048), 3, 4.0)
    x = _dev(f)
    out = torch.empty_like(x)
    geo.h_maxima(x, 25, Common_NL_SE.SESquare2D, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.h_maxima(f, 25, "SESquare2D"))


def test_one_path_through_every_tile():
    # a serpentine corridor: every tile is woken many times, one at a time
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    mask = np.zeros((300, 301), np.uint8)
    mask[::4] = 200
    mask[2::8, -1] = mask[1::8, -1] = mask[3::8, -1] = 200
    mask[6::8, 0] = mask[5::8, 0] = mask[7::8, 0] = 200
    marker = np.zeros_like(mask)
    marker[0, 0] = 190
    out = torch.empty(mask.shape, dtype=torch.uint8, device="cuda")
    for se in ("SESquare2D", "SECross2D"):
        geo.Reconstruction(geo.reconstruction_type.dilate, _dev(marker), _dev(mask), Common_NL_SE[se], out)
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.reconstruct(marker, mask, se, True))


def test_calls_on_several_streams():
    # concurrent calls, each with its own work area
    from poutre2_gb300 import geo, synthetic
    from poutre2_gb300.se import Common_NL_SE
    f = synthetic.smoothed_noise_u8((700, 900), 5, 4.0)
    exp = oracle.h_maxima_binary(f, 20, "SESquare2D")
    x = _dev(f)
    outs, streams = [torch.empty_like(x) for _ in range(4)], [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    for _ in range(5):
        for o, st in zip(outs, streams):
            with torch.cuda.stream(st):
                geo.h_maxima_binary(x, 20, Common_NL_SE.SESquare2D, o, check=False)
    torch.cuda.synchronize()
    for o in outs:
        np.testing.assert_array_equal(o.cpu().numpy(), exp)
