"""Reconstruction of volumes whose 32 x 8 x 8 bricks stay on the GPU from start to end, against the oracle; whole
numbers, equal.  Sizes around a brick's sides, one path through many bricks, and the first volume too large."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _volume(shape, dt, seed):
    rng = np.random.default_rng(seed)
    c = [(s + 3) // 4 for s in shape]
    a = np.kron(rng.integers(0, 40, c), np.ones((4, 4, 4), np.int64))[:shape[0], :shape[1], :shape[2]]
    return np.ascontiguousarray((a * 5 + rng.integers(0, 5, shape)) * (1 if dt == np.uint8 else 250)).astype(dt)


@pytest.mark.parametrize("dt", [np.uint8, np.uint16])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 9, 33), (8, 8, 32), (9, 7, 31), (7, 9, 65), (17, 16, 64), (25, 30, 70)])
def test_operations(dt, shape):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    s, h = Common_NL_SE.SECross3D, 30 if dt == np.uint8 else 7000
    f = _volume(shape, dt, sum(shape))
    x = torch.from_numpy(f).cuda()
    out = torch.empty_like(x)
    for name in ("h_maxima", "h_minima", "h_convex", "h_concave", "dynamic_pseudo_opening", "dynamic_pseudo_closing"):
        getattr(geo, name)(x, h, s, out)
        np.testing.assert_array_equal(out.cpu().numpy(), getattr(oracle, name)(f, h, "SECross3D"), err_msg=name)
    b = torch.empty(shape, dtype=torch.uint8, device="cuda")
    geo.h_maxima_binary(x, h, s, b)
    np.testing.assert_array_equal(b.cpu().numpy(), oracle.h_maxima_binary(f, h, "SECross3D"))
    m = f[::-1, ::-1, ::-1].copy()
    geo.leveling(x, torch.from_numpy(m).cuda(), s, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.leveling(f, m, "SECross3D"))
    for kind, marker in ((geo.reconstruction_type.dilate, f // 2), (geo.reconstruction_type.erode, f + (np.iinfo(dt).max - f) // 2)):
        marker = marker.astype(dt)
        geo.Reconstruction(kind, torch.from_numpy(marker).cuda(), x, s, out)
        np.testing.assert_array_equal(out.cpu().numpy(),
                                      oracle.reconstruct(marker, f, "SECross3D", kind == geo.reconstruction_type.dilate))


def test_one_path_through_many_bricks():
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    D, H, W = 20, 28, 70
    mask = np.zeros((D, H, W), np.uint8)
    for z in range(0, D, 2):
        for r in range(0, H, 3):
            mask[z, r, :] = 150
            mask[z, r:r + 3, W - 1 if (r // 3) % 2 == 0 else 0] = 150
        mask[z:z + 3, H - 1 if (z // 2) % 2 == 0 else 0, 5] = 150
    marker = np.zeros_like(mask)
    marker[0, 0, 0] = 140
    x, m = torch.from_numpy(mask).cuda(), torch.from_numpy(marker).cuda()
    out = torch.empty_like(x)
    geo.Reconstruction(geo.reconstruction_type.dilate, m, x, Common_NL_SE.SECross3D, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.reconstruct(marker, mask, "SECross3D", True))


@pytest.mark.parametrize("dt,side", [(np.uint8, 200), (np.uint16, 180)])
def test_a_volume_too_large(dt, side):
    # 7 x 25 x 25 (6 x 23 x 23) bricks are more than an SM's share: the launches of recon3d.cu run
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    f = _volume((side, side, side), dt, 8)
    x = torch.from_numpy(f).cuda()
    out = torch.empty_like(x)
    geo.h_maxima(x, 30, Common_NL_SE.SECross3D, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.h_maxima(f, 30, "SECross3D"))
