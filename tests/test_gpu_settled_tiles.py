"""Tiles of u8 images that a neighbour queues again after they settled skip the sweeps when their new halo moves no
border pixel: long propagations that touch tiles along every side and corner, against the oracle; equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _maze(shape, seed):
    """One-pixel corridors of slowly falling height between low walls, at every offset to the tile grid."""
    rng = np.random.default_rng(seed)
    f = rng.integers(0, 20, shape).astype(np.int64)
    y = np.arange(shape[0])
    for c in range(seed % 5, shape[1], 6):
        f[:, c] = 230 - (y + 3 * c) % 97
        row = (c // 6) % 2 * (shape[0] - 1)
        f[row, c:c + 7] = 200
    for d in range(0, min(shape), 3):  # diagonal steps: corners of tiles
        f[d, d] = 240
    return f.astype(np.uint8)


@pytest.mark.parametrize("se", ["SESquare2D", "SECross2D"])
@pytest.mark.parametrize("sweeps", [1, 2, 512])
def test_batches(se, sweeps):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    imgs = [_maze(s, i) for i, s in enumerate([(32, 32), (33, 64), (64, 31), (65, 97), (128, 128), (150, 203), (1, 90), (90, 1)])]
    xs = [torch.from_numpy(f).cuda() for f in imgs]
    outs = [torch.empty_like(x) for x in xs]
    for h in (1, 40):
        plan = geo.HMaximaBinaryBatch(xs, h, Common_NL_SE[se], outs, autotune=False)
        plan.set_config(32, sweeps)
        plan.run(check=True)
        for f, o in zip(imgs, outs):
            np.testing.assert_array_equal(o.cpu().numpy(), oracle.h_maxima_binary(f, h, se), err_msg=f"{f.shape} h {h}")


@pytest.mark.parametrize("erode", [False, True])
def test_more_tiles_than_stay_on_the_gpu(erode):
    from poutre2_gb300 import geo
    from poutre2_gb300.se import Common_NL_SE
    n = 32 * int(np.ceil(np.sqrt(32 * torch.cuda.get_device_properties(0).multi_processor_count))) + 5
    f = np.tile(_maze((160, 161), 7), (n // 160 + 1, n // 161 + 1))[:n, :n].copy()
    m = np.zeros_like(f)
    m[0, ::40] = f[0, ::40]
    if erode:
        f, m = 255 - f, 255 - m
    kind = geo.reconstruction_type.erode if erode else geo.reconstruction_type.dilate
    out = torch.empty((n, n), dtype=torch.uint8, device="cuda")
    geo.Reconstruction(kind, torch.from_numpy(m).cuda(), torch.from_numpy(f).cuda(), Common_NL_SE.SECross2D, out)
    want = oracle.reconstruct(m, f, "SECross2D", not erode)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
