"""Neighbour lists on both sides of the rule that takes their chords or gathers their offsets: the same list on a small
image, a narrow one and one large enough for the chords, against the oracle, bit-exact."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

LISTS = {
    "disk": [(y, x) for y in range(-6, 7) for x in range(-6, 7) if y * y + x * x <= 40],
    "diagonals": sorted({(t, s * t) for t in range(-12, 13) for s in (-1, 1)}),
    "tall": [(y, x) for y in (-60, -59, 0, 60) for x in range(-3, 4)],
    "far": [(0, x) for x in range(400, 420)] + [(-300, x) for x in range(-2, 3)] + [(20, x) for x in range(-1200, -1180)],
    "row": [(0, x) for x in range(-70, 71)],
    "most chords": [(y, 3 * x) for y in range(-20, 21) for x in range(-6, 6)],    # 492 chords
    "too many chords": [(y, 3 * x) for y in range(-20, 22) for x in range(-6, 7)],  # 546: gathered
}


def _check(a, offsets):
    from poutre2_gb300 import llm
    from poutre2_gb300.se import NeighborList
    x, nl = torch.from_numpy(a).cuda(), NeighborList(offsets)
    for dilate in (True, False):
        out = torch.empty_like(x)
        (llm.Dilate if dilate else llm.Erode)(x, nl, out)
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.erode_dilate_nl(a, offsets, dilate), err_msg=f"{a.shape}")


@pytest.mark.parametrize("dt", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("name", sorted(LISTS))
def test_images(dt, name):
    rng = np.random.default_rng(3)
    for shape in ((40, 50), (3000, 2), (1500, 33), (300, 501), (1203, 1402)):
        _check(rng.integers(0, 250, shape).astype(dt), LISTS[name])


@pytest.mark.parametrize("dt", [np.uint8, np.float32])
def test_volumes(dt):
    rng = np.random.default_rng(4)
    ball = [(z, y, x) for z in range(-3, 4) for y in range(-3, 4) for x in range(-3, 4) if z * z + y * y + x * x <= 12]
    for shape in ((6, 20, 8), (100, 32, 4), (20, 70, 300)):
        _check(rng.integers(0, 250, shape).astype(dt), ball)


def test_a_captured_list_outlives_the_call():
    # a small image, whose list would be gathered: in a graph it goes by value
    import ctypes

    from poutre2_gb300 import _lib
    from poutre2_gb300.image import descriptor
    L, driver = _lib.load(), ctypes.CDLL("libcuda.so.1")
    offsets = LISTS["disk"]
    a = np.random.default_rng(5).integers(0, 250, (50, 60)).astype(np.uint8)
    x = torch.from_numpy(a).cuda()
    out = torch.empty_like(x)
    dx, do = descriptor(x), descriptor(out)
    flat = (ctypes.c_int32 * (2 * len(offsets)))(*[v for o in offsets for v in o])
    stream = torch.cuda.Stream()
    s = ctypes.c_void_p(stream.cuda_stream)
    torch.cuda.synchronize()
    assert L.pg_dilate_nl(ctypes.byref(dx), flat, len(offsets), ctypes.byref(do), s) == 0  # the kernels are loaded
    stream.synchronize()
    assert driver.cuStreamBeginCapture_v2(s, 0) == 0
    assert L.pg_dilate_nl(ctypes.byref(dx), flat, len(offsets), ctypes.byref(do), s) == 0
    graph, ready = ctypes.c_void_p(), ctypes.c_void_p()
    assert driver.cuStreamEndCapture(s, ctypes.byref(graph)) == 0 and graph.value
    assert driver.cuGraphInstantiateWithFlags(ctypes.byref(ready), graph, ctypes.c_ulonglong(0)) == 0
    ctypes.memset(flat, 0, ctypes.sizeof(flat))
    junk = [np.full(n, 7, np.int32) for n in range(16, 4096, 16)]  # the call's host memory is somebody else's now
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        assert driver.cuGraphLaunch(ready, s) == 0
        stream.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.erode_dilate_nl(a, offsets, True))
    assert junk[0][0] == 7
    assert driver.cuGraphExecDestroy(ready) == 0 and driver.cuGraphDestroy(graph) == 0


def test_more_offsets_than_a_list_may_hold():
    from poutre2_gb300 import llm
    from poutre2_gb300._lib import PoutreError
    from poutre2_gb300.se import NeighborList
    x = torch.zeros((100, 100), dtype=torch.uint8, device="cuda")
    with pytest.raises(PoutreError):
        llm.Dilate(x, NeighborList([(y, x) for y in range(64) for x in range(65)]), torch.empty_like(x))
