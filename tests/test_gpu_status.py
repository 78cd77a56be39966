"""What a kernel recorded reaches the caller of pg_check_device, whatever other calls left behind."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

NOT_CONVERGED = 9


@pytest.fixture()
def L():
    from poutre2_gb300 import _lib
    lib = _lib.load()
    yield lib
    assert lib.pg_debug_set_limits(0, 0) == 0
    from poutre2_gb300.image import descriptor
    a, b = (torch.zeros(8, 8, dtype=torch.uint8, device="cuda") for _ in range(2))
    da, db = descriptor(a), descriptor(b)
    for _ in range(2):  # the first kernel launch after a pending error reports it
        status = lib.pg_erode(ctypes.byref(da), 2, 1, ctypes.byref(db), None)
    assert status == 0


def leave_an_error_pending(L):
    """A call that is refused while a stream captures leaves its error with the CUDA runtime of the library: no
    later call of it failed.  The capture ends without a graph."""
    driver = ctypes.CDLL("libcuda.so.1")
    stream, graph = torch.cuda.Stream(), ctypes.c_void_p()
    torch.cuda.synchronize()
    assert driver.cuStreamBeginCapture_v2(ctypes.c_void_p(stream.cuda_stream), 0) == 0
    assert L.pg_last_reconstruction_rounds() == -1
    driver.cuStreamEndCapture(ctypes.c_void_p(stream.cuda_stream), ctypes.byref(graph))
    assert not graph.value


def capped_reconstruction(L):
    """A reconstruction that gave up after one visit a tile."""
    s = capped_reconstruction_on(L, torch.cuda.current_stream())
    torch.cuda.synchronize()
    return s


def capped_reconstruction_on(L, stream):
    """Queues it on `stream` and waits for it there."""
    from poutre2_gb300.image import descriptor
    f = np.zeros((256, 256), np.uint8)
    f[::4] = 100
    f[2::8, -1] = f[1::8, -1] = f[3::8, -1] = 100
    f[6::8, 0] = f[5::8, 0] = f[7::8, 0] = 100
    m = np.zeros_like(f)
    m[0, 0] = 100
    k, mk = torch.from_numpy(f).cuda(), torch.from_numpy(m).cuda()
    out = torch.empty_like(k)
    torch.cuda.current_stream().synchronize()
    s = ctypes.c_void_p(stream.cuda_stream)
    d = [descriptor(x) for x in (mk, k, out)]
    assert L.pg_debug_set_limits(1, 0) == 0
    assert L.pg_reconstruction(1, ctypes.byref(d[0]), ctypes.byref(d[1]), 2, ctypes.byref(d[2]), s) == 0
    assert L.pg_debug_set_limits(0, 0) == 0
    stream.synchronize()
    return s


def test_a_status_is_kept_while_an_older_error_is_pending(L):
    capped_reconstruction(L)  # the kernels are loaded
    L.pg_check_device(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    leave_an_error_pending(L)
    s = capped_reconstruction(L)
    assert L.pg_check_device(s) == NOT_CONVERGED
    assert L.pg_check_device(s) == 0  # reported once


def test_a_failed_labelling_keeps_its_word_until_its_kernels_ended(L):
    # the call reports the pending error after its kernels were queued behind a long one: when it returns, none of
    # them can still write the count into a pinned word that another call has been given meanwhile
    from poutre2_gb300.image import descriptor
    x = torch.ones(64, 64, dtype=torch.uint8, device="cuda")
    out = torch.empty(64, 64, dtype=torch.int64, device="cuda")
    dx, do, count = descriptor(x), descriptor(out), ctypes.c_int64(-1)
    stream = torch.cuda.Stream()
    s = ctypes.c_void_p(stream.cuda_stream)
    assert L.pg_label_binary(ctypes.byref(dx), 2, ctypes.byref(do), ctypes.byref(count), s) == 0 and count.value == 1
    leave_an_error_pending(L)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)  # about 0.2 s
    assert not stream.query()
    assert L.pg_label_binary(ctypes.byref(dx), 2, ctypes.byref(do), ctypes.byref(count), s) != 0
    assert stream.query()


def test_more_calls_than_pinned_words(L):
    # 64 labellings behind a long kernel hold every word: the next count and the next status come by copies
    import threading

    from poutre2_gb300.image import descriptor
    n = 64
    busy, free = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(40, 70, dtype=torch.uint8, device="cuda")
    x[::3, ::4] = 1  # 14 x 18 pixels of their own
    outs = [torch.empty(40, 70, dtype=torch.int64, device="cuda") for _ in range(n + 1)]
    counts, statuses = [ctypes.c_int64(-1) for _ in range(n + 1)], [None] * (n + 1)
    dx, ds = descriptor(x), [descriptor(o) for o in outs]
    capped_reconstruction(L)
    L.pg_check_device(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()

    def label(i):
        s = ctypes.c_void_p((busy if i < n else free).cuda_stream)
        statuses[i] = L.pg_label_binary(ctypes.byref(dx), 3, ctypes.byref(ds[i]), ctypes.byref(counts[i]), s)

    label(n)
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)  # about a second
    threads = [threading.Thread(target=label, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    import time
    time.sleep(0.2)  # every thread is in its call
    counts[n].value = -1
    label(n)
    s = capped_reconstruction_on(L, free)
    status = L.pg_check_device(s)
    held = not busy.query()
    for t in threads:
        t.join()
    assert status == NOT_CONVERGED and L.pg_check_device(s) == 0
    assert statuses == [0] * (n + 1) and [c.value for c in counts] == [14 * 18] * (n + 1)
    assert held, "the words were not all taken for the whole time"
