"""CPU test of the shared host copies behind the host-buffer calls and the
server's submits: callers that copy at once do not wait for one another's jobs,
and every byte arrives.
"""
import ctypes
import threading
import time

import numpy as np

import fastimagingpipe_b200 as fip


class Seg(ctypes.Structure):
    _fields_ = [("dst", ctypes.c_void_p), ("src", ctypes.c_void_p), ("bytes", ctypes.c_size_t)]


def host_copy(pairs):
    f = fip.lib()._Z13fip_host_copyPK10FipCopySegi
    f.restype = None
    segs = (Seg * len(pairs))(*[Seg(d.ctypes.data, s.ctypes.data, s.nbytes) for d, s in pairs])
    f(segs, len(pairs))


def test_a_small_copy_does_not_wait_for_a_large_one():
    big = [(np.zeros(1 << 28, np.uint8), np.full(1 << 28, 7, np.uint8))] * 8  # 2 GB in all
    small = (np.zeros(1 << 21, np.uint8), np.full(1 << 21, 9, np.uint8))
    host_copy([small])  # the pool's threads exist
    small[0][:] = 0
    times = {}
    started = threading.Event()

    def large():
        started.set()
        t0 = time.perf_counter()
        host_copy(big)
        times["large"] = time.perf_counter() - t0

    th = threading.Thread(target=large)
    th.start()
    started.wait()
    time.sleep(0.01)
    t0 = time.perf_counter()
    host_copy([small])
    times["small"] = time.perf_counter() - t0
    th.join()
    # Behind the large copy the small one, a thousandth of it, would take all
    # but the first 10 ms of its time.
    assert times["small"] < 0.5 * (times["large"] - 0.01)
    assert (big[0][0] == 7).all() and (small[0] == 9).all()


def test_copies_at_once_are_complete():
    rng = np.random.default_rng(1)
    jobs = [[(np.zeros(n, np.uint8), rng.integers(0, 256, n, np.uint8))
             for n in rng.integers(1, 1 << 21, 3)] for _ in range(24)]
    work = list(jobs)
    lock = threading.Lock()

    def client():
        while True:
            with lock:
                if not work:
                    return
                job = work.pop()
            host_copy(job)

    threads = [threading.Thread(target=client) for _ in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for job in jobs:
        for d, s in job:
            np.testing.assert_array_equal(d, s)
