"""The host batch on pageable arrays, which several threads stage in small
chunks, against the same call on pinned arrays (one thread, copied directly):
the same bytes at counts around the chunk sizes, for every result format, with
callers running at once, and a time-out that leaves the scene usable."""
import os
import threading

import numpy as np
import pytest

from gonzales_b200 import GpuAccelerator, GzgError, scenes
from gonzales_b200 import _ffi as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rays():
    hs = scenes.raycast_scene(subdiv=4).build()
    n = (1 << 20) + 12345
    o, d, t = scenes.raycast_rays(hs, 1024, 512, n - 1024 * 512, seed=3)
    acc = GpuAccelerator(hs)
    yield acc, scenes.pack_reference_rays(o, d), t
    acc.close()


def _pinned(a):
    import torch

    return torch.from_numpy(a).pin_memory().numpy()


def _direct(acc, r6, t):
    import torch

    out = torch.zeros(len(t) * F.INTERSECTION_DTYPE.itemsize, dtype=torch.uint8).pin_memory().numpy()
    return acc.intersect_batch(_pinned(r6), _pinned(t), out=out.view(F.INTERSECTION_DTYPE))  # (a copy would drop padding)


@pytest.mark.parametrize("n", [1, 16383, 16384, 16385, 16384 * 8, 16384 * 16 + 1, (1 << 17) * 8 + 3, (1 << 20) + 12345])
def test_staged_equals_direct(rays, n):
    acc, r6, t = rays
    ref = _direct(acc, r6[:n], t[:n])
    got = acc.intersect_batch(r6[:n], t[:n])
    assert got.tobytes() == ref.tobytes()
    hits = acc.intersect_batch_hits(r6[:n], t[:n])
    assert hits[:, 0].tobytes() == ref["t_hit"].tobytes()
    occ = acc.occluded_batch(r6[:n], t[:n])
    assert np.array_equal(occ, (ref["hit"] != 0).astype(np.uint8))
    assert acc.error_word() == 0


def test_callers_at_once(rays):
    acc, r6, t = rays
    n = 300_000
    ref = acc.intersect_batch(r6[:n], t[:n])
    got = [None] * 6

    def call(k):
        got[k] = acc.intersect_batch(r6[k * 1000:n], t[k * 1000:n])

    threads = [threading.Thread(target=call, args=(k,)) for k in range(6)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for k in range(6):
        assert got[k].tobytes() == ref[k * 1000:].tobytes()


GZG_ERR_TIMEOUT = 8


def test_time_out_of_a_staged_call(rays, monkeypatch):
    """Every worker's wait runs out (on the host: 1 us), its chunk still in
    flight: the caller gets the time-out and its message, the slots' buffers are
    left to their chunks, every helper thread has ended, and the next calls are
    served as before, also while those chunks still run."""
    import torch

    acc, r6, t = rays
    n = 1_000_000
    ref = acc.intersect_batch(r6[:n], t[:n])
    threads = len(os.listdir("/proc/self/task"))
    for k in range(4):
        monkeypatch.setenv("GZG_WAIT_LIMIT_US", "1")
        with pytest.raises(GzgError) as e:
            acc.intersect_batch(r6[:n], t[:n])
        assert e.value.status == GZG_ERR_TIMEOUT and "GZG_WAIT_LIMIT_US" in str(e.value)
        monkeypatch.delenv("GZG_WAIT_LIMIT_US")
        if k % 2 == 0:
            torch.cuda.synchronize()  # the abandoned chunks have run
        again = acc.intersect_batch(r6[:n], t[:n])
        assert again.tobytes() == ref.tobytes()
        assert acc.error_word() == 0
    assert len(os.listdir("/proc/self/task")) == threads
    torch.cuda.synchronize()
    assert acc.occluded_batch(r6[:n], t[:n]).sum() == (ref["hit"] != 0).sum()


def test_callers_at_once_take_no_helpers(rays):
    """A call that runs by itself may take 7 helper threads; callers that run at
    the same time stage on their own threads (a chunk ring that wraps here), and
    give the same bytes."""
    acc, r6, t = rays
    r6, t = np.tile(r6, (3, 1)), np.tile(t, 3)
    ref = _direct(acc, r6, t)
    base, most, got = len(os.listdir("/proc/self/task")), [0], [None] * 8
    start = threading.Barrier(8)

    def call(k):
        start.wait()
        n = len(t) - 7777 * k if k < 3 else 300_000 + k  # over and under the ring's chunks
        for _ in range(1 if k < 3 else 6):
            got[k] = acc.intersect_batch(r6[:n], t[:n])
            most[0] = max(most[0], len(os.listdir("/proc/self/task")))

    def watch():
        while any(th.is_alive() for th in threads):
            most[0] = max(most[0], len(os.listdir("/proc/self/task")))

    threads = [threading.Thread(target=call, args=(k,)) for k in range(8)]
    for th in threads:
        th.start()
    watch()
    for th in threads:
        th.join()
    for k in range(8):
        assert got[k].tobytes() == ref[:len(got[k])].tobytes()
    assert most[0] <= base + 8 + 7, "more helpers than one call's"
    assert acc.error_word() == 0
