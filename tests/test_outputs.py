"""Memory of returned images (bcgx.context._Outputs): taken again only once no view, torch
tensor or container holds the image; bounded; given back with the context. CPU only."""
import numpy as np
import pytest

from bcgx.context import _Outputs

SHAPE = (400, 300, 3)


@pytest.mark.parametrize("hold", ["view", "torch", "dict", "none"])
def test_memory_returns_with_the_last_reference(hold):
    pool = _Outputs()
    a = pool.empty(SHAPE, np.float32)
    a[:] = 7.0
    at = a.ctypes.data
    assert a.flags.writeable and a.flags.c_contiguous and a.dtype == np.float32 and a.shape == SHAPE
    if hold == "view":
        keep = a[5:9, ::2]
    elif hold == "torch":
        keep = pytest.importorskip("torch").from_numpy(a)
    else:
        keep = {"linear": a} if hold == "dict" else None
    del a
    if hold != "none":
        b = pool.empty(SHAPE, np.float32)
        assert b.ctypes.data != at
        b[:] = 1.0
        assert float((keep["linear"] if hold == "dict" else keep).reshape(-1)[0]) == 7.0
        del keep
    c = pool.empty(SHAPE, np.uint32)  # same size, another type
    assert c.ctypes.data == at and c.dtype == np.uint32


def test_memory_is_bounded_and_given_back(monkeypatch):
    monkeypatch.setattr(_Outputs, "LIMIT", 4 << 20)
    pool = _Outputs()
    images = [pool.empty((512, 512, 3), np.float32) for _ in range(4)]  # 3 MB each
    last = images[3].ctypes.data
    for k in range(4):
        images[k] = None
    assert pool._bytes == 3 << 20 and pool._free[0].ctypes.data == last
    kept = pool.empty((512, 512, 3), np.float32)
    pool.close()
    kept[:] = 2.0  # outlives the pool
    assert kept.sum() == 2.0 * kept.size
    del kept
    assert pool._bytes == 0 and not pool._free
    small = pool.empty((4, 4), np.float32)
    assert small.flags.owndata


class _Collects(np.ndarray):
    """Memory in the pool whose look at the size runs a collection."""
    run = None

    @property
    def nbytes(self):
        if _Collects.run:
            run, _Collects.run = _Collects.run, None
            run()
        return self.size


@pytest.mark.parametrize("mb", [2, 3, 6])
def test_memory_that_returns_inside_a_scan_shifts_nothing(monkeypatch, mb):
    """A collection inside empty() may return other images, and their return may evict
    what the scan has passed."""
    monkeypatch.setattr(_Outputs, "LIMIT", 7 << 20)
    pool = _Outputs()
    pool._put(np.empty(3 << 20, np.uint8))
    pool._put(np.empty(3 << 20, np.uint8).view(_Collects))
    _Collects.run = lambda: pool._put(np.empty(mb << 20, np.uint8))
    a = pool.empty((512, 512, 3), np.float32)
    assert _Collects.run is None
    a[:] = 1.0
    assert a.sum() == a.size
    assert pool._bytes == sum(m.size for m in pool._free) <= pool.LIMIT


def test_pool_serves_several_threads():
    import threading
    pool, bad = _Outputs(), []

    def work(k):
        for i in range(300):
            a = pool.empty((256, 256 + 64 * (i % 3)), np.float32)
            a[:] = k
            if not (a == k).all():
                bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad and pool._bytes == sum(m.nbytes for m in pool._free)
