"""Counts in little device memory, and how much they take: the stream-ordered
allocations are made from a pool of the test's own, with a size of its own."""
import ctypes as C

import numpy as np
import pytest

import oracle
import trianglecount_gb300 as tc
from trianglecount_gb300 import generators as gen

pytestmark = pytest.mark.gpu

MB = 1 << 20


class PoolProps(C.Structure):
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int),
                ("location_id", C.c_int), ("security", C.c_void_p), ("max_size", C.c_size_t), ("usage", C.c_ushort),
                ("reserved", C.c_ubyte * 54)]


class Pool:
    """The device's current memory pool while entered; at most `size` bytes (0: as much as there is)."""
    RELEASE_THRESHOLD, RESERVED, USED = 4, 5, 7

    def __init__(self, size=0):
        self.cu, self.h, self.old = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_void_p()
        self.size = size

    def ok(self, status):
        assert status == 0, f"driver status {status}"

    def __enter__(self):
        self.ok(self.cu.cuDeviceGetMemPool(C.byref(self.old), 0))
        props = PoolProps(alloc_type=1, location_type=1, location_id=0, max_size=self.size)
        self.ok(self.cu.cuMemPoolCreate(C.byref(self.h), C.byref(props)))
        keep = C.c_uint64(2**64 - 1)
        self.ok(self.cu.cuMemPoolSetAttribute(self.h, self.RELEASE_THRESHOLD, C.byref(keep)))
        self.ok(self.cu.cuDeviceSetMemPool(0, self.h))
        return self

    def __exit__(self, *exc):
        self.ok(self.cu.cuDeviceSetMemPool(0, self.old))
        self.ok(self.cu.cuMemPoolDestroy(self.h))

    def get(self, attribute):
        v = C.c_uint64()
        self.ok(self.cu.cuMemPoolGetAttribute(self.h, attribute, C.byref(v)))
        return v.value


@pytest.fixture
def own():
    """A context of the test's own: graphs that hold memory of its pools go with it."""
    c = tc.Context(0)
    yield c
    c.close()


def among(rp, n_rows):
    return np.concatenate((rp, np.full(n_rows + 1 - len(rp), rp[-1], np.int32)))


def test_a_count_that_does_not_fit_packed_counts_on_plain_ids(own):
    """R-MAT 16 in 2 M rows: 154 MB of scratch packed, 77 MB for the plain-id tables."""
    rp, col, want = oracle.pipeline(*gen.rmat(16))
    rp = among(rp, 2_000_000)
    _, pr = oracle.count(rp, col, per_root=True)
    g, h = own.upload(rp, col), own.upload(rp, col)
    with Pool(112 * MB) as pool:
        for _ in range(3):
            got, st = own.count(g, stats=True)
            assert got == want and st["launches"] > 5
        g.free()
        own.synchronize()
        assert np.array_equal(own.count_per_root(h), pr)
        h.free()
        own.synchronize()
        assert pool.get(Pool.USED) == 0
    g = own.upload(rp, col)
    with Pool(112 * MB):
        b = own.batch([g])
        assert [list(b.run()) for _ in range(2)] == [[want]] * 2 and b.stats()["launches"] > 5
        b.free()
        assert own.count_parts_csr([(rp, col, len(rp) - 1)])[0] == want
        own.synchronize()
    assert own.count(g, stats=True)[1]["launches"] == 5 and own.count(g) == want
    g.free()


def test_a_count_that_does_not_fit_at_all_leaves_nothing_behind(own):
    rp, col, want = oracle.pipeline(*gen.rmat(16))
    rp = among(rp, 2_000_000)
    own.set_tuning(probe_kicks=0)  # the plain-id tables
    g = own.upload(rp, col)
    with Pool(32 * MB) as pool:
        used = []
        for _ in range(4):
            with pytest.raises(tc.TCError) as e:
                own.count(g)
            assert e.value.code == "TC_E_NOMEM"
            own.synchronize()
            used.append(pool.get(Pool.USED))
        assert max(used) < MB
        kept = own.upload(np.array([0, 2, 3, 3], np.int32), np.array([1, 2, 2], np.int32))
        assert own.count(kept) == 1
        kept.free()
        own.synchronize()
    assert own.count(g) == want
    g.free()
