"""Results in lent library buffers: a buffer goes back once, when the last view
of it is gone, and no more than the limits are lent."""
import ctypes as C
import gc

import numpy as np
import pytest

from compression_b200 import codecs as cc


@pytest.fixture
def freed(monkeypatch):
    got = []

    class Fake:
        @staticmethod
        def gd_free(p):
            got.append(p.value)

    monkeypatch.setattr(cc, "lib", lambda: Fake)
    return got


def _memory(n):
    m = (C.c_uint8 * n)()
    return m, C.addressof(m)


def test_given_back_with_the_last_view(freed):
    m, p = _memory(100)
    a = cc._Lent.take(p, 100)
    a[:] = 7
    assert a.flags.writeable and a.dtype == np.uint8 and bytes(m) == b"\x07" * 100
    views = [a[10:20].view(np.int16), a.reshape(10, 10).T, memoryview(a)[5:]]
    del a
    while views:
        gc.collect()
        assert freed == []
        views.pop()
    gc.collect()
    assert freed == [p]
    assert cc._Lent._buffers == cc._Lent._bytes == 0


@pytest.mark.parametrize("n,lent", [(1, cc._Lent.MAX_BUFFERS), (cc._Lent.MAX_BYTES // 2, 2),
                                    (cc._Lent.MAX_BYTES, 1), (cc._Lent.MAX_BYTES + 1, 0)])
def test_limits(freed, n, lent):
    _, p = _memory(16)
    held = [x for x in (cc._Lent.take(p, n) for _ in range(6)) if x is not None]
    assert len(held) == lent
    held.clear()
    gc.collect()
    assert len(freed) == lent and cc._Lent._buffers == cc._Lent._bytes == 0


def test_the_buffer_counts_not_the_result(freed):
    """A short result in a long recycled buffer keeps the whole buffer."""
    _, p = _memory(16)
    assert cc._Lent.take(p, 16, cc._Lent.MAX_BYTES + 1) is None
    a = cc._Lent.take(p, 16, cc._Lent.MAX_BYTES - 100)
    assert a is not None and cc._Lent.take(p, 101) is None
    b = cc._Lent.take(p, 100)
    assert b is not None
    del a, b
    gc.collect()
    assert freed == [p, p] and cc._Lent._buffers == cc._Lent._bytes == 0


def test_decode_host_copies_out_of_a_long_buffer(freed, monkeypatch):
    m, p = _memory(8)
    m[:] = range(8)

    class Lib:
        capacity = 8

        @staticmethod
        def gd_free(x):
            freed.append(x.value)

        @staticmethod
        def gd_buffer_bytes(x):
            assert x.value == p
            return Lib.capacity

        @staticmethod
        def gd_lzss_contig_decompress(data, size, out, n):
            out._obj.value, n._obj.value = p, 8
            return 0

    monkeypatch.setattr(cc, "lib", lambda: Lib)
    enc = cc.Encoded("lzss_contig", np.zeros(1, np.uint8), 8, 1, 8, {}, {"container": np.zeros(1, np.uint8)})
    for Lib.capacity, lent in ((8, True), (cc._Lent.MAX_BYTES + 1, False)):
        a = cc.decode_host(enc)
        assert a.tolist() == list(range(8)) and (freed == []) == lent
        del a
        gc.collect()
        assert freed == [p]
        freed.clear()
