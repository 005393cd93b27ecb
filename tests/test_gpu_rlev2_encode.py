"""The warp encoder of RLE v2 lane streams against the host encoder, byte for
byte, at its run edges: runs of equal values around 3, 10 and 128, general runs
around 128, triples at a run's end, every encoding and width, values whose
arithmetic wraps, and lanes shorter and longer than the value window."""
import numpy as np
import pytest

from compression_b200 import codecs as cc

pytestmark = pytest.mark.gpu


def _segment(rng) -> list:
    kind = int(rng.integers(0, 12))
    big = int(rng.integers(0, 55))
    v = int(rng.integers(0, 1 << big)) if big else 0
    n = int(rng.choice([1, 2, 3, 4, 9, 10, 11, 12, 63, 64, 100, 126, 127, 128, 129, 130, 131, 255, 256, 257]))
    if kind == 0:
        return [v] * n
    if kind == 1:
        return [-v - 1] * n
    if kind == 2:
        return list(rng.integers(0, 1 << max(1, big), n))
    if kind == 3:
        return list(np.cumsum(rng.integers(0, 1 + (1 << min(40, big)), n)))
    if kind == 4:
        return list((1 << 50) - np.cumsum(rng.integers(1, 1 + (1 << min(40, big)), n)))
    if kind == 5:
        d = int(rng.integers(-1000, 1000))
        return [(1 << 40) + d * i for i in range(n)]
    if kind == 6:  # outliers: PATCHED_BASE
        x = rng.integers(0, 1 << 9, n)
        k = rng.random(n) < 0.03
        x[k] = rng.integers(0, 1 << max(10, big), int(k.sum()))
        return list(x)
    if kind == 7:
        return list(rng.integers(-(1 << 30), 1 << 30, n))
    if kind == 8:  # pairs and triples at every place
        return list(np.repeat(rng.integers(0, 50, n), rng.integers(1, 4, n)))[:n]
    if kind == 9:  # a range that wraps
        return [-5] + list(rng.integers(0, 100, 6)) + [(1 << 63) - 1] + list(rng.integers(0, 100, max(0, n - 8)))
    if kind == 10:
        return list(rng.integers(1 << 20, (1 << 20) + 3, n)) + [1 << 54]
    return list(rng.integers(0, 2, n))


def _lane(rng, n: int) -> np.ndarray:
    x = []
    while len(x) < n:
        x += _segment(rng)
    return np.array(x[:n], dtype=np.int64)


@pytest.mark.parametrize("read_unit,slices", [(32, 1), (32, 2), (32, 8), (32, 32), (1, 1), (1, 31), (1, 33), (8, 37),
                                              (128, 5)])
def test_bytes(cuda, read_unit, slices):
    rng = np.random.default_rng(1000 * read_unit + slices)
    n = read_unit * slices           # values per lane stream
    chunks = 3
    col = np.empty((chunks, slices, 32, read_unit), np.int64)
    for c in range(chunks):
        for t in range(32):
            col[c, :, t, :] = _lane(rng, n).reshape(slices, read_unit)
    flat = col.reshape(-1)
    for cut in (0, 1, 32 * n // 2 + 3):  # the last chunk whole and partial
        raw = flat[: flat.size - cut] if cut < 32 * n else flat
        want = cc.rlev2_encode(raw, 256 * n, read_unit)
        got = cc.encode_gpu("rlev2", raw, 256 * n, read_unit=read_unit)
        for k in want.meta:
            assert np.array_equal(want.meta[k], got.meta[k]), (k, cut)
        assert np.array_equal(want.data, got.data), cut


def test_benchmark_column(cuda):
    raw = cc.gen_rlev2_ints(77, 3 * 32768 + 1234)
    want = cc.rlev2_encode(raw, 256 * 1024, 32)
    got = cc.encode_gpu("rlev2", raw, 256 * 1024, read_unit=32)
    assert np.array_equal(want.meta["col_len"], got.meta["col_len"])
    assert np.array_equal(want.data, got.data)
