"""The warp encoders of RLE v1 lane streams and LZSS columns against the host
encoders, byte for byte, at their edges: runs around 3 and 129 values, literal
groups around 127, differences around a byte's range, lanes shorter and longer
than the value window; columns from the shortest to twice the history, matches
of every length, self-similar and incompressible data."""
import numpy as np
import pytest

from compression_b200 import codecs as cc

pytestmark = pytest.mark.gpu


def _v1_lane(rng, n: int, bits: int) -> np.ndarray:
    x, top = [], 1 << (bits - 1)
    while len(x) < n:
        k = int(rng.choice([1, 2, 3, 4, 31, 32, 63, 126, 127, 128, 129, 130, 131, 258, 259, 260]))
        v = int(rng.integers(-top, top))
        d = int(rng.choice([0, 1, -1, 127, 128, -128, -129, 5, -7, 126]))
        kind = int(rng.integers(0, 4))
        if kind == 0:
            x += [v + d * i for i in range(k)]
        elif kind == 1:
            x += list(rng.integers(-top, top, k))
        elif kind == 2:
            x += list(rng.integers(0, 3, k))
        else:  # pairs of one difference, never three values
            x += [v + (i // 2) * 200 + (i % 2) * d for i in range(k)]
    mask = (1 << bits) - 1
    return np.array([int(v) & mask for v in x[:n]], dtype=np.uint64).astype(np.uint32 if bits == 32 else np.uint64)


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("ccl,slices", [(128, 1), (128, 4), (128, 32), (8, 1), (8, 33), (64, 17)])
def test_rlev1(cuda, elem, ccl, slices):
    wil = ccl // elem
    n = wil * slices
    if n < 2:
        pytest.skip("a lane of one value has no encoding")
    rng = np.random.default_rng(100 * ccl + slices + elem)
    col = np.stack([np.stack([_v1_lane(rng, n, 8 * elem).reshape(slices, wil) for _ in range(32)], 1) for _ in range(3)])
    flat = np.ascontiguousarray(col).reshape(-1)
    for cut in (0, 1, 16 * n + 3):
        raw = flat[: flat.size - cut]
        want = cc.rlev1_encode(raw, 32 * ccl * slices, ccl, elem)
        got = cc.encode_gpu("rlev1", raw, 32 * ccl * slices, comp_col_len=ccl, elem_bytes=elem)
        for k in want.meta:
            assert np.array_equal(want.meta[k], got.meta[k]), (k, cut)
        assert np.array_equal(want.data, got.data), cut


def _lz_column(rng, n: int, kind: int) -> np.ndarray:
    if kind == 0:
        return np.full(n, int(rng.integers(0, 256)), np.uint8)
    if kind == 1:
        return np.resize(rng.integers(0, 256, int(rng.integers(1, 70)), dtype=np.uint8), n)
    if kind == 2:
        return rng.integers(0, 256, n, dtype=np.uint8)
    if kind == 3:
        return rng.integers(0, 2, n, dtype=np.uint8)
    out = []  # copies of every length from every distance
    while len(out) < n:
        if not out or rng.random() < 0.3:
            out.append(int(rng.integers(0, 8)))
        else:
            d, k = int(rng.integers(1, len(out) + 1)), int(rng.integers(2, 50))
            for _ in range(k):
                out.append(out[-d])
    return np.array(out[:n], np.uint8)


@pytest.mark.parametrize("chunk", [128, 256, 2048, 4224, 65536, 66048, 131072])
def test_lzss(cuda, chunk):
    rng = np.random.default_rng(chunk)
    n = chunk // 32
    chunks = []
    for c in range(3):
        cols = [_lz_column(rng, n, (q + c) % 6) for q in range(32)]
        chunks.append(np.stack([x.reshape(-1, 4) for x in cols], 1).reshape(-1))
    raw = np.concatenate(chunks)
    for cut in (0, 5):
        want = cc.lzss_encode(raw[: raw.size - cut], chunk)
        got = cc.encode_gpu("lzss", raw[: raw.size - cut], chunk)
        for k in want.meta:
            assert np.array_equal(want.meta[k], got.meta[k]), (k, cut)
        assert np.array_equal(want.data, got.data), cut


@pytest.mark.parametrize("chunk", [2048, 65536, 131072])
def test_lzss_pairs(cuda, chunk):
    """Columns of 1 to 32 distinct bytes: 32 positions with anything from a
    few to thousands of older positions to compare, in one column a stretch of
    each."""
    rng = np.random.default_rng(7 * chunk)
    n = chunk // 32
    cols = [rng.integers(0, q + 1, n, dtype=np.uint8) for q in range(31)]
    cols.append(np.resize(np.concatenate([rng.integers(0, k, 96, dtype=np.uint8) for k in (1, 2, 64, 4, 16, 1, 256)]), n))
    raw = np.stack([x.reshape(-1, 4) for x in cols], 1).reshape(-1)
    want = cc.lzss_encode(raw, chunk)
    got = cc.encode_gpu("lzss", raw, chunk)
    for k in want.meta:
        assert np.array_equal(want.meta[k], got.meta[k]), k
    assert np.array_equal(want.data, got.data)
