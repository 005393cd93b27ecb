"""RLE v1 and v2 columns on both sides of the choice between a thread and a warp
per lane stream: the values of a lane, the number of lanes, and, in large columns,
short runs or none. The container is the host encoder's either way."""
import numpy as np
import pytest

from compression_b200 import codecs as cc

pytestmark = pytest.mark.gpu


def _column(rng, kind: str, n: int, dt) -> np.ndarray:
    if kind == "runs":
        v = np.repeat(rng.integers(0, 100, n // 5 + 1), rng.integers(3, 9, n // 5 + 1))
    elif kind == "values":
        v = rng.integers(0, 1 << 20, n)
    else:  # half of each: whichever the sample says, for all chunks
        v = np.concatenate([np.repeat(rng.integers(0, 100, n // 10), 5), rng.integers(0, 1 << 20, n)])
    return np.resize(v, n).astype(dt)


@pytest.mark.parametrize("kind", ["runs", "values", "both"])
@pytest.mark.parametrize("codec,elem,n,lanes", [
    ("rlev1", 4, 15, 64), ("rlev1", 4, 16, 8160), ("rlev1", 4, 16, 8192), ("rlev1", 4, 32, 32768), ("rlev1", 8, 63, 96),
    ("rlev1", 8, 64, 16352), ("rlev1", 8, 64, 16384), ("rlev1", 8, 64, 32768), ("rlev1", 4, 64, 65536), ("rlev1", 4, 512, 16416),
    ("rlev2", 8, 3, 64), ("rlev2", 8, 4, 8192), ("rlev2", 8, 16, 16384), ("rlev2", 8, 16, 32768), ("rlev2", 8, 32, 16384),
    ("rlev2", 8, 512, 16416)])
def test_choice(cuda, codec, elem, n, lanes, kind):
    rng = np.random.default_rng(n + lanes)
    unit = 16 if n % 16 == 0 else n
    raw = _column(rng, kind, n * lanes - 7, np.int32 if elem == 4 else np.int64)
    chunk = 32 * n * elem
    if codec == "rlev1":
        want = cc.rlev1_encode(raw, chunk, unit * elem, elem)
        got = cc.encode_gpu("rlev1", raw, chunk, comp_col_len=unit * elem, elem_bytes=elem)
    else:
        want = cc.rlev2_encode(raw, chunk, unit)
        got = cc.encode_gpu("rlev2", raw, chunk, read_unit=unit)
    for k in want.meta:
        assert np.array_equal(want.meta[k], got.meta[k]), k
    assert np.array_equal(want.data, got.data)
