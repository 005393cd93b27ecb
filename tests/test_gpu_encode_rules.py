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


@pytest.mark.parametrize("codec,elem", [("rlev1", 4), ("rlev1", 8), ("rlev2", 8)])
def test_short_runs_in_a_row(cuda, codec, elem):
    """Runs that a warp takes together: of 3 to 70 values, values of every
    width, up to the ends of the window and of the lane, literals between."""
    rng = np.random.default_rng(elem)
    n, dt = 700, np.int32 if elem == 4 else np.int64
    lanes = []
    for q in range(32):
        x = []
        while len(x) < n:
            k = int(rng.choice([3, 4, 5, 8, 9, 10, 11, 12, 30, 31, 32, 63, 64, 65, 70][:15 - q % 8]))
            base = int(rng.integers(-1 << int(rng.integers(1, 8 * elem - 1)), 1 << int(rng.integers(1, 8 * elem - 1))))
            x += [base + i * (int(rng.integers(-5, 6)) if codec == "rlev1" and q % 3 == 0 else 0) for i in range(k)]
            if q % 4 == 1 and rng.random() < 0.1:
                x += rng.integers(0, 1000, int(rng.integers(1, 40))).tolist()
        lanes.append(np.array(x[:n], np.int64).astype(dt))
    raw = np.concatenate(lanes)  # slices as long as the lanes: lane after lane
    if codec == "rlev1":
        want = cc.rlev1_encode(raw, raw.nbytes, n * elem, elem)
        got = cc.encode_gpu("rlev1", raw, raw.nbytes, comp_col_len=n * elem, elem_bytes=elem)
    else:
        want = cc.rlev2_encode(raw, raw.nbytes, n)
        got = cc.encode_gpu("rlev2", raw, raw.nbytes, read_unit=n)
    for k in want.meta:
        assert np.array_equal(want.meta[k], got.meta[k]), k
    assert np.array_equal(want.data, got.data)
