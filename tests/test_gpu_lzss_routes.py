"""LZSS decode on both sides of the choice between the block-per-columns and
the lane-per-column decoder: the number of chunks and the column length."""
import numpy as np
import pytest

from compression_b200 import codecs as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk,per_sm", [(3968, 0), (4096, 5), (16256, 5), (16384, 10)])
@pytest.mark.parametrize("over", [0, 1])
def test_number_of_chunks(cuda, chunk, per_sm, over):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = per_sm * sms + over if per_sm else 3 + over
    rng = np.random.default_rng(chunk + over)
    raw = np.resize(np.concatenate([rng.integers(0, k, 5 * chunk + 12, dtype=np.uint8) for k in (4, 256, 2, 1)]), n * chunk)
    job = cc.DeviceJob(cc.encode_gpu("lzss", raw, chunk))
    job.launch()
    torch.cuda.synchronize()
    assert not job.status().any()
    assert np.array_equal(job.output(), raw)


def _runs(rng, n: int, kind: int) -> np.ndarray:
    """A column of n bytes: repetitions of 1 to 5 bytes of any length one after
    the other (matches of one offset in a row, begun anywhere in it), or long
    stretches of literals between short repetitions."""
    out = []
    while len(out) < n:
        unit = rng.integers(0, 256, int(rng.integers(1, 6))).tolist()
        if kind == 0:
            out += (unit * 300)[:int(rng.choice([3, 34, 35, 36, 68, 70, 103, 200, 300]))]
        else:
            out += rng.integers(0, 256, int(rng.choice([7, 8, 31, 32, 33, 63, 64, 255, 256, 257, 300]))).tolist()
            out += (unit * 8)[:int(rng.integers(3, 9))]
    return np.array(out[:n], np.uint8)


@pytest.mark.parametrize("chunk", [4096, 16384, 65536, 131072])
def test_repetitions_and_literals(cuda, chunk):
    import torch
    rng = np.random.default_rng(chunk)
    raw = np.concatenate([np.stack([_runs(rng, chunk // 32, (q + c) % 2 if c else 0).reshape(-1, 4) for q in range(32)], 1)
                          .reshape(-1) for c in range(4)] + [rng.integers(0, 256, chunk, dtype=np.uint8), np.zeros(chunk, np.uint8)])
    job = cc.DeviceJob(cc.lzss_encode(raw, chunk))
    job.launch()
    torch.cuda.synchronize()
    assert not job.status().any()
    assert np.array_equal(job.output(), raw)
