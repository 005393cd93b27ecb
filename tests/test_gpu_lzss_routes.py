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
