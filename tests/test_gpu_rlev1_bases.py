"""RLE v1 runs whose bases are varints of every length, and lane streams cut
in their last run, against the oracle."""
import numpy as np
import pytest

from compression_b200 import codecs as cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem", [4, 8])
def test_bases(cuda, elem):
    import oracle
    rng = np.random.default_rng(elem)
    top = 5 if elem == 4 else 10
    v = []
    for i in range(3000):
        bits = 7 * (i % top) + int(rng.integers(1, 8))
        base = min((1 << bits) - 1, (1 << 8 * elem) - 200) if i % 3 else int(rng.integers(0, 1 << min(bits, 8 * elem - 1)))
        v += [(base + k * (i % 5)) & ((1 << 8 * elem) - 1) for k in range(int(rng.choice([3, 4, 8, 33, 129])))]
    v = np.array(v, np.uint64).astype(np.uint32 if elem == 4 else np.uint64)
    chunk = 32 * 128 * 4
    enc = cc.rlev1_encode(v, chunk, 128, elem)
    job = cc.DeviceJob(enc, cuda)
    job.launch()
    assert not job.status().any() and np.array_equal(job.output(), v.view(np.uint8))
    # a lane's stream cut inside its last word (the block's rows stay as they are)
    lens = enc.meta["col_len"].copy().reshape(-1, 32)
    for c in range(0, enc.n_chunks - 1):
        spare = (lens[c].astype(int) - 1) % 4
        lane = int(rng.choice(np.flatnonzero(spare)))
        lens[c, lane] -= int(rng.integers(1, spare[lane] + 1))
    lens = lens.reshape(-1)
    enc.meta["col_len"] = lens
    job = cc.DeviceJob(enc, cuda)
    job.launch()
    st = job.status()
    assert (st[:-1] != 0).all() and st[-1] == 0
    assert oracle.decode(enc)[0] != 0
