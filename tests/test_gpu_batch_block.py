"""Batch launches where whole blocks take Deflate tasks: Deflate alone, first,
last and mixed in, in every placement, and with lane streams so long that the
blocks have four warps."""
import numpy as np
import pytest

from compression_b200 import batch as B
from compression_b200 import codecs as cc
from compression_b200 import costmodel as CM

pytestmark = pytest.mark.gpu


def _deflate(seed, n):
    raw = cc.gen_markov_copy(seed, n, 32768)
    return B.Item("deflate", raw, B.encode_item("deflate", raw, seed))


def _items(kind: str) -> list:
    if kind == "deflate":
        return [_deflate(i, n) for i, n in enumerate([16, 4096, 300000, 70000, 1000, 128 * 1024] * 7)]
    if kind == "no deflate":
        return B.make_mixed_batch(5, 60, 12 << 20, mix=(0.25, 0.25, 0.2, 0.3, 0.0))
    if kind == "mixed":
        return B.make_mixed_batch(6, 200, 24 << 20)
    v = cc.gen_rlev1_ints(7, 1 << 19)  # 1 MiB chunks: lane streams of some 23 KB
    long = B.Item("rlev1", v.view(np.uint8), cc.rlev1_encode(v, 1 << 20, 128, 4))
    return [long] + [_deflate(20 + i, 50000 * (i + 1)) for i in range(6)] + B.make_mixed_batch(8, 30, 4 << 20)


@pytest.mark.parametrize("kind", ["deflate", "no deflate", "mixed", "long lanes"])
def test_orders(cuda, kind):
    import torch
    import oracle
    items = _items(kind)
    plan = B.build_plan(items)
    # the few RLE v2 items whose container does not round-trip in the reference
    expect = {i: oracle.decode(it.enc)[1][: it.enc.n_out] for i, it in enumerate(items) if it.codec == "rlev2"}
    size = plan.tasks["dst_len"].astype(np.float64)
    n = plan.tasks.size
    orders = [None, CM.lpt_order(size), CM.lpt_order(-size),
              torch.from_numpy(np.random.default_rng(1).permutation(n).astype(np.int32)).cuda(),
              CM.lpt_order(np.log(size + 1.0), CM.task_groups(plan), plan.tasks["codec"])]
    for k, order in enumerate(orders):
        for dynamic in (True, False):
            for bps in (0, 1):
                plan.d_out.zero_()
                plan.d_status.fill_(77)
                B.launch(plan, order, dynamic=dynamic, timing=k == 0, blocks_per_sm=bps)
                torch.cuda.synchronize()
                assert B.verify(plan, expect), (k, dynamic, bps, np.unique(plan.d_status.cpu().numpy()))
    if kind == "long lanes":
        assert B.n_warps(plan) % 4 == 0 and plan.max_lane > 16000
