"""Performance cases: the codec calls a program makes, over the sizes it makes them at.

Every case is one kind of call on one seeded column:

  decode   a container already in device memory, decoded by DeviceJob.launch
           (the compressed bytes and metadata a scan keeps resident);
  encode   a column in device memory written as a container by encode_device,
           with the buffers of an earlier call reused;
  batch    thousands of warp-sized tasks of all five codecs in one launch
           through the work queue, longest output first;
  host     the synchronous call on host buffers (copy in, decode, copy out).

Columns come from the library's generators, which restate the benchmark's
data: alternating runs and literal groups (RLE v1), short byte runs (byte-RLE),
delta / repeat / direct / outlier segments (RLE v2), and a Markov source with
copies (LZSS, Deflate).
"""
from __future__ import annotations

import concurrent.futures as cf
import math
import os
import random

import numpy as np
import torch

from compression_b200 import batch as B
from compression_b200 import codecs as cc
from compression_b200 import costmodel as CM

KiB, MiB = 1 << 10, 1 << 20

# compressed bytes per column byte of the generators' data, to three digits
RATIO = {"brle": 0.0836, "rlev1": 0.701, "rlev1_64": 0.331, "rlev2": 0.480, "lzss": 0.715, "deflate": 0.0537,
         "batch": 0.411}


def listed() -> list[dict]:
    return [
        # a full byte column (flags, dictionary codes) read by a scan
        {"name": "brle_decode_256m", "op": "decode", "codec": "brle", "n": 256 * MiB, "chunk": 256 * KiB},
        # a full int32 column
        {"name": "rlev1_decode_64m", "op": "decode", "codec": "rlev1", "n": 64 * MiB, "chunk": 128 * KiB, "elem": 4},
        # one small int64 row group with a partial last chunk: latency and launches count
        {"name": "rlev1_decode_i64_1m", "op": "decode", "codec": "rlev1", "n": 1 * MiB + 24 * KiB + 8,
         "chunk": 128 * KiB, "elem": 8},
        # a full int64 column (timestamps, keys, measures)
        {"name": "rlev2_decode_256m", "op": "decode", "codec": "rlev2", "n": 256 * MiB, "chunk": 256 * KiB},
        # a full text-like column
        {"name": "lzss_decode_256m", "op": "decode", "codec": "lzss", "n": 256 * MiB, "chunk": 64 * KiB},
        # thousands of zlib streams of uneven size (pages of a file), 3% of them fixed or stored
        {"name": "inflate_256m", "op": "decode", "codec": "deflate", "n": 256 * MiB, "streams": 2048, "lo": 4 * KiB,
         "hi": 1 * MiB, "level": 6},
        # one page group of few uniform streams, the last one short: the chip is nearly idle
        {"name": "inflate_few_5m", "op": "decode", "codec": "deflate", "n": 5000003, "chunk": 128 * KiB, "level": 6},
        # a mixed batch of items of uneven size (4 KiB to 2 MiB before scaling)
        {"name": "batch_256m", "op": "batch", "n": 256 * MiB, "items": 1024},
        # columns written on the device
        {"name": "rlev1_encode_64m", "op": "encode", "codec": "rlev1", "n": 64 * MiB, "chunk": 128 * KiB, "elem": 4},
        {"name": "rlev2_encode_64m", "op": "encode", "codec": "rlev2", "n": 64 * MiB, "chunk": 256 * KiB},
        {"name": "lzss_encode_64m", "op": "encode", "codec": "lzss", "n": 64 * MiB, "chunk": 64 * KiB},
        # a small column of odd size decoded from host memory to host memory
        {"name": "brle_host_3m", "op": "host", "codec": "brle", "n": 3000001},
    ]


def _size(rng: random.Random, lo: int, hi: int, granule: int) -> int:
    """Log-uniform in [lo, hi], a multiple of the value size."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(granule, int(x) // granule * granule)


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["brle", "rlev1", "rlev2", "lzss", "inflate", "inflate_uniform", "batch", "enc_rlev1",
                       "enc_rlev2", "enc_lzss", "host"])
    if kind == "brle":
        return {"op": "decode", "codec": "brle", "n": _size(rng, MiB, 256 * MiB, 1), "chunk": 256 * KiB}
    if kind == "rlev1":
        e = rng.choice([4, 8])
        return {"op": "decode", "codec": "rlev1", "n": _size(rng, MiB, 64 * MiB, e), "chunk": 128 * KiB, "elem": e}
    if kind == "rlev2":
        return {"op": "decode", "codec": "rlev2", "n": _size(rng, MiB, 256 * MiB, 8), "chunk": 256 * KiB}
    if kind == "lzss":
        return {"op": "decode", "codec": "lzss", "n": _size(rng, MiB, 256 * MiB, 1),
                "chunk": rng.choice([64, 128]) * KiB}
    if kind == "inflate":
        n = _size(rng, 4 * MiB, 256 * MiB, 1)
        return {"op": "decode", "codec": "deflate", "n": n, "streams": max(8, n // (128 * KiB)), "lo": 4 * KiB,
                "hi": 1 * MiB, "level": rng.choice([1, 6, 9])}
    if kind == "inflate_uniform":
        return {"op": "decode", "codec": "deflate", "n": _size(rng, MiB, 64 * MiB, 1),
                "chunk": rng.choice([64, 128, 256]) * KiB, "level": rng.choice([1, 6, 9])}
    if kind == "batch":
        n = _size(rng, 64 * MiB, 256 * MiB, 16)
        return {"op": "batch", "n": n, "items": n // (256 * KiB)}
    if kind == "enc_rlev1":
        e = rng.choice([4, 8])
        return {"op": "encode", "codec": "rlev1", "n": _size(rng, MiB, 64 * MiB, e), "chunk": 128 * KiB, "elem": e}
    if kind == "enc_rlev2":
        return {"op": "encode", "codec": "rlev2", "n": _size(rng, MiB, 64 * MiB, 8), "chunk": 256 * KiB}
    if kind == "enc_lzss":
        return {"op": "encode", "codec": "lzss", "n": _size(rng, MiB, 64 * MiB, 1),
                "chunk": rng.choice([64, 128]) * KiB}
    return {"op": "host", "codec": "brle", "n": _size(rng, MiB, 16 * MiB, 1)}


def _column(case: dict, seed: int) -> np.ndarray:
    c, n = case["codec"], case["n"]
    if c == "brle":
        return cc.gen_brle_bytes(seed, n)
    if c == "rlev1":
        v = cc.gen_rlev1_ints(seed, n // case["elem"])
        return v if case["elem"] == 4 else v.astype(np.int64)
    if c == "rlev2":
        return cc.gen_rlev2_ints(seed, n // 8)
    return cc.gen_markov_copy(seed, n, 4096 if c == "lzss" else 32768)


def _encode(case: dict, seed: int) -> cc.Encoded:
    raw = _column(case, seed)
    c = case["codec"]
    if c == "brle":
        return cc.brle_encode(raw)
    if c == "rlev1":
        return cc.rlev1_encode(raw, case["chunk"], 128, case["elem"])
    if c == "rlev2":
        return cc.rlev2_encode(raw, case["chunk"], 32)
    if c == "lzss":
        return cc.lzss_encode(raw, case["chunk"])
    n = case["n"]
    if "streams" in case:
        sizes = cc.loguniform_sizes(seed, case["streams"], case["lo"], case["hi"], n, 1)
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    else:
        off = np.append(np.arange(0, n, case["chunk"]), n).astype(np.uint64)
    u = np.random.default_rng(seed).random(off.size - 1)
    mode = np.where(u < 0.015, 1, np.where(u < 0.03, 2, 0)).astype(np.uint8)
    return cc.deflate_encode(raw, off, case["level"], mode, 1)


def _batch_items(case: dict, seed: int) -> list:
    """Items of all codecs, sizes log-uniform over 4 KiB to 2 MiB and scaled to
    the total: 20% RLE v1, 20% RLE v2, 10% byte-RLE, 25% LZSS, 25% Deflate.
    The layout (sizes and codecs) belongs to the case, the values to the seed."""
    k = case["items"]
    sizes = cc.loguniform_sizes(k, k, 4 * KiB, 2 * MiB, case["n"], 16)
    order = np.repeat(["rlev1", "rlev2", "brle", "lzss", "deflate"], [20, 20, 10, 25, 25])
    codecs = np.random.default_rng(k).permutation(np.resize(order, k))

    def one(i: int):
        codec, g = str(codecs[i]), B.GRANULE[str(codecs[i])]
        n = max(g, int(sizes[i]) // g * g)
        raw = _column({"codec": codec, "n": n, "elem": 4}, seed * 100003 + i).view(np.uint8)
        return B.Item(codec, raw, B.encode_item(codec, raw, k * 7 + i))

    with cf.ThreadPoolExecutor(os.cpu_count() or 1) as ex:
        return list(ex.map(one, range(k)))


def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    if op == "decode":
        return {"op": op, "job": cc.DeviceJob(_encode(case, seed))}
    if op == "host":
        return {"op": op, "enc": _encode(case, seed)}
    if op == "batch":
        plan = B.build_plan(_batch_items(case, seed))
        t = plan.tasks
        # longest first by output bytes (an RLE task writes a 32nd of its chunk)
        out = t["dst_len"].astype(np.float64) / np.where(np.isin(t["codec"], (1, 2)), 32.0, 1.0)
        order = CM.lpt_order(np.log(out + 1.0), CM.task_groups(plan), t["codec"])
        return {"op": op, "plan": plan, "order": order}
    col = torch.from_numpy(_column(case, seed).view(np.uint8)).cuda()
    kw = {"elem_bytes": case["elem"]} if "elem" in case else {}
    bufs = cc.encode_device(case["codec"], col, case["chunk"], **kw)  # the buffers a program keeps
    bufs["data"].zero_()  # the container ends before the buffer does
    return {"op": op, "codec": case["codec"], "col": col, "chunk": case["chunk"], "kw": kw, "bufs": bufs}


def run(state: dict):
    op = state["op"]
    if op == "decode":
        job = state["job"]
        job.launch()
        return {"out": job.d_out[:job.out_n], "status": job.d_status}
    if op == "host":
        return {"out": cc.decode_host(state["enc"])}
    if op == "batch":
        plan = state["plan"]
        B.launch(plan, state["order"], dynamic=True, timing=False)
        return {"out": plan.d_out, "status": plan.d_status}
    b = cc.encode_device(state["codec"], state["col"], state["chunk"], bufs=state["bufs"], **state["kw"])
    out = {"data": b["data"], "blk_off": b["blk_off"], "col_len": b["col_len"],
           "status": b["status"]}
    if state["codec"] == "lzss":
        out["col_map"] = b["col_map"]
    return out


def work(case: dict) -> dict:
    """Compressed and decompressed bytes, each moved once, and 8 bytes of
    length per lane stream; no floating-point work."""
    n = case["n"]
    codec = case.get("codec", "batch")
    r = RATIO["rlev1_64" if case.get("elem") == 8 else codec]
    meta = 0
    if codec in ("rlev1", "rlev2", "lzss"):
        meta = 8 * 33 * -(-n // case["chunk"])
    return {"bytes": int(n * (1.0 + r)) + meta, "flops": 0}
