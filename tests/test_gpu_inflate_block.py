"""The block-per-stream inflate kernels at the sizes and contents where they can
go wrong: segment, batch, placement and window edges, codes that never fall
back into step, long runs, every block type and header, unaligned outputs.
Bytes are exact, against zlib."""
import struct
import zlib

import numpy as np
import pytest

from compression_b200 import codecs as cc

pytestmark = pytest.mark.gpu
rng = np.random.default_rng(5)


def _deflate(data: bytes, level=6, strategy=zlib.Z_DEFAULT_STRATEGY, wbits=15, flush_every=0) -> bytes:
    c = zlib.compressobj(level, zlib.DEFLATED, wbits, 9, strategy)
    if not flush_every:
        return c.compress(data) + c.flush()
    out = b""
    for i in range(0, len(data), flush_every):
        out += c.compress(data[i:i + flush_every]) + c.flush(zlib.Z_FULL_FLUSH)
    return out + c.flush()


def _streams() -> list:
    mk = cc.gen_markov_copy(9, 1 << 20, 32768).tobytes()
    flat = bytes(rng.integers(0, 128, 70000, dtype=np.uint8))   # equal 7-bit codes: no segment falls back into step
    far = bytes(rng.integers(0, 256, 32768, dtype=np.uint8))
    s = [(b"", {}), (b"a", {}), (b"ab" * 2, {}), (mk[:257], {}), (mk[:4097], {}), (mk, {}), (mk, {"level": 1}),
         (mk, {"level": 9, "flush_every": 777}), (mk[:200001], {"level": 0}), (mk[:300000], {"strategy": zlib.Z_FIXED}),
         (mk[:300000], {"strategy": zlib.Z_HUFFMAN_ONLY}), (flat, {"strategy": zlib.Z_HUFFMAN_ONLY}),
         (bytes(1 << 20), {}), (b"abc" * 100000, {}), (mk[:100] * 3000, {}), (far * 4, {}),   # distance 32768
         ((far[:300] + bytes(900)) * 60, {"level": 9}), (mk[:5000] + far + mk[:5000], {"flush_every": 4096})]
    for n in (1, 2, 3, 15, 16, 17, 31, 33, 8031, 8032, 8033, 16225, 32609):
        s.append((mk[n:2 * n], {}))
    return s


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("hdr", [0, 1, 2])
def test_streams(cuda, variant, hdr):
    import compression_b200.autotune as at
    wbits = {0: -15, 1: 15, 2: 31}[hdr]
    raws, comps = [], []
    for data, kw in _streams():
        raws.append(np.frombuffer(data, np.uint8))
        comps.append(np.frombuffer(_deflate(data, wbits=wbits, **kw), np.uint8))
    off, pos = [], 0
    for c in comps:  # odd starts: the kernels read aligned words around them
        off.append(pos)
        pos += c.size + 3
    data = np.zeros(pos, np.uint8)
    for o, c in zip(off, comps):
        data[o:o + c.size] = c
    oo = np.concatenate([[0], np.cumsum([r.size for r in raws])]).astype(np.uint64)
    enc = cc.Encoded("deflate", data, int(oo[-1]), len(raws), 0,
                     {"comp_off": np.array(off + [pos], np.uint64),
                      "comp_len": np.array([c.size for c in comps], np.uint64), "out_off": oo}, {"zlib_header": hdr})
    prev = at.set_knob(at.TUNE_INFLATE_VARIANT, variant)
    try:
        job = cc.DeviceJob(enc, cuda)
        job.launch()
        st, out = job.status(), job.output()
    finally:
        at.set_knob(at.TUNE_INFLATE_VARIANT, prev)
    assert (st == 0).all(), np.flatnonzero(st)
    assert np.array_equal(out, np.concatenate(raws))


@pytest.mark.parametrize("variant", [1, 2, 3, 4])
def test_malformed(cuda, variant):
    """Cut, damaged and mis-sized streams: a status of their own, the others whole."""
    import compression_b200.autotune as at
    raw = cc.gen_markov_copy(3, 40 * 30000, 32768)
    oo = np.arange(0, 41 * 30000, 30000, dtype=np.uint64)
    enc = cc.deflate_encode(raw, oo, 6)
    bad = {}
    co, cl = enc.meta["comp_off"], enc.meta["comp_len"].copy()
    for i in range(0, 40, 4):
        o, n = int(co[i]), int(cl[i])
        if i % 3 == 0:
            cl[i] = max(8, n * (i + 1) // 48)               # truncated
        elif i % 3 == 1:
            enc.data[o + 2] |= 7                            # block type 3
        else:
            enc.data[o + n // 2:o + n // 2 + 40] ^= 0x5A    # damaged symbols
        bad[i] = True
    enc.meta["comp_len"] = cl
    prev = at.set_knob(at.TUNE_INFLATE_VARIANT, variant)
    try:
        job = cc.DeviceJob(enc, cuda)
        job.launch()
        st, out = job.status(), job.output()
    finally:
        at.set_knob(at.TUNE_INFLATE_VARIANT, prev)
    for i in range(40):
        if i not in bad:
            assert st[i] == 0 and np.array_equal(out[i * 30000:(i + 1) * 30000], raw[i * 30000:(i + 1) * 30000]), i
        elif i % 3 != 2:
            assert st[i] in (2, 3), (i, st[i])


def _stored(n: int, size: int) -> tuple:
    """n bytes in stored blocks of `size`, after a compressed block of 5 bytes."""
    raw = b"abcde" + rng.bytes(n)
    c = zlib.compressobj(6, zlib.DEFLATED, -15)
    comp = c.compress(raw[:5]) + c.flush(zlib.Z_FULL_FLUSH)
    for i in range(5, len(raw), size):
        p = raw[i:i + size]
        comp += struct.pack("<BHH", i + size >= len(raw), len(p), len(p) ^ 0xffff) + p
    return np.frombuffer(raw, np.uint8), np.frombuffer(comp, np.uint8)


STORED = [16384 - 33, 16384 + 7, 32768 - 16, 32768 + 40, 65535]


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4])
def test_stored_blocks_around_the_window(cuda, variant):
    import compression_b200.autotune as at
    raws, comps = zip(*[_stored(300001, size) for size in STORED for _ in range(60)])
    off = np.concatenate([[0], np.cumsum([c.size + 3 for c in comps])])
    data = np.zeros(int(off[-1]), np.uint8)
    for o, c in zip(off, comps):
        data[o:o + c.size] = c
    oo = np.concatenate([[0], np.cumsum([r.size for r in raws])]).astype(np.uint64)
    enc = cc.Encoded("deflate", data, int(oo[-1]), len(raws), 0,
                     {"comp_off": off.astype(np.uint64), "comp_len": np.array([c.size for c in comps], np.uint64),
                      "out_off": oo}, {"zlib_header": 0})
    prev = at.set_knob(at.TUNE_INFLATE_VARIANT, variant)
    try:
        job = cc.DeviceJob(enc, cuda)
        job.launch()
        st, out = job.status(), job.output()
    finally:
        at.set_knob(at.TUNE_INFLATE_VARIANT, prev)
    assert (st == 0).all() and np.array_equal(out, np.concatenate(raws))


@pytest.mark.parametrize("long_lanes", [False, True])
def test_stored_blocks_in_a_batch(cuda, long_lanes):
    """By blocks of eight warps, and of four (lane streams of some 23 KB)."""
    import torch
    from compression_b200 import batch as B
    items = []
    for size in STORED * 4:
        raw, comp = _stored(100003, size)
        meta = {"comp_off": np.array([0, comp.size], np.uint64), "comp_len": np.array([comp.size], np.uint64),
                "out_off": np.array([0, raw.size], np.uint64)}
        items.append(B.Item("deflate", raw, cc.Encoded("deflate", comp, raw.size, 1, 0, meta, {"zlib_header": 0})))
    if long_lanes:
        v = cc.gen_rlev1_ints(7, 1 << 19)
        items.append(B.Item("rlev1", v.view(np.uint8), cc.rlev1_encode(v, 1 << 20, 128, 4)))
    plan = B.build_plan(items, cuda)
    for dynamic in (True, False):
        plan.d_out.zero_()
        B.launch(plan, None, dynamic=dynamic)
        torch.cuda.synchronize()
        assert B.verify(plan)


def test_largest_stream(cuda):
    """A stream of 2^32 - 1 bytes, the most an entry point takes."""
    n, mid = 2**32 - 1, 16 << 20
    head, tail = rng.bytes(70000), rng.bytes(70001)
    c = zlib.compressobj(6, zlib.DEFLATED, -15)
    first = c.compress(head) + c.flush(zlib.Z_FULL_FLUSH)
    zeros = c.compress(bytes(mid)) + c.flush(zlib.Z_FULL_FLUSH)
    k, rest = divmod(n - len(head) - len(tail), mid)
    comp = np.frombuffer(first + zeros * k + c.compress(bytes(rest) + tail) + c.flush(), np.uint8)
    enc = cc.Encoded("deflate", comp, n, 1, 0,
                     {"comp_off": np.array([0, comp.size], np.uint64), "comp_len": np.array([comp.size], np.uint64),
                      "out_off": np.array([0, n], np.uint64)}, {"zlib_header": 0})
    job = cc.DeviceJob(enc, cuda)
    job.launch()
    assert (job.status() == 0).all()
    out = job.d_out[:n]
    assert out[:len(head)].cpu().numpy().tobytes() == head and out[n - len(tail):].cpu().numpy().tobytes() == tail
    for a in range(len(head), n - len(tail), 1 << 30):
        assert not out[a:min(a + (1 << 30), n - len(tail))].any()
