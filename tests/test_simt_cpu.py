"""Device code run on the host, one block, a fiber per CUDA thread, under
schedules in which chosen warps or lanes are as late as the code allows
(tests/simt/cuda_runtime.h): what one thread reads after a barrier, the others
have had the time to change up to the next one.  A missing barrier gives a
wrong result here, a warp that comes apart a kernel that does not end."""
import ctypes as C
import struct
import subprocess
import zlib
from pathlib import Path

import numpy as np
import pytest

from compression_b200 import codecs as cc
from compression_b200._lib import lib

ROOT = Path(__file__).resolve().parent.parent
SIMT = ROOT / "tests" / "simt"
SCHEDULES = [0, 1, 2, 3, 4, 11, 12, 100, 101]  # see simt::schedule


def _compile(src: Path, out: Path, *flags) -> C.CDLL:
    cmd = ["g++", "-std=c++20", "-O1", "-w", "-fno-extern-tls-init", "-shared", "-fPIC", "-I", str(SIMT), "-I",
           str(ROOT / "compression_b200" / "csrc"), *flags, str(src), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(out))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.fixture(scope="module")
def turns(tmp_path_factory):
    f = _compile(SIMT / "batch_turns.cpp", tmp_path_factory.mktemp("simt") / "turns.so").turns

    def run(wpb, deflate, order, dynamic, grid, kind):
        d = np.asarray(deflate, np.uint8)
        o = None if order is None else np.asarray(order, np.uint32)
        w, b = np.zeros(d.size, np.uint32), np.zeros(d.size, np.uint32)
        n = d.size if o is None else o.size
        assert f(wpb, n, _p(d), None if o is None else _p(o), int(dynamic), grid, kind, _p(w), _p(b)) == 0, "hangs"
        return w, b
    return run


@pytest.mark.parametrize("kind", SCHEDULES)
@pytest.mark.parametrize("wpb", [8, 4])
@pytest.mark.parametrize("dynamic", [True, False])
def test_every_task_once(turns, wpb, dynamic, kind):
    rng = np.random.default_rng(wpb + kind)
    for n in (1, 7, 8, 9, 60):
        for share in (0.0, 0.1, 0.5, 1.0):
            deflate = rng.random(n) < share
            for order in (None, rng.permutation(n)):
                w, b = turns(wpb, deflate, order, dynamic, 2, kind)
                assert (w == np.where(deflate, 0, 32)).all() and (b == np.where(deflate, 32 * wpb, 0)).all(), (n, share)


@pytest.mark.parametrize("kind", [0, 4])
@pytest.mark.parametrize("dynamic", [True, False])
def test_entries_out_of_range(turns, dynamic, kind):
    """An order entry that names no task costs nobody a task."""
    rng = np.random.default_rng(kind)
    n = 120
    deflate = rng.random(n) < 0.2
    order = rng.permutation(n).astype(np.uint32)
    order = order[: n - 40]
    for k in rng.choice(order.size, 20, replace=False):
        order[k] = [n, n + 5, 0xffffffff, 0xfffffffe, 0x80000000][k % 5]
    named = np.isin(np.arange(n), order)
    w, b = turns(8, deflate, np.concatenate([order, np.full(40, n, np.uint32)]), dynamic, 2, kind)
    assert (w == np.where(named & ~deflate, 32, 0)).all() and (b == np.where(named & deflate, 256, 0)).all()


@pytest.fixture(scope="module")
def inflate(tmp_path_factory):
    lib_ = _compile(SIMT / "inflate_block.cpp", tmp_path_factory.mktemp("simt") / "inflate.so")

    def run(shape, comp: bytes, n: int, kind: int, at: int = 0):
        """The n bytes written at an address `at` above a multiple of 16."""
        src = np.zeros(len(comp) + 32, np.uint8)
        s0 = -src.ctypes.data % 16
        src[s0:s0 + len(comp)] = np.frombuffer(comp, np.uint8)
        dst = np.full(n + 64, 0x5A, np.uint8)
        d0 = -dst.ctypes.data % 16 + at
        w = C.c_uint32()
        st = lib_.inflate(shape, _p(src[s0:]), len(comp), _p(dst[d0:]), n, 0, kind, C.byref(w))
        assert st == 0 and w.value == n
        assert (dst[:d0] == 0x5A).all() and (dst[d0 + n:] == 0x5A).all()
        return dst[d0:d0 + n]
    run.write_at = lib_.write_at
    run.barriers = lib_.barriers
    run.barriers.restype = C.c_uint64
    return run


def _stored(parts) -> bytes:
    """The parts as stored blocks, after a compressed one of 5 bytes."""
    c = zlib.compressobj(6, zlib.DEFLATED, -15)
    out = c.compress(b"abcde") + c.flush(zlib.Z_FULL_FLUSH)
    for i, p in enumerate(parts):
        out += struct.pack("<BHH", i == len(parts) - 1, len(p), len(p) ^ 0xffff) + p
    return out


@pytest.mark.parametrize("shape,window", [(1, 65536), (2, 32768), (3, 32768), (4, 16384), (5, 16384)])
@pytest.mark.parametrize("kind", [0, 4])
def test_stored_blocks_around_the_window(inflate, shape, window, kind):
    """Stored blocks of about the window's length at odd places."""
    rng = np.random.default_rng(shape)
    for at in (0, 3):
        parts = [rng.bytes(min(65535, window + k)) for k in (-33, 40, 7, 100)]
        got = inflate(shape, _stored(parts), 5 + sum(map(len, parts)), kind, at)
        assert got.tobytes() == b"abcde" + b"".join(parts)


@pytest.fixture(scope="module")
def lzss_columns(tmp_path_factory):
    text = (ROOT / "compression_b200" / "csrc" / "encode.cu").read_text()
    tmp = tmp_path_factory.mktemp("simt")
    (tmp / "cols.inc").write_text(text[text.index("constexpr uint32_t LZ_WPB"):text.index("// A warp per chunk: slots")])
    return _compile(SIMT / "lzss_columns.cpp", tmp / "lzss.so", f'-DLZSS_COLUMNS="{tmp / "cols.inc"}"').lzss_columns


@pytest.mark.parametrize("chunk", [1024, 8192, 8320, 65536, 131072])
@pytest.mark.parametrize("kind", [0, 1, 2, 11])
def test_lzss_columns_match_the_host_encoder(lzss_columns, chunk, kind):
    rng = np.random.default_rng(chunk)
    n = chunk // 32
    text = cc.gen_markov_copy(3, n, 4096)
    fresh = np.zeros(n, np.uint8)  # words repeated at once, not seen before
    for p in range(0, n - 31, 32):
        fresh[p:p + 8] = fresh[p + 10:p + 18] = rng.integers(1, 256, 8) if p % 96 == 0 else 0
    cols = [fresh, rng.integers(0, 2, n, dtype=np.uint8), text, rng.integers(0, 12, n, dtype=np.uint8)]
    raw = np.stack([(cols * 8)[q].reshape(-1, 4) for q in range(32)], 1).reshape(-1).copy()
    cap = n + n // 8 + 12 & ~3
    scratch, raw_len = np.zeros(32 * cap, np.uint8), np.zeros(32, np.uint32)
    assert lzss_columns(_p(raw), C.c_uint64(chunk), 0, 4, _p(scratch), cap, _p(raw_len), kind) == 0
    for q in range(4):
        want = np.zeros(cap, np.uint8)
        m = lib().gd_lzss_encode_stream(_p(cols[q]), n, _p(want), cap)
        assert raw_len[q] == m and np.array_equal(scratch[q * cap:q * cap + m], want[:m]), q


@pytest.mark.parametrize("stored", [0, 1])
def test_output_positions_past_32_bits(inflate, stored):
    """The last bytes of a stream of up to 2^32 - 1 bytes, whose output may
    start up to 15 bytes after a multiple of 16."""
    rng = np.random.default_rng(stored)
    for start in (2**32 - 8192, 2**32 - 4096 - 5, 2**32 - 16, 2**32 - 1, 5):
        for n in (1, 15, 16, 33, 4095, 8190):
            src, dst = rng.integers(0, 256, n + 32, dtype=np.uint8), np.full(n + 64, 0x5A, np.uint8)
            s0, d0 = -src.ctypes.data % 16, -dst.ctypes.data % 16 + start % 16
            assert inflate.write_at(start % 2**32, _p(src[s0:]), n, _p(dst[d0:]), stored, 4) == 0
            assert np.array_equal(dst[d0:d0 + n], src[s0:s0 + n])
            assert (dst[:d0] == 0x5A).all() and (dst[d0 + n:] == 0x5A).all(), (start, n)


@pytest.mark.parametrize("shape,most", [(1, 300), (2, 450), (3, 650), (4, 650), (5, 800)])
def test_codes_that_do_not_fall_back_into_step(inflate, shape, most):
    """Random 7-bit values: codes of one length, whose phase a thread keeps.
    The threads' starts travel along the segments, a barrier or two each; they
    do so once, and only over the segments that a step has room for."""
    raw = np.random.default_rng(1).integers(0, 128, 20000, dtype=np.uint8)
    c = zlib.compressobj(6, zlib.DEFLATED, -15, 8, zlib.Z_HUFFMAN_ONLY)
    before = inflate.barriers()
    assert np.array_equal(inflate(shape, c.compress(raw.tobytes()) + c.flush(), raw.size, 0), raw)
    assert inflate.barriers() - before <= most
