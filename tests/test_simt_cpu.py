"""Device code run on the host, one block, a fiber per CUDA thread, under
schedules in which chosen warps or lanes are as late as the code allows
(tests/simt/cuda_runtime.h): what one thread reads after a barrier, the others
have had the time to change up to the next one.  A missing barrier gives a
wrong result here, a warp that comes apart a kernel that does not end."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
SIMT = ROOT / "tests" / "simt"
SCHEDULES = [0, 1, 2, 3, 4, 11, 12, 100, 101]  # see simt::schedule


def _compile(src: Path, out: Path, *flags) -> C.CDLL:
    cmd = ["g++", "-std=c++20", "-O1", "-w", "-shared", "-fPIC", "-I", str(SIMT), "-I",
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
