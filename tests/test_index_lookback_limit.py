"""The decoders' index waits with a limit too.

The CTA-wide look-back that turns a stream's size index into offsets runs over
tiles of which one never publishes: the tiles behind it give up after a small
number of polls, the call reports it, and the next call works.  With nothing
withheld the prefixes are exact.  Scan 2 reads the status words sixteen bytes at
a time, scan 3 one by one (words behind an odd multiple of eight bytes)."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

ERR_LOOKBACK = 1


@pytest.fixture(scope="module")
def L():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required")
    from szx_gb300 import build
    build.build()
    from szx_gb300._lib import lib
    L = lib()
    L.SZxG_selftest_lookback.restype = C.c_int
    L.SZxG_selftest_lookback.argtypes = [C.c_int, C.c_int, C.c_int, C.c_uint, C.c_void_p, C.c_void_p]
    return L


def _run(L, scan, ntiles, withheld, limit):
    import torch
    pre = np.zeros(ntiles, np.uint64)
    t0 = time.perf_counter()
    rc = L.SZxG_selftest_lookback(scan, ntiles, withheld, limit, pre.ctypes.data,
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return rc, pre, time.perf_counter() - t0


@pytest.mark.parametrize("scan", [2, 3])
@pytest.mark.parametrize("ntiles", [1, 2, 5, 128, 129, 1000])
def test_prefixes_are_exact(L, scan, ntiles):
    rc, pre, _ = _run(L, scan, ntiles, -1, 1 << 22)
    assert rc == 0
    t = np.arange(ntiles, dtype=np.uint64)
    assert np.array_equal(pre, t * (t + 1) // 2)


@pytest.mark.parametrize("scan", [2, 3])
@pytest.mark.parametrize("withheld", [0, 37, 999])
def test_gives_up_on_a_tile_that_never_publishes(L, scan, withheld):
    import szx_gb300 as S
    rc, pre, dt = _run(L, scan, 1000, withheld, 4000)
    t = np.arange(withheld, dtype=np.uint64)
    assert np.array_equal(pre[:withheld], t * (t + 1) // 2)   # tiles before the gap are exact
    if withheld == 999:   # nobody waits on the last tile
        assert rc == 0
    else:
        assert rc == ERR_LOOKBACK
        assert L.SZxG_get_last_error() == ERR_LOOKBACK
    assert dt < 5.0
    # the context is still usable: a decompress whose index runs that look-back
    x = np.sin(np.arange(3_000_001, dtype=np.float32) / 50)
    s = S.fast_compress_args(3, x, S.ABS, 1e-3)
    assert S.fast_decompress(3, np.float32, s, x.size).tobytes() == O.decompress(3, np.float32, s, x.size).tobytes()


def test_other_scans_are_refused(L):
    for scan in (-1, 4):
        rc, _, _ = _run(L, scan, 8, -1, 100)
        assert rc != 0
