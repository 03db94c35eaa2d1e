"""Blocks with NaNs (quiet, signalling, with payloads), infinities and both
zeros, where the reference's order of comparison and the x86 NaN rules decide:
first, last and inside a block, alone and all through it, beside zero extremes.
Streams equal the oracle's in every layout."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

BITS = {np.float32: (np.uint32, 0x7F800000, 0x00400000, 0x80000000),
        np.float64: (np.uint64, 0x7FF0000000000000, 0x0008000000000000, 0x8000000000000000)}


def _specials(dt):
    """(quiet NaN with a payload, negative signalling NaN, inf, -inf, +0, -0) as patterns."""
    u, inf, quiet, sign = BITS[dt]
    return np.array([inf | quiet | 5, sign | inf | 3, inf, sign | inf, 0, sign], u)


def _field(dt, bs, kind, rng):
    """61 blocks and a part of one; block b holds special b % 6 (and a second one in half of them)."""
    n = 61 * bs + max(1, bs // 3)
    x = (np.sin(np.arange(n) / 9.0) + 0.1 * rng.normal(size=n)) * (3.0 if kind != "positive" else 1.0)
    if kind == "positive":
        x = np.abs(x) + 0.0
    x = x.astype(dt)
    v = x.view(BITS[dt][0])
    sp = _specials(dt)
    for b in range(62):
        lo, hi = b * bs, min(n, (b + 1) * bs)
        if b % 8 == 7:
            continue   # left as it is
        at = {"first": lo, "last": hi - 1}.get(kind, int(rng.integers(lo, hi)))
        v[at] = sp[b % 6]
        if b % 2:
            v[int(rng.integers(lo, hi))] = sp[int(rng.integers(0, 6))]
        if b % 9 == 4:
            v[lo:hi] = sp[b % 6]
        if b % 11 == 6:
            v[lo:hi:2] = sp[5]
            v[lo + 1:hi:2] = sp[4]
    return x


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["first", "last", "inside", "positive"])
def test_streams_of_special_blocks(dt, kind):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for the gpu tests")
    import szx_gb300 as szx
    from szx_gb300 import build
    build.build()
    for bs in (1, 15, 16, 17, 64, 100, 128, 200, 255):
        rng = np.random.default_rng(bs)
        x = _field(dt, bs, kind, rng)
        xt = torch.tensor(x.view(np.int32 if dt == np.float32 else np.int64), device="cuda").view(
            torch.float32 if dt == np.float32 else torch.float64)
        for mode in (1, 2, 3, 4):
            for eb in (1e-3, 0.3):
                codec = szx.DeviceCodec(mode, dt, x.size, bs)
                codec.compress(xt, szx.ABS, eb)
                want = O.fast_compress_args(mode, x, 0, eb, 0.0, bs)
                assert codec.stream_bytes().cpu().numpy().tobytes() == want, (bs, mode, eb)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_non_blocked_differences_that_overflow(dt):
    """fastMode 1: differences from the median that are infinite, and NaNs among them."""
    import szx_gb300 as szx
    from szx_gb300 import build
    build.build()
    rng = np.random.default_rng(2)
    top = float(np.finfo(dt).max)
    for n in (1, 17, 4097, 20_011):
        x = (rng.uniform(-1, 1, n) * top).astype(dt)
        for extra in ((), (np.nan,), (np.inf, np.nan)):
            y = x.copy()
            for v in extra:
                y[rng.integers(0, n, max(1, n // 50))] = v
            for rel in (1e-3, 1e-5):
                assert szx.fast_compress_args(1, y, szx.REL, 0.0, rel) == O.fast_compress_args(1, y, 1, 0.0, rel, 128), (n, extra)
