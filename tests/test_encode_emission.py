"""Blocked encoder at the edges of its payload emission and of its double
arithmetic: lanes whose values store no byte or a single one, whole words that
several lanes share, blocks shorter than a lane's run, inputs at every element
alignment, tiles that end in the middle of a block, and doubles whose
statistics meet subnormals, ties of the rounding to float and the ends of the
exponent range.  Streams equal the oracle's byte for byte."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def szx():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for the gpu tests")
    import szx_gb300
    from szx_gb300 import build
    build.build()
    return szx_gb300


def fields(dt, n):
    rng = np.random.default_rng(7)
    yield "held", np.repeat(rng.normal(size=n // 5 + 1), 5)[:n].astype(dt), 1e-3          # most values store nothing
    yield "spikes", np.where(rng.random(n) < 0.03, rng.normal(size=n) * 1e3, 1.0).astype(dt), 1e-2
    yield "smooth", (1 + 1e-3 * np.sin(np.arange(n) / 9)).astype(dt), 1e-6
    yield "rough", rng.normal(size=n).astype(dt), 1e-7
    u = np.dtype("u4" if dt == np.float32 else "u8")
    bits = rng.integers(0, np.iinfo(u).max, n, dtype=u, endpoint=True)
    yield "patterns", np.where(np.isfinite(bits.view(dt)), bits.view(dt), dt(0)), 1e-2   # every exponent
    tiny = (rng.integers(-9, 9, n) * np.finfo(dt).smallest_subnormal).astype(dt)
    yield "subnormal", tiny, 1e-44
    if dt == np.float64:
        m = rng.integers(1, 1 << 24, n).astype(np.float64)
        yield "ties", m + 0.5 * (rng.random(n) < 0.5) + rng.choice([0.0, 2.0 ** -29, -(2.0 ** -29)], n), 1.0
        yield "edges", np.exp2(rng.choice([-1074, -1022, -1021, -150, -149, -127, -126, 126, 127, 128, 1023], n)), 1e30


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("bs", [1, 7, 16, 33, 64, 100, 128, 250])
def test_streams_at_emission_edges(szx, dt, bs):
    import torch
    tile = 32 * bs
    for n in (bs, tile - 1, 3 * tile + 2 * bs + 3):
        codec = {m: szx.DeviceCodec(m, dt, n + 4, bs) for m in (2, 3, 4)}
        for name, x, eb in fields(dt, n):
            for off in range(4):
                buf = torch.zeros(n + 4, dtype=torch.float32 if dt == np.float32 else torch.float64, device="cuda")
                buf[off:off + n] = torch.from_numpy(x).cuda()
                for mode, c in codec.items():
                    c.compress(buf[off:off + n], szx.ABS, eb)
                    got = c.stream_bytes().cpu().numpy().tobytes()
                    assert got == O.compress(mode, x, eb, bs), (name, n, off, mode)
                    if off == 0:
                        break   # the other layouts share the encoder: one of them suffices there


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4097, 5 * 4096 + 37])
def test_non_blocked_streams_at_emission_edges(szx, dt, n):
    """The one-chain layout: runs that share words across lanes and warps, a
    last thread with 1..16 values, NaNs beside the run's start."""
    import torch
    codec = szx.DeviceCodec(1, dt, n + 4)
    cases = list(fields(dt, n))
    x = np.random.default_rng(3).normal(size=n).astype(dt)
    x[n // 2::511] = np.nan
    cases.append(("nan", x, 1e-3))
    for name, x, eb in cases:
        for off in (0, 1):
            buf = torch.zeros(n + 4, dtype=torch.float32 if dt == np.float32 else torch.float64, device="cuda")
            buf[off:off + n] = torch.from_numpy(x).cuda()
            codec.compress(buf[off:off + n], szx.ABS, eb)
            assert codec.stream_bytes().cpu().numpy().tobytes() == O.compress(1, x, eb, 128), (name, off)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("tiles", [2, 3, 700, 4 * 608])
def test_non_blocked_placement(szx, dt, tiles):
    """Tiles placed from the CTA's previous one: fewer tiles than CTAs, each CTA
    with one to several, a window beyond the counts' end, byte counts of tiles
    from nothing stored to every byte."""
    n = tiles * 4096 - 5
    rng = np.random.default_rng(5)
    x = rng.normal(size=n).astype(dt)
    for t in rng.choice(tiles, tiles // 2, replace=False):
        x[t * 4096:(t + 1) * 4096] = 0.25
    import torch
    codec = szx.DeviceCodec(1, dt, n)
    codec.compress(torch.from_numpy(x).cuda(), szx.ABS, 1e-12)
    assert codec.stream_bytes().cpu().numpy().tobytes() == O.compress(1, x, 1e-12, 128)
