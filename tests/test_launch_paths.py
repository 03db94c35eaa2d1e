"""Call paths whose launches depend on the size: the one-cluster value range
and the ticketed one, the one-CTA stream index and the persistent one, at and
around the sizes where they change over; and compress and decompress captured
in a CUDA graph and replayed on new values.  Streams and values equal the
oracle's."""
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


def field(dt, n, seed):
    rng = np.random.default_rng(seed)
    x = np.sin(np.arange(n) / 300.0) + 0.01 * rng.normal(size=n)
    for b in range(0, n - 300, 5000):
        x[b:b + 300] = 0.25
    x[n // 3] = -7.5
    return x.astype(dt)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [1, 2, 3, 4])
def test_sizes_around_the_changeovers(szx, dt, mode):
    import torch
    es = np.dtype(dt).itemsize
    for n, bs in (((2 << 20) // es, 128), ((2 << 20) // es + 1, 128), (16384 * 32, 32), (16384 * 32 + 1, 32),
                  (16384 * 4 - 3, 4), (16385 * 4, 4), (16384, 1), (16385, 1)):
        x = field(dt, n, n % 97)
        for off in (0, 1):
            codec = szx.DeviceCodec(mode, dt, n, bs)
            buf = torch.zeros(n + 1, dtype=torch.float32 if dt == np.float32 else torch.float64, device="cuda")
            buf[off:off + n] = torch.from_numpy(x).cuda()
            codec.ws.random_(0, 256)   # a workspace holds anything before a call
            codec.compress(buf[off:off + n], szx.REL, 0.0, 1e-3)
            s = codec.stream_bytes()
            want = O.fast_compress_args(mode, x, 1, 0.0, 1e-3, bs)
            assert s.cpu().numpy().tobytes() == want, (n, bs, off)
            codec.ws.random_(0, 256)
            y = codec.decompress(s, n)
            assert codec.status() == 0, (n, bs, off)
            z = O.decompress(mode, dt, want, n)
            assert np.array_equal(y.cpu().numpy().view(np.uint8), z.view(np.uint8)), (n, bs, off)


@pytest.mark.parametrize("mode", [1, 2, 3])
@pytest.mark.parametrize("n", [50_000, 3_000_001])
def test_captured_in_a_graph(szx, mode, n):
    import torch
    x = torch.from_numpy(field(np.float32, n, 1)).cuda()
    codec = szx.DeviceCodec(mode, np.float32, n)
    codec.compress(x, szx.REL, 0.0, 1e-3)
    s = codec.stream_bytes().clone()
    y = torch.empty(n, dtype=torch.float32, device="cuda")
    dec = szx.DeviceCodec(mode, np.float32, n)
    dec.decompress(s, n, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        codec.compress(x, szx.REL, 0.0, 1e-3)
        dec.decompress(s, n, y)
    for seed in (2, 3):
        v = field(np.float32, n, seed)
        x.copy_(torch.from_numpy(v))
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert codec.stream_bytes().cpu().numpy().tobytes() == O.fast_compress_args(mode, v, 1, 0.0, 1e-3, 128)
        z = O.decompress(mode, np.float32, s.cpu().numpy().tobytes(), n)
        assert dec.status() == 0 and np.array_equal(y.cpu().numpy().view(np.uint8), z.view(np.uint8))


@pytest.mark.parametrize("mode", [2, 3, 4])
@pytest.mark.parametrize("nb", [16385, 9 * 2048, 9 * 2048 + 1, 65536 + 7])
def test_index_at_every_byte_alignment(szx, mode, nb):
    """The persistent index over streams at any address: whole, partial and
    missing last tiles of either scan, no coded block, none but coded ones, and
    a coded few whose index ends right before the payloads."""
    import torch
    bs, n = 4, 4 * nb - 1
    rng = np.random.default_rng(nb)
    noise = rng.normal(size=n).astype(np.float32)
    some = np.where(np.repeat(rng.random(nb) < 0.3, bs)[:n], noise, np.float32(2.5))
    few = np.full(n, 1.5, np.float32)
    few[n - 9:] = noise[:9]
    for x in (noise, some, few, np.zeros(n, np.float32)):
        want = O.compress(mode, x, 1e-3, bs)
        z = O.decompress(mode, np.float32, want, n)
        for off in range(4):
            buf = torch.empty(off + len(want), dtype=torch.uint8, device="cuda")
            s = buf[off:]
            s.copy_(torch.frombuffer(bytearray(want), dtype=torch.uint8))
            codec = szx.DeviceCodec(mode, np.float32, n, bs)
            codec.ws.random_(0, 256)
            y = codec.decompress(s, n)
            assert codec.status() == 0
            assert np.array_equal(y.cpu().numpy().view(np.uint8), z.view(np.uint8)), off


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("skew", [8, 16])
def test_decode_workspace_at_any_word(szx, mode, skew):
    """A decompress workspace needs the alignment of its words, no more."""
    import torch
    for n in (300_000, 40_000 * 16 + 3):
        x = field(np.float32, n, 5)
        want = O.compress(mode, x, 1e-3, 16)
        codec = szx.DeviceCodec(mode, np.float32, n, 16)
        ws = torch.empty(codec.wsb + 64, dtype=torch.uint8, device="cuda").random_(0, 256)
        codec.ws = ws[skew:skew + codec.wsb]
        s = torch.frombuffer(bytearray(want), dtype=torch.uint8).cuda()
        y = codec.decompress(s, n)
        assert codec.status() == 0
        z = O.decompress(mode, np.float32, want, n)
        assert np.array_equal(y.cpu().numpy().view(np.uint8), z.view(np.uint8)), n


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_non_blocked_stream_at_every_byte_alignment(szx, dt):
    """Lead codes loaded as words around any address: fields of less than a
    word of codes, ends of every kind, whole and partial tiles and groups."""
    import torch
    for n in (1, 15, 17, 32, 33, 127, 4095, 4096 + 16, 8 * 4096, 9 * 4096 + 37):
        x = field(dt, max(n, 4), 11)[:n]
        want = O.compress(1, x, 1e-3, 128)
        z = O.decompress(1, dt, want, n)
        codec = szx.DeviceCodec(1, dt, n)
        for off in range(16):
            buf = torch.empty(off + len(want), dtype=torch.uint8, device="cuda")
            buf[off:].copy_(torch.frombuffer(bytearray(want), dtype=torch.uint8))
            y = codec.decompress(buf[off:], n)
            assert codec.status() == 0
            assert np.array_equal(y.cpu().numpy().view(np.uint8), z.view(np.uint8)), (n, off)
