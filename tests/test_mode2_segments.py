"""Decoding of streams without a size index at the edges of the boundary
search: payloads of one, a few and many segments (32 maximal blocks each),
block sizes whose lead bytes end inside a word or a byte, a short last block
that is coded or constant, blocks of the smallest and largest payload, and
streams at odd byte addresses.  Values equal the oracle's bit for bit."""
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


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("bs", [1, 2, 3, 5, 18, 37, 64, 100, 128, 255])
def test_decode_across_segments(szx, dt, bs):
    import torch
    rng = np.random.default_rng(bs)
    for nb, eb in ((1, 1e-3), (31, 1e-7), (33, 1e-2), (200, 1e-4), (1500, 1e-3)):
        for n in (nb * bs, nb * bs - bs // 2):
            if n < 1:
                continue
            x = np.cumsum(rng.normal(size=n)) * 0.1
            x[rng.random(n) < 0.01] *= 50                              # a few blocks with many required bytes
            for b in np.nonzero(rng.random(nb) < 0.2)[0]:
                x[b * bs:(b + 1) * bs] = x[b * bs] if b * bs < n else 0     # constant blocks, the last one among them
            x = x.astype(dt)
            s = O.compress(2, x, eb, bs)
            want = O.decompress(2, dt, s, n)
            codec = szx.DeviceCodec(2, dt, n, bs)
            off = int(rng.integers(0, 16))
            buf = torch.zeros(len(s) + 16, dtype=torch.uint8, device="cuda")
            buf[off:off + len(s)] = torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda()
            got = codec.decompress(buf[off:off + len(s)], n)
            assert codec.status() == 0, (nb, n, eb)
            assert np.array_equal(got.cpu().numpy().view(np.uint8), want.view(np.uint8)), (nb, n, eb)
