"""fastMode-2 streams of small blocks: a segment's walk by one warp or by eight
(payloads of up to 160 bytes and above), with few candidates, many false ones
and several segments.  Values equal the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _field(kind, n, dt, rng):
    if kind == "smooth":
        x = np.sin(np.arange(n) / 30.0) + 0.01 * rng.normal(size=n)
    elif kind == "noise":
        x = rng.normal(size=n)
    else:   # periodic: walks from false starts survive
        x = np.tile(rng.normal(size=37), n // 37 + 1)[:n]
    x[n // 4:n // 4 + n // 9] = 0.5   # constant blocks
    return x.astype(dt)


# largest payloads of 10, 14, 18, 27, 39, 73, 154, 158 | 163, 248 bytes (float32) and 14, 22, 38, 71, 154 | 162, 302
@pytest.mark.parametrize("dt,sizes", [(np.float32, (1, 2, 3, 5, 8, 16, 35, 36, 37, 57)),
                                      (np.float64, (1, 2, 4, 8, 18, 19, 36))])
@pytest.mark.parametrize("kind", ["smooth", "noise", "periodic"])
def test_small_blocks(dt, sizes, kind):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for the gpu tests")
    import szx_gb300 as szx
    from szx_gb300 import build
    build.build()
    for bs in sizes:
        for n in (1, bs, 32 * bs + 1, 1000 * bs + bs // 2 + 1, 40_003):
            rng = np.random.default_rng(bs + n)
            x = _field(kind, n, dt, rng) if n > 40 else rng.normal(size=n).astype(dt)
            codec = szx.DeviceCodec(2, dt, n, bs)
            codec.compress(torch.from_numpy(x).cuda(), szx.ABS, 1e-3)
            s = codec.stream_bytes()
            want = O.fast_compress_args(2, x, 0, 1e-3, 0.0, bs)
            assert s.cpu().numpy().tobytes() == want, (bs, n)
            codec.ws.random_(0, 256)
            y = codec.decompress(s.clone(), n)
            assert codec.status() == 0, (bs, n)
            assert np.array_equal(y.cpu().numpy().view(np.uint8), O.decompress(2, dt, want, n).view(np.uint8)), (bs, n)
