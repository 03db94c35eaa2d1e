"""The value range of a field by one cluster and by the whole grid, around the
size where they change over (512 KiB): streams equal the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("mode", [1, 3])
def test_sizes_around_the_changeover(dt, mode):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for the gpu tests")
    import szx_gb300 as szx
    from szx_gb300 import build
    build.build()
    edge = (512 << 10) // np.dtype(dt).itemsize
    for n in (edge - 1, edge, edge + 1, edge + 7):
        for at in (0, n // 2, n - 1):
            rng = np.random.default_rng(n % 89 + at)
            x = np.sin(np.arange(n) / 300.0) + 0.01 * rng.normal(size=n)
            x[at] = -9.25          # the extreme at either end and inside
            x[n - 1 - at] = 8.5
            x = x.astype(dt)
            codec = szx.DeviceCodec(mode, dt, n, 128)
            codec.ws.random_(0, 256)   # a workspace holds anything before a call
            codec.compress(torch.from_numpy(x).cuda(), szx.REL, 0.0, 1e-3)
            assert codec.stream_bytes().cpu().numpy().tobytes() == O.fast_compress_args(mode, x, 1, 0.0, 1e-3, 128), (n, at)
