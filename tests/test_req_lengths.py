"""The reqLength byte of a stream: a fastMode-1 header whose reqLength is 0 or
above the type's bits describes no value and is refused."""
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


@pytest.mark.parametrize("dt,bits", [(np.float32, 32), (np.float64, 64)])
def test_non_blocked_header_refuses_what_describes_no_value(szx, dt, bits):
    x = np.random.default_rng(7).normal(size=70_001).astype(dt)
    s = szx.fast_compress_args(1, x, szx.ABS, 1e-3)
    for req in (0, bits + 1, bits + 8, bits + 9, 64 if bits == 32 else 72, 65, 255):
        bad = bytearray(s)
        bad[4] = req
        with pytest.raises(szx.SZxError):
            szx.fast_decompress(1, dt, bytes(bad), x.size)
    assert szx.fast_decompress(1, dt, s, x.size).tobytes() == O.decompress(1, dt, s, x.size).tobytes()
