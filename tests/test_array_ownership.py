"""Decoded host arrays own the library's buffer: writable, valid after the
other handles are gone, and freed with the last view."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_decoded_array_outlives_everything_else():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for the gpu tests")
    import szx_gb300 as S
    from szx_gb300 import build
    build.build()
    for dt in (np.float32, np.float64):
        x = np.linspace(0, 1, 300_001).astype(dt)
        s = S.fast_compress_args(3, x, S.ABS, 1e-3)
        a = S.fast_decompress(3, dt, s, x.size)
        b = S.decompress_host(3, dt, s, x.size)
        assert type(a) is np.ndarray and a.dtype == dt and a.shape == x.shape and a.flags.writeable
        assert np.array_equal(a, b) and np.abs(a.astype(np.float64) - x).max() <= 1e-3 * (1 + 1e-6)
        v, keep = a[1000:2000], a[1000:2000].copy()
        a[0] = 7
        del a, b, s
        gc.collect()
        for _ in range(4):   # later calls do not reuse its memory
            S.fast_decompress(3, dt, S.fast_compress_args(3, x * 2, S.ABS, 1e-3), x.size)
        assert np.array_equal(v, keep)
