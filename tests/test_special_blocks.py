"""Special values in fastMode 1: differences from the median that are infinite,
and NaNs among them."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

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
