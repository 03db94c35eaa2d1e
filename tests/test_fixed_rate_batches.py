"""Fixed-rate selection over many fields: what a field gets does not depend on
how many others the batch holds, and the ratio reported is the coded stream's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def LR():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for the gpu tests")
    from szx_gb300 import build, learned
    build.build()
    return learned


def _fields(torch, count, lo, hi, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k in range(count):
        n = int(np.exp2(rng.uniform(lo, hi)))
        x = np.sin(np.arange(n) / rng.uniform(20, 400)) + 0.02 * rng.normal(size=n)
        if k % 4 == 1:
            x = np.repeat(rng.normal(size=n // 700 + 1), 700)[:n] + 1e-3 * rng.normal(size=n)
        if k % 7 == 3:
            x[rng.random(n) < 0.01] = rng.choice([np.nan, np.inf, -0.0])
        if k % 11 == 5:
            x[:] = 2.5   # every bound gives the same ratio
        out.append(torch.tensor(x.astype(np.float32), device="cuda"))
    return out


def _zero_network(LR):
    n = LR.Mlp(0).count
    return LR.Mlp(0, params=np.concatenate([np.zeros(32), np.ones(32), np.zeros(n - 64)]).astype(np.float32))


@pytest.mark.parametrize("network", [False, True])
def test_a_field_gets_the_same_in_any_batch(LR, network):
    """1500 fields in one plan, whose passes measure few or no bounds ahead, against plans of 30 of them."""
    import torch
    xs = _fields(torch, 1500, 7, 13, 3)
    net = _zero_network(LR) if network else None
    b = LR.Batch(xs)
    eb, cr, ps = b.fixed_rate(12.0, net, 0.05, 14)
    sizes = b.sizes()
    b.close()
    assert ps.max() > 4   # some searches run on
    for a in range(0, len(xs), 30):
        c = LR.Batch(xs[a:a + 30])
        e2, c2, p2 = c.fixed_rate(12.0, net, 0.05, 14)
        assert np.array_equal(e2.view(np.uint32), eb[a:a + 30].view(np.uint32)), a
        assert np.array_equal(c2, cr[a:a + 30]) and np.array_equal(p2, ps[a:a + 30]), a
        assert np.array_equal(c.sizes(), sizes[a:a + 30]), a
        c.close()


@pytest.mark.parametrize("mode", [2, 3, 4])
def test_the_ratio_is_the_coded_streams(LR, mode):
    """Reached targets, missed ones and the pass limit: the ratio is the input's bytes over the stream's."""
    import torch
    xs = _fields(torch, 60, 0, 16, 5)
    b = LR.Batch(xs, fastMode=mode)
    for target, passes, net in ((8.0, 20, None), (8.0, 20, _zero_network(LR)), (3.0, 2, None), (1000.0, 6, None)):
        eb, cr, ps = b.fixed_rate(target, net, 0.02, passes)
        want = (b.n * 4.0 / b.sizes()).astype(np.float32)
        assert np.array_equal(cr, want), (target, passes)
    b.close()
