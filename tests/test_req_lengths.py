"""The reqLength byte of a stream, over its whole range.

A value stores the top ceil(reqLength / 8) bytes less its leading code, so a
stream may ask for one byte a value although this library's encoders never ask
for less than two (floats 9, doubles 12 bits).  A fastMode-1 header whose
reqLength is 0 or above the type's bits describes no value and is refused."""
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


def _codes(lead):
    """2-bit leading codes, four to a byte, the first on top."""
    c = np.zeros((len(lead) + 3) // 4 * 4, np.uint8)
    c[:len(lead)] = lead
    return (c[0::4] << 6 | c[1::4] << 4 | c[2::4] << 2 | c[3::4]).tobytes()


def _stored(rng, req, lead):
    """Random stored bytes of values with these leading codes."""
    return rng.integers(0, 256, int(np.maximum((req + 7) // 8 - lead, 0).sum()), dtype=np.uint8).tobytes()


def _be32(median):
    return np.array(median, ">f4").tobytes()


def _random_access(rng, mode, n, bs, reqs, lead_p):
    """A fastMode 3/4 stream of random blocks with these reqLengths, one block in five constant."""
    nb = (n + bs - 1) // bs
    coded = rng.random(nb) >= 0.2
    sizes, medians, payloads = [], [], []
    for b in range(nb):
        m = rng.normal()
        if not coded[b]:
            medians.append(np.array(m, ">f4" if mode == 3 else "<f4").tobytes())
            continue
        req, k = int(rng.choice(reqs)), min(bs, n - b * bs)
        lead = rng.choice(4, k, p=lead_p)
        payloads.append(bytes([req]) + _be32(m) + _codes(lead) + _stored(rng, req, lead))
        sizes.append(len(payloads[-1]))
    state = np.packbits(coded).tobytes()
    return (bytes([1, 1, 1, 1]) + bs.to_bytes(8, "big") + int((~coded).sum()).to_bytes(8, "big")
            + np.array(sizes, "<u2").tobytes() + state + b"".join(medians) + b"".join(payloads))


def _same(a, b):
    return np.array_equal(a.view(np.uint8), b.view(np.uint8))


LEADS = ([0.25, 0.25, 0.25, 0.25], [0.02, 0.03, 0.05, 0.9])


@pytest.mark.parametrize("dt,bits", [(np.float32, 32), (np.float64, 64)])
@pytest.mark.parametrize("mode", [3, 4])
def test_blocks_of_every_req_length(szx, dt, bits, mode):
    """Blocks of 1..bits required bits, side by side and with one byte a value throughout, decode as the format says."""
    import torch
    rng = np.random.default_rng(23 + mode)
    for bs in (1, 5, 16, 31, 100, 128, 256):
        n = 301 * bs - (bs > 1)
        for reqs in (np.arange(1, bits + 1), np.arange(1, 9), np.arange(1, 17)):
            for p in LEADS:
                s = _random_access(rng, mode, n, bs, reqs, p)
                codec = szx.DeviceCodec(mode, dt, n, bs)
                y = codec.decompress(torch.tensor(np.frombuffer(s, np.uint8).copy(), device="cuda"), n)
                assert codec.status() == 0, (bs, reqs[-1])
                assert _same(y.cpu().numpy(), O.decompress(mode, dt, s, n)), (bs, reqs[-1], p)


@pytest.mark.parametrize("dt,bits", [(np.float32, 32), (np.float64, 64)])
def test_non_blocked_streams_of_every_req_length(szx, dt, bits):
    """The same for fastMode 1: several tiles, the last one ragged, and leads that carry bytes over many values."""
    rng = np.random.default_rng(29)
    for req in range(1, bits + 1):
        for n in ((40_003,) if req > 17 else (1, 17, 4096, 4097, 40_003)):
            for p in LEADS + ([0.0005, 0.0005, 0.0005, 0.9985],):
                lead = rng.choice(4, n, p=p)
                s = (bytes([1, 1, 1, 0, req]) + _be32(rng.normal()) + ((n + 3) // 4).to_bytes(8, "big") + _codes(lead)
                     + _stored(rng, req, lead))
                assert _same(szx.fast_decompress(1, dt, s, n), O.decompress(1, dt, s, n)), (req, n, p)
