"""Performance cases of szx_gb300: the calls its users make, each with the data it meets in use.

A case is one field (or one batch of fields) with its codec options and one operation:

* ``compress`` / ``decompress`` -- ``DeviceCodec`` on a device tensor, as a simulation or a training job calls it on
  fields that are on the GPU already.  A compress leaves the stream and its place in device memory and waits for
  nothing; a decompress takes a stream whose length is known.
* ``roundtrip`` -- both in turn, as a checkpoint test or an in-memory cache does: the stream's length is read between.
* ``batch`` -- ``learned.Batch``: many fields of different sizes under one plan with their own absolute bounds.
* ``fixed_rate`` -- ``Batch.fixed_rate``: bounds that give every field of a batch a target ratio, with a trained
  network; the streams are then packed into one archive.
* ``host`` -- the reference's C interface on host arrays with a fixed-rate target, stream and values back on the host.

Sizes are the ones the repository's benchmark and tests name (512^3 float32, 1024 x 1024 x 256 float64, batches of
mixed sizes), and generic odd ones down to a few thousand values.

Streams have lengths of their own, so what a pass returns is the caller's buffer that holds them (zeroed once, before
the first pass) with their places.
"""
import numpy as np
import torch

import szx_gb300 as S
from szx_gb300 import learned

DT = {"float32": torch.float32, "float64": torch.float64}


# ------------------------------------------------------------------ cases

def listed():
    return [
        # a small variable of a checkpoint, or one slice of a field: launches and latency decide
        {"name": "small_f32_roundtrip", "op": "roundtrip", "mode": 3, "dtype": "float32", "n": 65536, "bs": 128,
         "err": "rel", "bound": 1e-3, "field": "spectral"},
        # a medium 2-D or 3-D variable of odd size with a block size of the caller's choice
        {"name": "ragged_f32_roundtrip", "op": "roundtrip", "mode": 3, "dtype": "float32", "n": 5000011, "bs": 100,
         "err": "rel", "bound": 1e-4, "field": "spectral"},
        # the benchmark's field: one large simulation variable, random-access layout
        {"name": "field_f32_compress", "op": "compress", "mode": 3, "dtype": "float32", "n": 512 ** 3, "bs": 128,
         "err": "rel", "bound": 1e-3, "field": "spectral"},
        {"name": "field_f32_decompress", "op": "decompress", "mode": 3, "dtype": "float32", "n": 512 ** 3, "bs": 128,
         "err": "rel", "bound": 1e-3, "field": "spectral"},
        # the non-blocked layout on the same field
        {"name": "chain_f32_compress", "op": "compress", "mode": 1, "dtype": "float32", "n": 512 ** 3, "bs": 128,
         "err": "rel", "bound": 1e-3, "field": "spectral"},
        {"name": "chain_f32_decompress", "op": "decompress", "mode": 1, "dtype": "float32", "n": 512 ** 3, "bs": 128,
         "err": "rel", "bound": 1e-3, "field": "spectral"},
        # a large double-precision field with a trend and outliers, absolute bounds, both ends of the block sizes used
        {"name": "field_f64_compress", "op": "compress", "mode": 3, "dtype": "float64", "n": 1 << 28, "bs": 64,
         "err": "abs", "bound": 1e-1, "field": "trend"},
        {"name": "field_f64_decompress", "op": "decompress", "mode": 3, "dtype": "float64", "n": 1 << 28, "bs": 256,
         "err": "abs", "bound": 1e-3, "field": "trend"},
        # reading back a stream without a size index (what fixed-rate compression writes)
        {"name": "noindex_f32_decompress", "op": "decompress", "mode": 2, "dtype": "float32", "n": 1 << 26, "bs": 128,
         "err": "rel", "bound": 1e-3, "field": "spectral"},
        # all variables of a time step at once: many sizes, three kinds of data, a bound each
        {"name": "batch_f32_compress", "op": "batch", "fields": 48, "lo": 14, "hi": 24, "sizes": 11, "mode": 3, "bs": 128},
        # the same with a target ratio instead of bounds
        {"name": "batch_fixed_rate", "op": "fixed_rate", "fields": 24, "lo": 18, "hi": 23, "sizes": 7, "ratio": 16.0},
        # the reference's interface on host arrays, fixed rate, one field
        {"name": "host_fixed_rate", "op": "host", "dtype": "float32", "n": 1 << 22, "ratio": 10.0, "tolerance": 0.1,
         "field": "spectral"},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    op = rng.choice(["compress", "compress", "decompress", "decompress", "roundtrip", "roundtrip", "batch",
                     "fixed_rate", "host"])
    if op == "batch":
        return {"op": op, "fields": rng.randint(4, 60), "lo": 14, "hi": rng.randint(18, 24), "sizes": rng.randint(1, 10 ** 6),
                "mode": rng.choice([2, 3]), "bs": rng.choice([64, 128, 128, 224])}
    if op == "fixed_rate":
        return {"op": op, "fields": rng.randint(4, 24), "lo": 18, "hi": rng.randint(19, 23), "sizes": rng.randint(1, 10 ** 6),
                "ratio": rng.choice([8.0, 16.0, 32.0])}
    if op == "host":
        return {"op": op, "dtype": rng.choice(["float32", "float64"]), "n": int(_log(rng, 1 << 16, 1 << 22)),
                "ratio": rng.choice([6.0, 10.0, 20.0]), "tolerance": 0.1, "field": rng.choice(["spectral", "sinusoid"])}
    dtype = rng.choice(["float32", "float32", "float64"])
    n = int(_log(rng, 4096, (1 << 20) if op == "roundtrip" else (1 << 27)))
    mode = rng.choice([3, 3, 3, 1, 1, 2, 4])
    return {"op": op, "mode": mode, "dtype": dtype, "n": n, "bs": rng.choice([32, 64, 100, 128, 128, 128, 200, 248]),
            "err": "rel", "bound": _log(rng, 1e-5, 1e-2),
            "field": rng.choice(["spectral", "sinusoid", "levels"] + (["trend"] if dtype == "float64" else []))}


# ------------------------------------------------------------------ data

def _spectral(n, g, dtype):
    """The first n values of a periodic cube with an isotropic k^-5/3 spectrum, zero mean and unit variance, one plane
    in twenty zero (land, vacuum)."""
    side = max(16, -(-int(round(n ** (1 / 3) + 0.499)) // 16) * 16)
    while side ** 3 < n:
        side += 16
    f = torch.fft.rfftn(torch.randn((side,) * 3, generator=g, device="cuda", dtype=dtype))
    k = torch.fft.fftfreq(side, device="cuda", dtype=dtype)
    kr = torch.fft.rfftfreq(side, device="cuda", dtype=dtype)
    for z in range(0, side, 64):   # in slabs: the amplitudes never exist whole
        k2 = k[z:z + 64, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2
        f[z:z + 64] *= torch.where(k2 > 0, k2.clamp_min(1e-12) ** (-5.0 / 12.0), torch.zeros_like(k2))
    x = torch.fft.irfftn(f, s=(side,) * 3)
    del f
    x /= x.std()
    x[torch.rand(side, generator=g, device="cuda") < 0.05] = 0
    return x.reshape(-1)[:n].clone()


def _field(kind, n, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "spectral":
        return _spectral(n, g, dtype)
    if kind == "trend":   # pressure-like: large values, a linear trend, one value in a hundred an outlier
        x = _spectral(n, g, dtype)
        x = x.mul_(1e6).add_(torch.linspace(-3e5, 3e5, n, device="cuda", dtype=dtype))
        for a in range(0, n, 1 << 26):
            b = min(n, a + (1 << 26))
            out = torch.rand(b - a, generator=g, device="cuda") < 0.01
            x[a:b] = torch.where(out, torch.randn(b - a, generator=g, device="cuda", dtype=dtype) * 1e8, x[a:b])
        return x
    if kind == "sinusoid":   # eight sinusoids with noise, one block of 128 in ten constant
        t = torch.arange(n, device="cuda", dtype=torch.float64) * (2 * np.pi / n)
        x = torch.zeros(n, device="cuda", dtype=torch.float64)
        for _ in range(8):
            w, a = torch.rand(2, generator=g, device="cuda", dtype=torch.float64).tolist()
            x += (0.1 + 0.9 * a) * torch.sin((1 + int(63 * w)) * t)
        x = (x + 1e-3 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)).to(dtype)
        blocks = x[: n // 128 * 128].view(-1, 128)
        flat = torch.rand(blocks.shape[0], generator=g, device="cuda") < 0.1
        blocks.copy_(torch.where(flat[:, None], blocks[:, :1].clone(), blocks))
        return x
    if kind == "levels":   # piecewise constant with a little noise
        run = 64 + int(torch.randint(0, 4000, (1,), generator=g, device="cuda").item())
        lv = torch.randn(n // run + 1, generator=g, device="cuda", dtype=dtype)
        return torch.repeat_interleave(lv, run)[:n] + 1e-3 * torch.randn(n, generator=g, device="cuda", dtype=dtype)
    return torch.randn(n, generator=g, device="cuda", dtype=dtype)   # "noise"


def _sizes(case):
    """Sizes of a batch's fields: log-uniform, fixed by the case (only the values change with the seed)."""
    r = np.random.default_rng(case["sizes"])
    return np.exp2(r.uniform(case["lo"], case["hi"], case["fields"])).astype(np.int64).tolist()


def _kind_of(k):
    return ("spectral", "levels", "noise")[k % 3]


def _batch_fields(case, seed):
    return [_field(_kind_of(k), n, seed * 1000 + k, torch.float32) for k, n in enumerate(_sizes(case))]


def _stored(case):
    """Stream bytes per value, near enough for a traffic count (measured within a fifth on the listed cases): bits
    from the sign to the bound at the spread of a block, a lead code, less what a value shares with the one before."""
    w = 4 if case["dtype"] == "float32" else 8
    if case["field"] == "trend":
        return 0.25 + (10 + np.log2(1e6 / (case["bound"] if case["err"] == "abs" else 1e9 * case["bound"]))) / 8
    if case["field"] == "spectral":
        return float(min(w, 0.45 + (10 + np.log2(0.1 / case["bound"])) / 8))
    noise = 6e-3 / (8 * case["bound"])   # spread of a block of these two kinds, in bounds
    least = 0.1 if case["field"] == "levels" else 0.7
    return float(max(least, 0.1 + (10 + np.log2(noise)) / 8 if noise >= 2 else 0))


def work(case):
    """Each input read once and each output written once; the operations are integer work and not counted."""
    op = case["op"]
    if op == "batch":
        return {"bytes": sum(_sizes(case)) * (4 + 2.0), "flops": 0}
    if op == "fixed_rate":
        return {"bytes": sum(_sizes(case)) * 4 * (1 + 1 / case["ratio"]), "flops": 0}
    w = 4 if case["dtype"] == "float32" else 8
    if op == "host":
        return {"bytes": 2 * case["n"] * w * (1 + 1 / case["ratio"]), "flops": 0}
    return {"bytes": case["n"] * (w + _stored(case)) * (2 if op == "roundtrip" else 1), "flops": 0}


# ------------------------------------------------------------------ a pass

def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        xs = _batch_fields(case, seed)
        bounds = [float((x.max() - x.min()).item()) * 10 ** (-2 - 3 * ((7 * k) % 10) / 10) for k, x in enumerate(xs)]
        b = learned.Batch(xs, bounds, fastMode=case["mode"], blockSize=case["bs"])
        for o in b.outs:
            o.zero_()
        return {"case": case, "batch": b}
    if op == "fixed_rate":
        # the network a user would have trained before, on smaller fields of the same kinds
        small = learned.Batch([_field(_kind_of(k), 20000 + 9000 * k, 77 + k, torch.float32) for k in range(12)])
        X, y, _ = learned.training_set(small, passes=6, seed=1)
        mlp, _ = learned.train(X, y, seed=1, epochs=20, batch=64)
        small.close()
        b = learned.Batch(_batch_fields(case, seed))
        return {"case": case, "batch": b, "mlp": mlp, "archive": torch.zeros(5 * int(b.n.sum()), dtype=torch.uint8,
                                                                            device="cuda")}
    x = _field(case["field"], case["n"], seed, DT[case["dtype"]])
    if op == "host":
        return {"case": case, "x": x.cpu().numpy(), "file": np.zeros(2 * x.numel() * x.element_size(), np.uint8)}
    dt = np.dtype(case["dtype"])
    codec = S.DeviceCodec(case["mode"], dt, case["n"], case["bs"])
    codec.out.zero_()
    state = {"case": case, "x": x, "codec": codec, "out": torch.empty_like(x)}
    if op == "decompress":
        _compress(state)
        state["stream"] = codec.stream_bytes().clone()
        del state["x"]
    return state


def _compress(state):
    case, codec = state["case"], state["codec"]
    if case["err"] == "rel":
        codec.compress(state["x"], S.REL, 0.0, case["bound"])
    else:
        codec.compress(state["x"], S.ABS, case["bound"])


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "batch":
        b = state["batch"]
        b.run()
        return b.outs + [b.info]
    if op == "fixed_rate":
        b = state["batch"]
        eb, ratio, passes = b.fixed_rate(case["ratio"], state["mlp"])
        infos = b.infos()
        size = [int(i.size) for i in infos]
        torch.cat([o[i.offset:i.offset + i.size] for o, i in zip(b.outs, infos)], out=state["archive"][:sum(size)])
        return [eb, ratio, passes, np.array(size), state["archive"]]
    if op == "host":
        s = S.fast_compress_args(S.WITH_BLOCK, state["x"], S.FXR, compressionRatio=case["ratio"],
                                 tolerance=case["tolerance"])
        state["file"][:len(s)] = np.frombuffer(s, np.uint8)
        return [len(s), state["file"], S.fast_decompress(S.WITH_BLOCK, state["x"].dtype, s, case["n"])]
    codec = state["codec"]
    if op == "decompress":
        return codec.decompress(state["stream"], case["n"], state["out"])
    _compress(state)
    if op == "compress":
        return [codec.out, codec.info]
    return [codec.out, codec.info, codec.decompress(codec.stream_bytes(), case["n"], state["out"])]


def exact(case, seed):
    """A stream is bytes and has no such value; decoded values stand for the field itself, in 64 bits."""
    op = case["op"]
    if op in ("compress", "batch", "fixed_rate"):
        return None
    x = _field(case["field"], case["n"], seed, DT[case["dtype"]]).double()
    return x if op == "decompress" else [None, None, x.cpu().numpy() if op == "host" else x]
