"""The work that users have this codec do, as measurable cases.

``listed`` names the cases, ``draw`` gives more of the same ranges, ``prepare``
makes what a caller has in hand (fields in HBM, or in host memory for the host
API, output buffers, streams to decompress, batch plans), ``run`` is one pass
through the public entry points (a stream comes back as its size and the
caller's whole buffer, which is zero past it), ``work`` the bytes a pass cannot do without and
``exact`` the decompressed values from 64-bit arithmetic.

A case's keys: ``kind`` (compress, decompress, roundtrip, pipeline, reduce,
lorenzo, batch, host), ``field`` (walk, fourier, laplace), ``n`` values (or
``nx``, ``ny``, ``nz``), ``dtype`` (f32, f64), ``mode`` (rel, abs) with its ``bound`` (a
fraction of the value range, except laplace's absolute bound), ``block``,
``segments`` and ``fastmode``.
"""
import ctypes
import math

import numpy as np
import torch

import szp_gb300 as szp

_BASE = {"kind": "roundtrip", "field": "walk", "n": 0, "dtype": "f32", "mode": "rel", "bound": 1e-3,
         "block": 32, "segments": 16, "fastmode": 1}


def _case(name=None, **kw):
    c = dict(_BASE, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small field per call (the smallest size of the batched and served
        # requests): launches and latency count
        _case("small_roundtrip", n=4099),
        # the median field of the batched and served requests, 1 MB, one call
        # each way
        _case("median_roundtrip", n=262_147, bound=1e-4),
        # the reference's own calls on a field in ordinary host memory: into a
        # buffer of the caller's, and back
        _case("host_roundtrip", kind="host", field="fourier", n=256 ** 3, mode="abs"),
        # the benchmark's field, compressed with a relative bound: the largest call
        _case("field_compress", kind="compress", field="fourier", n=512 ** 3),
        # and decompressed
        _case("field_decompress", kind="decompress", field="fourier", n=512 ** 3),
        # compress and decompress queued without waiting for the size, a 1-D
        # series at a tight absolute bound
        _case("walk_pipeline", kind="pipeline", n=1 << 24, mode="abs", bound=1e-4),
        # a large 2-D field with 40% empty blocks, many segments (a 72-core host)
        _case("zero_blocks_pipeline", kind="pipeline", field="laplace", n=8192 * 8192, mode="abs", bound=1e-5,
              segments=72),
        # fastmode2 (random access) with longer blocks
        _case("fastmode2_roundtrip", field="fourier", n=384 ** 3, bound=1e-4, block=64, fastmode=2),
        # float64 data, an odd length
        _case("float64_roundtrip", field="fourier", n=(1 << 25) + 1, dtype="f64", bound=1e-6),
        # the homomorphic sum of two compressed fields (a step of a collective)
        _case("reduce_sum", kind="reduce", field="fourier", n=384 ** 3, mode="abs"),
        # the multidimensional Lorenzo variant
        _case("lorenzo_roundtrip", kind="lorenzo", field="fourier", n=500 * 384 * 256, nx=500, ny=384, nz=256),
        # many fields of uneven sizes and bounds, one launch sequence each way
        _case("batch_roundtrip", kind="batch", field="mixed", n=256, layout=11),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["compress", "decompress", "roundtrip", "roundtrip", "pipeline", "pipeline", "reduce", "lorenzo",
                       "batch", "host"])
    segments = rng.choice([1, 7, 16, 16, 16, 72, 144])
    rel = 10.0 ** rng.uniform(-5, -2)
    if kind == "batch":
        return _case(kind="batch", field="mixed", n=_log_uniform(rng, 8, 250), layout=rng.randrange(1 << 20),
                     segments=rng.choice([7, 16, 16]))
    if kind == "lorenzo":
        nx, ny, nz = _log_uniform(rng, 20, 600), _log_uniform(rng, 10, 400), _log_uniform(rng, 1, 200)
        return _case(kind="lorenzo", field="fourier", n=nx * ny * nz, nx=nx, ny=ny, nz=nz, bound=rel,
                     mode=rng.choice(["rel", "abs"]), segments=segments)
    field = rng.choice(["walk", "fourier", "fourier", "laplace"])
    mode, bound = rng.choice([("rel", rel), ("abs", rel)])
    if kind == "host":
        mode = "abs"
    if field == "laplace":
        mode, bound = "abs", 10.0 ** rng.uniform(-5.5, -3.5)
    dtype = rng.choice(["f32", "f32", "f32", "f64"]) if kind in ("compress", "decompress", "roundtrip") else "f32"
    block = rng.choice([32, 32, 32, 32, 32, 16, 64, 128, 48])
    fastmode = rng.choice([1, 1, 1, 2])
    most = {"compress": 1 << 27, "decompress": 1 << 27, "reduce": 50_000_000, "host": 1 << 24}.get(kind, 1 << 26)
    if dtype == "f64":
        most //= 2
    if block == 48:
        block = block if kind != "reduce" else 64
        most = min(most, 1 << 23)
    return _case(kind=kind, field=field, n=_log_uniform(rng, 4096, most), dtype=dtype, mode=mode, bound=bound,
                 block=block, segments=segments, fastmode=fastmode)


# ---------------------------------------------------------------- fields ---

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _walk(n, seed):
    """Gaussian steps (sigma 0.01) plus a slow sine; the sum runs on integers so
    that a seed always gives the same values."""
    steps = (torch.randn(n, generator=_generator(seed), device="cuda") * (0.01 * 2 ** 30)).to(torch.int64)
    v = torch.cumsum(steps, 0).to(torch.float64) * 2.0 ** -30
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    return v + torch.sin(i * (2 * math.pi / 4096.0))


def _fourier(nx, ny, nz, seed, dtype):
    """16 random Fourier modes (|k| 1..32, amplitude |k|^-5/3) plus N(0, 1e-3) noise."""
    rng = np.random.default_rng(int(seed))
    f = torch.zeros((nz, ny, nx), device="cuda", dtype=dtype)
    axes = [torch.arange(m, device="cuda", dtype=torch.float32) * (2 * math.pi / m) for m in (nx, ny, nz)]
    modes = 0
    while modes < 16:
        k = rng.integers(-32, 33, size=3)
        norm = float(np.sqrt((k * k).sum()))
        if not 1.0 <= norm <= 32.0:
            continue
        modes += 1
        arg = ((float(k[0]) * axes[0]).view(1, 1, nx) + (float(k[1]) * axes[1]).view(1, ny, 1) +
               (float(k[2]) * axes[2] + float(rng.uniform(0, 2 * math.pi))).view(nz, 1, 1))
        f += torch.sin(arg).mul_(norm ** (-5.0 / 3.0))
    f += torch.randn(f.shape, generator=_generator(seed + 1), device="cuda", dtype=dtype).mul_(1e-3)
    return f.reshape(-1)


def _laplace(n, seed):
    """A 2-D Laplace(0, 1e-3) field with rectangular patches of zeros over 40% of it."""
    side = max(1, math.isqrt(n - 1) + 1)
    g = _generator(seed)
    u = torch.rand(side * side, generator=g, device="cuda") - 0.5
    f = (-1e-3 * torch.sign(u) * torch.log1p(-2.0 * u.abs().clamp(max=0.4999999))).view(side, side)
    rng = np.random.default_rng(int(seed))
    zero = np.zeros((64, 64), dtype=bool)  # coverage on a coarse grid
    while zero.mean() < 0.42:
        h, w = int(rng.integers(2, 17)), int(rng.integers(8, 33))
        y, x = int(rng.integers(0, 65 - h)), int(rng.integers(0, 65 - w))
        zero[y:y + h, x:x + w] = True
        cut = [side * v // 64 for v in (y, y + h, x, x + w)]
        f[cut[0]:cut[1], cut[2]:cut[3]] = 0.0
    return f.reshape(-1)[:n].clone()


def _field(case, seed):
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    n = case["n"]
    if case["field"] == "walk":
        return _walk(n, seed).to(dtype)
    if case["field"] == "laplace":
        return _laplace(n, seed).to(dtype)
    if "nx" in case:
        return _fourier(case["nx"], case["ny"], case["nz"], seed, dtype)
    side = 1
    while side ** 3 < n:
        side += 1
    nz = -(-n // (side * side))
    f = _fourier(side, side, nz, seed, dtype)
    return f if f.numel() == n else f[:n].clone()


def _bound(case, x):
    """(errBoundMode, absErrBound, relBoundRatio) of a call on x."""
    if case["mode"] == "rel":
        return szp.REL, 0.0, case["bound"]
    if case["field"] == "laplace":
        return szp.ABS, case["bound"], 0.0
    return szp.ABS, case["bound"] * max(float(x.max() - x.min()), 1e-6), 0.0


def _stream():
    return torch.cuda.current_stream().cuda_stream


# --------------------------------------------------------------- batches ---

def _layout(case):
    """Sizes (log-normal, 4 KB to 64 MB, median 1 MB), bounds and slab offsets of a batch's fields."""
    rng = np.random.default_rng(case["layout"])
    size = np.clip(np.exp(rng.normal(math.log(1 << 18), 1.4, case["n"])), 1024, 1 << 24).astype(np.int64)
    rels = 10.0 ** rng.uniform(-5, -2, case["n"])
    kinds = rng.integers(0, 2, case["n"])
    at = np.concatenate([[0], np.cumsum((size + 127) // 128 * 128)])
    return [int(v) for v in size], [float(v) for v in rels], [int(v) for v in kinds], [int(v) for v in at]


def _batch_fields(case, seed):
    size, _, kinds, at = _layout(case)
    x = _walk(at[-1], seed).to(torch.float32)
    base = _fourier(256, 256, 256, seed + 2, torch.float32)
    rng = np.random.default_rng(int(seed))
    for n, k, o in zip(size, kinds, at):
        if k:
            b = int(rng.integers(0, base.numel() - n + 1))
            x[o:o + n] = base[b:b + n]
    return x


# --------------------------------------------------------------- prepare ---

def prepare(case, seed):
    s = dict(case)
    if case["kind"] == "batch":
        return _prepare_batch(s, seed)
    x = _field(case, seed)
    n, block, T, fm = case["n"], case["block"], case["segments"], case["fastmode"]
    s["bounds"] = _bound(case, x)
    if case["kind"] == "host":
        szp.set_segments(T)
        s["x"] = x.cpu().numpy()
        s["out"] = np.zeros(4 + 4 * n, dtype=np.uint8)
        return s
    f64 = case["dtype"] == "f64"
    if case["kind"] == "lorenzo":
        s["dims"] = (case["nz"], case["ny"], case["nx"])
        cap = szp.lorenzo_max_stream_bytes(s["dims"], T)
    else:
        cap = (szp.max_stream_bytes_f64 if f64 else szp.max_stream_bytes)(n, block, T, fm)
    s["x"], s["cap"] = x, cap
    s["out"] = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    if case["kind"] == "decompress":
        s["size"] = _compress(s)
        s["out"] = s["out"][:s["size"]].clone()
        del s["x"]
    if case["kind"] == "reduce":
        first = s["out"]
        s["size_a"] = _compress(s)
        s["a"] = first[:s["size_a"]].clone()
        s["x"] = torch.flip(x, [0])
        s["size_b"] = _compress(s)
        s["b"] = first[:s["size_b"]].clone()
        del s["x"], first
        s["out"] = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    if case["kind"] in ("decompress", "roundtrip", "pipeline", "lorenzo"):
        s["y"] = torch.empty(n, dtype=x.dtype, device="cuda")
    if case["kind"] == "pipeline":
        s["d_size"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    return s


def _prepare_batch(s, seed):
    size, rels, _, at = _layout(s)
    T, nf = s["segments"], len(size)
    caps = [szp.max_stream_bytes(n, 32, T, 1) for n in size]
    off = np.concatenate([[0], np.cumsum([(c + 255) // 256 * 256 for c in caps])])
    s["x"] = _batch_fields(s, seed)
    s["streams"] = torch.zeros(int(off[-1]), dtype=torch.uint8, device="cuda")
    s["y"] = torch.zeros(at[-1], dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()  # a batch tunes itself on its fields, on a stream of its own
    x0, s0, y0 = s["x"].data_ptr(), s["streams"].data_ptr(), s["y"].data_ptr()
    cf = [dict(input=x0 + 4 * at[i], output=s0 + int(off[i]), output_bytes=caps[i], nbEle=size[i],
               errBoundMode=szp.REL, relBoundRatio=rels[i]) for i in range(nf)]
    s["cb"] = szp.Batch(szp.BATCH_COMPRESS, cf, 32, T, szp.BATCH_AUTOTUNE)
    s["cb"].run(_stream())
    s["cb"].sync()
    df = [dict(input=s0 + int(off[i]), input_bytes=caps[i], input_len_dev=s["cb"].sizes_dev() + 8 * i,
               output=y0 + 4 * at[i], output_bytes=4 * size[i], nbEle=size[i]) for i in range(nf)]
    s["db"] = szp.Batch(szp.BATCH_DECOMPRESS, df, 32, T, szp.BATCH_AUTOTUNE)
    return s


# ------------------------------------------------------------------- run ---

def _compress(s):
    mode, eb, rel = s["bounds"]
    f = szp.compress_dev_f64 if s["dtype"] == "f64" else szp.compress_dev
    return f(s["x"].data_ptr(), s["n"], s["out"].data_ptr(), s["cap"], mode, eb, rel, s["block"], s["segments"],
             s["fastmode"], _stream())


def _decompress(s, size):
    f = szp.decompress_dev_f64 if s["dtype"] == "f64" else szp.decompress_dev
    f(s["out"].data_ptr(), size, s["n"], s["y"].data_ptr(), s["block"], s["segments"], s["fastmode"], _stream())


def run(s):
    kind = s["kind"]
    if kind == "compress":
        return [_compress(s), s["out"]]
    if kind == "decompress":
        _decompress(s, s["size"])
        return s["y"]
    if kind == "roundtrip":
        size = _compress(s)
        _decompress(s, size)
        return [size, s["out"], s["y"]]
    if kind == "pipeline":
        mode, eb, rel = s["bounds"]
        args = (s["block"], s["segments"], s["fastmode"], _stream())
        szp.compress_dev_async(s["x"].data_ptr(), s["n"], s["out"].data_ptr(), s["cap"], s["d_size"].data_ptr(), mode,
                               eb, rel, *args)
        szp.decompress_dev_async(s["out"].data_ptr(), s["cap"], s["d_size"].data_ptr(), s["n"], s["y"].data_ptr(),
                                 *args)
        return [s["d_size"], s["out"], s["y"]]
    if kind == "reduce":
        size = szp.reduce_sum_dev(s["a"].data_ptr(), s["size_a"], s["b"].data_ptr(), s["size_b"], s["n"],
                                  s["out"].data_ptr(), s["cap"], s["block"], s["segments"], s["fastmode"],
                                  szp.SZ_FLOAT, _stream())
        return [size, s["out"]]
    if kind == "lorenzo":
        mode, eb, rel = s["bounds"]
        size = szp.lorenzo_compress_dev(s["x"].data_ptr(), s["dims"], s["out"].data_ptr(), s["cap"], mode, eb, rel,
                                        s["segments"], _stream())
        szp.lorenzo_decompress_dev(s["out"].data_ptr(), size, s["dims"], s["y"].data_ptr(), s["segments"], _stream())
        return [size, s["out"], s["y"]]
    if kind == "batch":
        s["cb"].run(_stream())
        s["db"].run(_stream())
        return [s["streams"], s["y"]]
    size = ctypes.c_size_t(0)
    f = (szp.lib.szp_float_openmp_threadblock_arg if s["fastmode"] == 1
         else szp.lib.szp_float_openmp_threadblock_randomaccess_arg)
    f(s["out"].ctypes.data, s["x"].ctypes.data, ctypes.byref(size), s["bounds"][1], s["n"], s["block"])
    y = szp.szp_decompress(s["out"][:size.value], s["n"], s["block"], s["fastmode"])
    return [size.value, s["out"], y]


# ------------------------------------------------------------------ work ---

def _block_bits(case, n, rel=None):
    """About how many bits a block of this field takes per value: the width of
    its largest of `block` deltas, in steps of the bound."""
    bound = rel or case["bound"]
    if case["field"] == "walk":
        step, span = 0.025, 2.0 + 0.016 * math.sqrt(n)
    elif case["field"] == "fourier":
        step, span = 0.035, 1.0
    else:
        step, span = 6e-3, 1.0
    return max(1.0, math.log2(1.0 + step / (bound * span)))


def _stream_bytes(case, n, rel=None):
    """The stream's size, estimated: a byte a block, and for the blocks that are
    not all zero their sign bits and the values' bits."""
    full = 0.6 if case["field"] == "laplace" else 1.0
    block = case["block"]
    bits = _block_bits(case, n, rel)
    return n / block * (1 + (4 if case["fastmode"] == 2 else 0) + full * block * (1 + bits) / 8)


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "batch":
        size, rels, kinds, _ = _layout(case)
        data = 4.0 * sum(size)
        packed = sum(_stream_bytes(dict(case, field="fourier" if k else "walk"), m, r)
                     for m, r, k in zip(size, rels, kinds))
        return {"bytes": 2 * (data + packed), "flops": 0.0}
    data = n * (8.0 if case["dtype"] == "f64" else 4.0)
    packed = _stream_bytes(case, n)
    if kind == "reduce":
        return {"bytes": 3 * packed, "flops": 0.0}
    if kind in ("compress", "decompress"):
        return {"bytes": data + packed, "flops": 0.0}
    return {"bytes": 2 * (data + packed), "flops": 0.0}


# ----------------------------------------------------------------- exact ---

def _values(x, rel=None, eb=None):
    """The values a stream of x stands for: trunc(x * (1 / eb)) * eb, with eb and
    its inverse of x's own type, as the format has it, and the rest in 64 bits."""
    one = torch.ones((), dtype=x.dtype, device=x.device)
    eb = (x.max() - x.min()) * (one * rel) if eb is None else one * eb
    return torch.trunc(x.double() * (one / eb).double()) * eb.double()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("compress", "reduce"):
        return None
    if kind == "batch":
        size, rels, _, at = _layout(case)
        x = _batch_fields(case, seed)
        y = torch.zeros(at[-1], dtype=torch.float64, device="cuda")
        for n, r, o in zip(size, rels, at):
            y[o:o + n] = _values(x[o:o + n], rel=r)
        return [None, y]
    x = _field(case, seed)
    mode, eb, rel = _bound(case, x)
    y = _values(x, rel=rel) if mode == szp.REL else _values(x, eb=eb)
    if kind == "decompress":
        return y
    return [None, None, y.cpu().numpy() if kind == "host" else y]
