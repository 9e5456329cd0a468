"""The work a program has this library do, as cases that can be timed: compress a field on the device, decompress a
stream (whole, at reduced resolution, or by boxes and slices), serve a burst of requests from a resident stream, and
the round trip of a program whose arrays are on the host.

Every case goes through the Python binding's public entry points (`Context`, `Server`) or, for the bytes of a stream,
the C entry point the binding declares. Fields are the library's three synthetic families (Gaussian random field,
lognormal, shear fronts) made on the GPU from the seed; sizes and bounds are those of the benchmark configurations
and the tests, and their neighbours.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sc25-stz2_b200"))
import stz_b200  # noqa: E402

_DTYPES = {"f32": torch.float32, "f64": torch.float64}

# A program keeps one context for all the fields it codes (a device, its streams and grow-only buffers).
_context = None


def _ctx():
    global _context
    if _context is None:
        _context = stz_b200.Context(torch.cuda.current_device())
    return _context


# ---- fields ------------------------------------------------------------------
def _grf(shape, alpha, seed):
    """Unit-variance Gaussian random field with power spectrum k^-alpha, float32 on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
    kz, ky = (torch.fft.fftfreq(n, device="cuda") for n in shape[:2])
    kx = torch.fft.rfftfreq(shape[2], device="cuda")
    k2 = kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    f *= k2.pow(-alpha / 4.0)
    f[0, 0, 0] = 0.0
    del k2
    f = torch.fft.irfftn(f, s=shape)
    return f / f.std()


def _field(case, seed):
    """The case's field (z, y, x) on the GPU, in its type."""
    shape = (case["nz"], case["ny"], case["nx"])
    if case["field"] == "grf":
        f = _grf(shape, 3.0, seed)
    elif case["field"] == "lognormal":
        f = torch.exp(1.5 * _grf(shape, 3.0, seed))
    else:  # tanh shear fronts over a rough field
        f = _grf(shape, 5.0 / 3.0, seed).double()
        r = np.random.default_rng(seed + 7919)
        z, y, x = (torch.arange(n, device="cuda", dtype=torch.float64) for n in shape)
        for _ in range(20):
            nv = r.standard_normal(3)
            nv /= np.linalg.norm(nv)
            c, w = r.uniform(0, 1, 3) * np.array(shape[::-1]), r.uniform(2, 8)
            sz, sy, sx = (z - c[2]) * (nv[2] / w), (y - c[1]) * (nv[1] / w), (x - c[0]) * (nv[0] / w)
            f += 3.0 * torch.tanh(sz[:, None, None] + sy[None, :, None] + sx[None, None, :])
    return f.to(_DTYPES[case["dtype"]]).contiguous()


# ---- cases -------------------------------------------------------------------
def _case(name, op, dims, field, dtype, eb, predictor="dynamic", chunk=32, **more):
    c = {"op": op, "nx": dims[0], "ny": dims[1], "nz": dims[2], "field": field, "dtype": dtype, "eb": eb,
         "predictor": predictor, "chunk": chunk, **more}
    return {"name": name, **c} if name else c


def listed():
    cube, wide = (512, 512, 512), (384, 384, 256)
    return [
        # the smallest fields in use: a solver's 64^3 block, one call after another, where launches and latency count
        _case("compress_64_f32", "compress", (64, 64, 64), "grf", "f32", 1e-3),
        _case("decompress_64_f32", "decompress", (64, 64, 64), "grf", "f32", 1e-3),
        # the headline workload: a 512^3 snapshot at the usual bound
        _case("compress_512_f32", "compress", cube, "lognormal", "f32", 1e-3),
        _case("decompress_512_f32", "decompress", cube, "lognormal", "f32", 1e-3),
        # the same snapshot at the tight end of the bound sweep: four times the stream
        _case("compress_512_f32_tight", "compress", cube, "lognormal", "f32", 1e-4),
        _case("decompress_512_f32_tight", "decompress", cube, "lognormal", "f32", 1e-4),
        # double precision with sharp fronts at a tight bound (unpredictable values, wide codebooks)
        _case("compress_384_f64", "compress", wide, "fronts", "f64", 1e-6),
        _case("decompress_384_f64", "decompress", wide, "fronts", "f64", 1e-6),
        # a preview of the snapshot at half resolution, before it is worth decoding whole
        _case("half_res_512_f32", "level", cube, "lognormal", "f32", 1e-3, level=1),
        # an analysis that reads boxes and slices of uneven size from a resident stream, one at a time
        _case("boxes_384_f64", "box", wide, "fronts", "f64", 1e-6, requests=24),
        # a server's burst of small boxes from many clients on one resident field
        _case("serve_512_f32", "serve", cube, "grf", "f32", 1e-3, requests=64),
        # host arrays in and out, a ragged field, small marker chunks and the fixed-weight predictor
        _case("host_ragged_f32", "host", (336, 272, 208), "grf", "f32", 1e-3, predictor="cubic", chunk=8),
    ]


# Bytes of the largest drawn fields: the 512^3 float32 snapshot for whole-field work, half of it where a pass costs
# more per byte (double precision, the staged predictors), a quarter for host arrays.
_FULL, _HALF, _HOST = 4 << 27, 4 << 26, 4 << 25


def draw(rng):
    op = rng.choice(["compress", "compress", "decompress", "decompress", "level", "box", "serve", "host"])
    dtype = rng.choice(["f32", "f32", "f64"])
    predictor = rng.choice(["dynamic"] * 6 + ["cubic", "cubic", "staged", "truncated"])
    if op in ("box", "serve") and predictor in ("staged", "truncated"):  # the server does not take these streams
        predictor = "dynamic"
    field = rng.choice(["grf", "lognormal", "fronts"])
    chunk = rng.choice([32, 32, 32, 8])
    most = _HOST if op == "host" else _FULL if dtype == "f32" and predictor in ("dynamic", "cubic") else _HALF
    if op in ("box", "serve"):
        least = 128
    else:
        least = 64
    grain = 2 * chunk  # edges are whole numbers of finest-level marker chunks
    edges = []
    for _ in range(3):
        e = math.exp(rng.uniform(math.log(least), math.log(640)))
        edges.append(max(least, int(round(e / grain)) * grain))
    size = 8 if dtype == "f64" else 4
    while edges[0] * edges[1] * edges[2] * size > most:
        i = edges.index(max(edges))
        edges[i] -= grain
    tight = -4.0 if dtype == "f32" else -6.0
    eb = float("%.2g" % 10 ** rng.uniform(tight, -2.0))
    more = {}
    if op == "level":
        more["level"] = rng.choice([1, 1, 2, 3])
    elif op == "box":
        more["requests"] = rng.randint(4, 24)
    elif op == "serve":
        more["requests"] = rng.randint(1, 64)
    return _case(None, op, edges, field, dtype, eb, predictor, chunk, **more)


# ---- requests ----------------------------------------------------------------
def _requests(case, seed):
    """(lo, hi) inclusive corners (x, y, z): boxes with edges in [16, 128] and one slice in six, or 64^3 boxes. Their
    extents belong to the case, where they lie to the seed."""
    shape, place = np.random.default_rng(case["requests"]), np.random.default_rng(seed)
    dims = (case["nx"], case["ny"], case["nz"])
    out = []
    for i in range(case["requests"]):
        if case["op"] == "box" and i % 6 == 5:
            edge = list(dims)
            edge[int(shape.integers(0, 3))] = 1
        else:
            edge = [int(e) for e in shape.integers(16, 129, 3)] if case["op"] == "box" else [64, 64, 64]
        lo = [int(place.integers(0, d - e + 1)) for d, e in zip(dims, edge)]
        out.append((lo, [v + e - 1 for v, e in zip(lo, edge)]))
    return out


def _crop(f, lo, hi):
    return f[lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1]


# ---- one pass ----------------------------------------------------------------
class _DeviceArray:
    """A served result as a CUDA array, where it lies in the server's output arena (the tensor made from it keeps
    this object, and so the server, alive)."""

    def __init__(self, server, res, dtype):
        self.server = server
        self.__cuda_array_interface__ = {"shape": res.shape, "typestr": dtype, "data": (res.out_dev, False), "version": 2}


class _StreamBytes(dict):
    """A stream's length and its serialized bytes. The bytes stay where the library has them (stz_stream_bytes), as
    for a program that writes them to a file; who reads them here gets them zero-padded to a size that every stream of
    the case fits, since streams of other fields have other lengths."""

    def __init__(self, stream, case):
        p, n = ctypes.c_void_p(), ctypes.c_size_t()
        if stz_b200.load_library().stz_stream_bytes(stream.handle, ctypes.byref(p), ctypes.byref(n)):
            raise RuntimeError("stz_stream_bytes failed")
        super().__init__(length=n.value, bytes=p.value)
        self._stream, self._size = stream, int(4 * _coded_bytes(case)) + (2 << 20)

    def __getitem__(self, key):
        if key != "bytes":
            return super().__getitem__(key)
        n = self["length"]
        out = np.zeros(self._size, np.uint8)
        out[:n] = np.ctypeslib.as_array((ctypes.c_uint8 * n).from_address(super().__getitem__(key)))
        return out


def prepare(case, seed):
    ctx = _ctx()
    chunk = case["chunk"]
    o = stz_b200.default_opts(eb=case["eb"], eb_mode="rel", predictor=case["predictor"], chunk_high=chunk,
                              chunk_low=chunk // 2)
    f = _field(case, seed)
    st = {"case": dict(case), "opts": o, "op": case["op"]}
    if case["op"] == "compress":
        st["field"] = f
        return st
    if case["op"] == "host":
        st["array"] = f.cpu().numpy()
        return st
    stream = ctx.parse(ctx.compress(f, opts=o).to_bytes())  # as read back from a file
    if case["op"] == "serve":
        st["server"] = stz_b200.Server(torch.cuda.current_device(), arena_bytes=256 << 20)
        st["id"] = st["server"].add_stream(stream)
        st["requests"] = _requests(case, seed)
        st["tickets"] = []
        return st
    st["stream"] = stream
    if case["op"] == "box":
        ctx.upload(stream)
        st["requests"] = _requests(case, seed)
        st["out"] = [torch.empty_like(_crop(f, lo, hi), memory_format=torch.contiguous_format)
                     for lo, hi in st["requests"]]
    else:
        lv = case.get("level", 0)
        st["out"] = torch.empty((case["nz"] >> lv, case["ny"] >> lv, case["nx"] >> lv), dtype=f.dtype, device="cuda")
    return st


def run(st):
    ctx, op = _ctx(), st["op"]
    if op == "compress":
        st["stream"] = None  # the last snapshot's stream has been written out
        st["stream"] = ctx.compress(st["field"], opts=st["opts"])
        return _StreamBytes(st["stream"], st["case"])
    if op in ("decompress", "level"):
        return ctx.decompress(st["stream"], level=st["case"].get("level", 0), out=st["out"])
    if op == "box":
        return [ctx.decompress_box(st["stream"], lo, hi, out=o) for (lo, hi), o in zip(st["requests"], st["out"])]
    if op == "serve":
        srv = st["server"]
        for t in st["tickets"]:  # the last burst's results have been read
            srv.release(t)
        st["tickets"] = [srv.submit_box(st["id"], lo, hi) for lo, hi in st["requests"]]
        done = [srv.wait(t) for t in st["tickets"]]
        dtype = "<f8" if st["case"]["dtype"] == "f64" else "<f4"
        return [torch.as_tensor(_DeviceArray(srv, r, dtype), device="cuda") for r in done]
    st["stream"] = None
    st["stream"] = ctx.compress(st["array"], opts=st["opts"])
    return [_StreamBytes(st["stream"], st["case"]), ctx.decompress(st["stream"])]


def exact(case, seed):
    """What a decode would return without its error bound: the field's own values, where the bound leaves them within
    a tenth of the values' norm. A stream has no such value."""
    if case["op"] == "compress":
        return None
    f = _field(case, seed).double()
    level = case.get("level", 0)
    share = 1.0 if level == 0 else 2.7 / 8.2 if level == 1 else 0.7 / 8.2  # the coarser levels' share of the bound
    bound = share * case["eb"] * float(f.max() - f.min())

    def near(v):
        return v.contiguous() if bound <= 0.1 * float(v.square().mean().sqrt()) else None

    if case["op"] == "host":
        return [None, near(f)]
    if case["op"] in ("box", "serve"):
        return [near(_crop(f, lo, hi)) for lo, hi in _requests(case, seed)]
    return near(f[::1 << level, ::1 << level, ::1 << level])


# Coded bits per value near a relative bound of 1e-3, and how many more a tenth of the bound costs.
_BITS = {"grf": (6.0, 3.3), "lognormal": (0.6, 2.1), "fronts": (5.0, 3.6)}


def _coded_bytes(case, n=None):
    """About the coded size of n values (all of the field's) of the case."""
    base, slope = _BITS[case["field"]]
    n = case["nx"] * case["ny"] * case["nz"] if n is None else n
    return n * max(0.1, base + slope * (-math.log10(case["eb"]) - 3.0)) / 8


def work(case):
    """Bytes: the field or boxes once, and the coded stream (or the boxes' share of it) once. Flops: the predictor's
    about 216 operations for the seven values of a cell."""
    n = case["nx"] * case["ny"] * case["nz"]
    if case["op"] == "level":
        n >>= 3 * case["level"]
    elif case["op"] in ("box", "serve"):
        n = sum(math.prod(b - a + 1 for a, b in zip(lo, hi)) for lo, hi in _requests(case, 0))
    both = 2 if case["op"] == "host" else 1
    size = 8 if case["dtype"] == "f64" else 4
    return {"bytes": both * (n * size + _coded_bytes(case, n)), "flops": both * 27 * n}
