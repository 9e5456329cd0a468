"""The decoder that gives every plane a thread: whole decodes of resident
streams and large boxes equal to the oracle's where its launches are large
enough (256 items of 128 planes, 64 of planes past 1024 codes) and below, for plane sizes
that are multiples of 8, for plane counts that leave its last threads idle, for
codes of every length (a few symbols, long codes, every code value, 24 bits), for lone
symbols, for streams with run symbols or planes of odd sizes among the others,
and served. Codes are chosen as in test_gpu_codebook: a zero coarse grid,
multipliers 1, eb 0.5."""
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

import pyoracle as po
from conftest import ROOT

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _codes(kind, n, rng):
    if kind == "rough":  # codes of up to about 20 bits
        return np.rint(rng.laplace(0, 300, n))
    if kind == "narrow":  # two or three bits a code, few runs
        return rng.integers(-2, 3, n)
    if kind == "widest":  # nearly all code values
        return rng.permutation(np.arange(n) % 65000 - 32500)
    if kind == "longest":  # Fibonacci counts: codes up to the 24-bit cap, and a bit for most
        f = [1, 1]
        while sum(f) + f[-1] + f[-2] < n // 2:
            f.append(f[-1] + f[-2])
        v = np.repeat(np.arange(1, len(f) + 1), f)
        return rng.permutation(np.concatenate([v, np.full(n - v.size, -1)]))
    if kind == "lone":
        return np.full(n, 3)
    return np.where(rng.random(n) < 0.02, rng.integers(-30, 31, n), 0)  # "runs"


def _field(kinds, dims, dtype, rng):
    f = np.zeros(dims, dtype)
    n = f.size // 8
    for si in range(1, 8):
        v = _codes(kinds[si % len(kinds)], n, rng)
        f[si >> 2 & 1::2, si >> 1 & 1::2, si & 1::2] = v.reshape(dims[0] // 2, dims[1] // 2, -1)
    return f


def _launches(ctx, fn):
    ctx.profile_reset()
    out = fn()
    n = {k: v[1] for k, v in ctx.profile_read().items()}
    return out, n.get("k_decode_planes", 0), n.get("k_decode", 0)


# (kinds, dims, chunk, the whole decode goes by plane)
CASES = [
    (["rough"], (144, 144, 144), 8, True),       # 7 x 46 items, the last of each 9 chunks of 16
    (["narrow"], (144, 144, 144), 8, True),
    (["widest"], (144, 144, 144), 8, False),     # 16 bits a code: count for half
    (["widest"], (176, 176, 176), 8, True),
    (["longest"], (160, 144, 144), 8, True),
    (["lone"], (144, 144, 144), 8, True),        # no bits at all
    (["rough", "runs", "lone"], (200, 200, 200), 10, False),  # planes of 100 codes: not a multiple of 8
    (["rough", "rough", "runs"], (192, 192, 192), 8, True),   # a launch of both kinds
    (["rough"], (240, 240, 240), 20, True),      # 6 chunks of 20 planes an item
    (["rough"], (96, 96, 96), 8, False),         # too few items
    (["runs"], (144, 144, 144), 8, False),
    (["rough"], (144, 144, 144), 4, True),       # planes of 16 codes
    (["rough"], (144, 144, 144), 2, False),      # of 4
]


@pytest.mark.parametrize("kinds,dims,chunk,by_plane", CASES)
def test_decodes_by_plane_are_the_oracles(ctx, kinds, dims, chunk, by_plane):
    f = _field(kinds, dims, np.float32, np.random.default_rng(chunk + len(kinds) + sum(dims)))
    low = next(c for c in range(chunk, 0, -1) if all(d // 4 % c == 0 for d in dims))
    want = po.compress(f, 0.5, chunk_high=chunk, chunk_low=low, mults=(1.0, 1.0, 1.0))
    full = po.decompress(want)
    s = ctx.parse(want)
    assert np.array_equal(ctx.decompress(s).view(np.uint32), full.view(np.uint32))
    ctx.upload(s)
    for _ in range(2):  # whatever the buffers held
        out, np_, ng = _launches(ctx, lambda: ctx.decompress(s))
        assert np.array_equal(out.view(np.uint32), full.view(np.uint32))
        assert (np_ > 0) == by_plane
        assert ng > 0 or by_plane
    nz, ny, nx = dims
    lo, hi = (1, 0, 2), (nx - 2, ny - 1, nz - 3)
    box = ctx.decompress_box(s, lo, hi)
    assert np.array_equal(box.view(np.uint32), full[2:nz - 2, :, 1:nx - 1].copy().view(np.uint32))


@pytest.mark.parametrize("dims,chunk,by_plane", [((264, 132, 132), 33, False), ((288, 288, 288), 48, True)])
def test_planes_past_the_shared_buffers(ctx, dims, chunk, by_plane):
    """1089 and 2304 codes: by lane groups with codes straight to memory, or by plane."""
    f = _field(["rough", "widest", "runs"] if not by_plane else ["rough"], dims, np.float32, np.random.default_rng(chunk))
    low = next(c for c in range(chunk, 0, -1) if all(d // 4 % c == 0 for d in dims))
    want = po.compress(f, 0.5, chunk_high=chunk, chunk_low=low, mults=(1.0, 1.0, 1.0))
    full = po.decompress(want)
    s = ctx.parse(want)
    ctx.upload(s)
    out, np_, _ = _launches(ctx, lambda: ctx.decompress(s))
    assert (np_ > 0) == by_plane
    assert np.array_equal(out.view(np.uint32), full.view(np.uint32))


def test_served_levels_by_plane(ctx):
    """The bulk lane's whole decodes, with boxes of the fast lane beside them."""
    from stz_b200 import Server

    dims = (144, 144, 144)
    f = _field(["rough", "rough", "runs"], dims, np.float32, np.random.default_rng(1))
    f[::3, 1::2, ::5] += 1e6  # a list of unpredictable values
    want = po.compress(f, 0.5, chunk_high=8, chunk_low=4, mults=(1.0, 1.0, 1.0))
    full = po.decompress(want)
    srv = Server(0, arena_bytes=1 << 30)
    try:
        sid = srv.add_stream(ctx.parse(want))
        t = [srv.submit_level(sid, level) for level in (0, 1, 0)] + [srv.submit_box(sid, (3, 4, 5), (90, 91, 92))]
        r = [srv.copy_out(srv.wait(x), np.float32) for x in t]
        assert np.array_equal(r[0].view(np.uint32), full.view(np.uint32))
        assert np.array_equal(r[1].view(np.uint32), po.decompress(want, 1).view(np.uint32))
        assert np.array_equal(r[2].view(np.uint32), full.view(np.uint32))
        assert np.array_equal(r[3].view(np.uint32), full[5:93, 4:92, 3:91].copy().view(np.uint32))
        for x in t:
            srv.release(x)
    finally:
        srv.close()


CHILD = r"""
import hashlib, sys
sys.path[:0] = sys.argv[1:3]
import numpy as np
import stz_b200
ctx = stz_b200.Context(0)
s = ctx.parse(open(sys.argv[3], "rb").read())
ctx.upload(s)
ctx.profile_reset()
out = ctx.decompress(s)
print(ctx.profile_read().get("k_decode_planes", (0, 0))[1], hashlib.sha256(out.tobytes()).hexdigest())
"""


@pytest.mark.parametrize("bits,by_plane", [(None, True), ("0", True), ("200", True), ("1000", False), ("4294967295", False)])
def test_the_switch_between_the_two_forms(tmp_path, bits, by_plane):
    """STZ_DECODE_SEQ_BITS, read once a process: the least payload bits a plane
    (64 codes of about 10 bits here) for a thread per plane. Same output."""
    dims = (144, 144, 144)
    f = _field(["rough"], dims, np.float32, np.random.default_rng(2))
    want = po.compress(f, 0.5, chunk_high=8, chunk_low=4, mults=(1.0, 1.0, 1.0))
    (tmp_path / "s").write_bytes(want)
    env = {k: v for k, v in os.environ.items() if k != "STZ_DECODE_SEQ_BITS"}
    if bits is not None:
        env["STZ_DECODE_SEQ_BITS"] = bits
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "sc25-stz2_b200"), ROOT, str(tmp_path / "s")],
                       capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr
    n, h = r.stdout.split()[-2:]
    assert (int(n) > 0) == by_plane
    assert h == hashlib.sha256(po.decompress(want).tobytes()).hexdigest()
