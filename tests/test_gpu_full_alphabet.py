"""Decodes of streams that use every code value: 65500 codes of the finest
level (the centre and code 0 among them) and the 36 run symbols of 32 x 32
planes make 65536 symbols, so the last canonical index is 0xffff. Whole
decodes, boxes and slices equal to the oracle's, with and without the last few
symbols in use. Codes are chosen as in test_gpu_codebook: a zero coarse grid,
multipliers 1, eb 0.5."""
import struct

import numpy as np
import pytest

import pyoracle as po
import stream_tools

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

RADIUS, PLANE, SLOTS = 32768, 1024, 36


def _finest(dropped, rng):
    """Codes (minus the radius) of one sub-block of 64^3: a free block of SLOTS
    code values, `dropped` more unused, every other value at least once, and
    centre codes in runs of every length."""
    free = set(range(100, 100 + SLOTS)) | set(range(-30000, -30000 + dropped))
    lits = [k for k in range(1 - RADIUS, RADIUS) if k and k not in free]
    lits += [10 ** 6] * 3  # code 0
    lits = [int(v) for v in rng.permutation(lits)]
    out = []
    for rep in range(2):
        for r in range(1, 31):
            out += [0] * r + [lits.pop()]
        out += [0] * (-len(out) % PLANE)
        for r in (64, 128, 256, 511):
            out += [0] * r + [lits.pop()]
        out += [0] * (-len(out) % PLANE)
        out += [0] * 600 + [lits.pop()]
        out += [0] * (-len(out) % PLANE)
        out += [0] * PLANE
    for v in lits:
        out += [v] if rng.random() < 0.5 else [0] * int(rng.integers(1, 4)) + [v]
    assert len(out) <= 64 ** 3
    return np.array(out + [0] * (64 ** 3 - len(out)), np.float64)


def _field(dropped, dtype, rng):
    f = np.zeros((128, 128, 128), dtype)
    codes = _finest(dropped, rng).reshape(2, 2, 2, 32, 32, 32)  # chunk by chunk
    blk = codes.transpose(0, 3, 1, 4, 2, 5).reshape(64, 64, 64)
    f[1::2, 0::2, 0::2] = blk
    return f


def symbols_used(b):
    """(symbols, first run symbol, run symbols) of every stream's codebook."""
    out, sizes = [], stream_tools.frame_sizes(b)
    pos = len(b) - sum(x[3] for x in sizes)
    for _, _, kind, stored, raw in sizes:
        if kind == "header":
            h = stream_tools._unzstd(b[pos:pos + stored], raw)
            nu = struct.unpack_from("<I", h, 0)[0]
            out.append((nu,) + struct.unpack_from("<2I", h, 4 + 3 * nu))
        pos += stored
    return out


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dropped", [0, 1, 200])
def test_every_code_value_in_use(ctx, dtype, dropped):
    f = _field(dropped, dtype, np.random.default_rng(dropped))
    kw = dict(chunk_high=32, chunk_low=16)
    want = po.compress(f, 0.5, mults=(1.0, 1.0, 1.0), **kw)
    assert max(symbols_used(want))[0::2] == (65536 - dropped, SLOTS)
    s = ctx.compress(torch.from_numpy(f).cuda(), eb=0.5, eb_mode="abs", bound_mode="reference", mult_base=1.0,
                     mult_low=1.0, mult_high=1.0, **kw)
    assert s.to_bytes() == want
    full = po.decompress(want)
    bits = np.uint32 if dtype == np.float32 else np.uint64
    s = ctx.parse(want)
    assert np.array_equal(ctx.decompress(s).view(bits), full.view(bits))
    ctx.upload(s)
    for lo, hi in (((0, 0, 0), (127, 127, 127)), ((3, 5, 7), (90, 41, 126)), ((0, 0, 63), (127, 127, 63))):
        box = ctx.decompress_box(s, lo, hi)
        assert np.array_equal(box.view(bits), full[lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].copy().view(bits))
