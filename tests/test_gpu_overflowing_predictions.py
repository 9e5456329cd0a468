"""float32 fields whose predictions overflow: second differences of about 3e6
and more make the blended weights (products of three squares) infinite and the
prediction NaN, as in the reference, and the residual of a finite value is then
NaN on both sides. The container is the oracle's but for the bits of such NaNs
(the GPU gives 0x7fffffff, x86 0xffc00000): every frame but the values, every
finite value, the places of the NaNs and the decoded field agree. Fields of
double precision, and float32 fields without such jumps, have no exception."""
import struct

import numpy as np
import pytest

import pyoracle as po
import stream_tools

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _streams(b):
    """Per stream (header bytes without the values, values, payload bytes)."""
    sizes = stream_tools.frame_sizes(b)
    pos, out = len(b) - sum(x[3] for x in sizes), []
    for _, _, kind, stored, raw in sizes:
        f = stream_tools._unzstd(b[pos:pos + stored], raw)
        pos += stored
        if kind == "header":
            p = 4 + 3 * struct.unpack_from("<I", f, 0)[0] + 8
            n = struct.unpack_from("<Q", f, p)[0]
            out.append([f[:p + 8] + f[p + 8 + 4 * n:], np.frombuffer(f, np.uint32, n, p + 8), b""])
        else:
            out[-1][2] += f
    return out


@pytest.mark.parametrize("share", [0.001, 0.3, 1.0])
@pytest.mark.parametrize("dims,high,low", [((64, 64, 64), 1, 1), ((96, 96, 96), 3, 3), ((80, 80, 160), 20, 10),
                                           ((128, 128, 64), 32, 16), ((128, 128, 256), 64, 32)])
def test_float32_values_lost_on_every_level(ctx, share, dims, high, low):
    rng = np.random.default_rng(high)
    f = rng.integers(-40, 41, dims).astype(np.float32)
    f += np.where(rng.random(dims) < share, 1e6 * rng.standard_normal(dims), 0).astype(np.float32)
    kw = dict(chunk_high=high, chunk_low=low)
    got = ctx.compress(torch.from_numpy(f).cuda(), eb=0.5, eb_mode="abs", bound_mode="reference", mult_base=1.0,
                       mult_low=1.0, mult_high=1.0, radius=64, **kw).to_bytes()
    want = po.compress(f, 0.5, radius=64, mults=(1.0, 1.0, 1.0), **kw)
    a, b = _streams(got), _streams(want)
    assert len(a) == len(b)
    nans = 0
    for (ha, va, pa), (hb, vb, pb) in zip(a, b):
        assert ha == hb and pa == pb
        na, nb = np.isnan(va.view(np.float32)), np.isnan(vb.view(np.float32))
        assert np.array_equal(na, nb) and np.array_equal(va[~na], vb[~nb])
        nans += int(na.sum())
    if share < 0.01:
        assert nans == 0 and got == want
    else:
        assert nans > 0
    full = po.decompress(want)
    out = ctx.decompress(ctx.parse(got))
    assert np.array_equal(np.isnan(out), np.isnan(full))
    assert np.array_equal(out[~np.isnan(out)].view(np.uint32), full[~np.isnan(full)].view(np.uint32))
