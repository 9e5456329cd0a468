"""Unpredictable values through the gather and the scatter: whole decodes and
boxes bit-equal to the oracle's for chunk volumes that are a warp's work, fill
the CTA's pass, span several passes, or are no multiple of the 16-byte loads,
with few values, values in every place, and in one place of each chunk only."""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("share", [0.001, 1.0, "last"])
@pytest.mark.parametrize("dims,chunk", [((32, 32, 32), 2), ((40, 40, 40), 5), ((64, 64, 64), 16), ((64, 128, 64), 32),
                                        ((128, 128, 128), 64)])
def test_unpredictable_values_are_the_oracles(ctx, dtype, share, dims, chunk):
    rng = np.random.default_rng(chunk)
    f = np.zeros(dims, dtype)
    half = tuple(d // 2 for d in dims)
    for si in range(1, 8):
        if share == "last":
            m = np.zeros(half, bool)
            m[chunk - 1::chunk, chunk - 1::chunk, chunk - 1::chunk] = True
        else:
            m = rng.random(half) < share
        f[si >> 2 & 1::2, si >> 1 & 1::2, si & 1::2] = np.where(m, 1e6 + rng.standard_normal(half), 0)
    low = next(c for c in range(chunk, 0, -1) if all(d // 4 % c == 0 for d in dims))
    s = ctx.compress(torch.from_numpy(f).cuda(), eb=0.5, eb_mode="abs", bound_mode="reference", mult_base=1.0,
                     mult_low=1.0, mult_high=1.0, radius=64, chunk_high=chunk, chunk_low=low)
    want = po.compress(f, 0.5, radius=64, chunk_high=chunk, chunk_low=low, mults=(1.0, 1.0, 1.0))
    assert s.to_bytes() == want
    full = po.decompress(want)
    assert np.array_equal(ctx.decompress(s).view(np.uint8), full.view(np.uint8))
    nz, ny, nx = dims
    ctx.upload(s)
    box = ctx.decompress_box(s, (1, 0, 3), (nx - 2, ny // 2, nz // 2 + 3))
    assert np.array_equal(box.view(np.uint8), full[3:nz // 2 + 4, :ny // 2 + 1, 1:nx - 1].copy().view(np.uint8))
