"""The entropy decoder at the edges of its plane shapes: whole decodes and
boxes equal to the oracle's for plane sizes that take each lane count (1 to 32
lanes), are no multiple of the 16-byte stores, or exceed the shared buffers
(chunk edge 64), and for planes whose payload exceeds the staged words (16-bit
codes), is nothing but one run, or ends in a long code. Codes are chosen as in
test_gpu_codebook: a zero coarse grid, multipliers 1, eb 0.5."""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _field(kind, dims, rng):
    f = np.zeros(dims, np.float32)
    n = f.size // 8
    for si in range(1, 8):
        if kind == "sparse":
            v = np.where(rng.random(n) < 0.01, rng.integers(-5, 6, n), 0)
        elif kind == "rough":
            v = np.rint(rng.laplace(0, 300, n))
        elif kind == "widest":
            v = rng.permutation(np.arange(n) % 65000 - 32500)
        else:  # one value in the whole stream, at a plane's last code
            v = np.zeros(n)
            v[-1] = 7
        f[si >> 2 & 1::2, si >> 1 & 1::2, si & 1::2] = v.reshape(dims[0] // 2, dims[1] // 2, -1)
    return f


@pytest.mark.parametrize("kind", ["sparse", "rough", "lone"])
@pytest.mark.parametrize("dims,chunk", [
    ((64, 64, 64), 1), ((40, 40, 80), 5), ((56, 56, 28), 7), ((48, 96, 48), 12), ((64, 128, 64), 16),
    ((120, 60, 60), 30), ((64, 64, 64), 32), ((128, 128, 128), 64),
])
def test_decode_of_every_plane_shape_is_the_oracles(ctx, kind, dims, chunk):
    _check(ctx, _field(kind, dims, np.random.default_rng(chunk + len(kind))), chunk)


def test_decode_of_planes_past_the_staged_words_is_the_oracles(ctx):
    _check(ctx, _field("widest", (128, 128, 128), np.random.default_rng(3)), 32)


def _check(ctx, f, chunk):
    low = next(c for c in range(chunk, 0, -1) if all(d // 4 % c == 0 for d in f.shape))
    want = po.compress(f, 0.5, chunk_high=chunk, chunk_low=low, mults=(1.0, 1.0, 1.0))
    s = ctx.parse(want)
    full = po.decompress(want)
    assert np.array_equal(ctx.decompress(s).view(np.uint32), full.view(np.uint32))
    nz, ny, nx = f.shape
    lo, hi = (1, 2, 3), (nx - 3, ny // 2, nz - 1)
    ctx.upload(s)
    box = ctx.decompress_box(s, lo, hi)
    assert np.array_equal(box.view(np.uint32), full[lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].copy().view(np.uint32))
