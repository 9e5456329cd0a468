"""Codebooks built on the device: streams byte-identical to the oracle's for
fields whose finest-level code histograms are chosen. With a zero coarse grid
every prediction is zero, so at multipliers 1 and eb 0.5 a fine value k is
coded as radius + k. The cases sit where the construction can go wrong: one
and two symbols, all-equal counts (ties), symbol counts around the one-warp
and whole-CTA merges, Fibonacci counts (the longest codes,
past the 24-bit cap), geometric counts, codes over the whole range with
unpredictable values, a radius that leaves no room for run symbols, and
planes of one code (no run symbols at all)."""
import numpy as np
import pytest

import pyoracle as po
import stz_b200

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _codes(kind, n, rng):
    """n values to code in one sub-block (0 is the centre code)."""
    if kind == "one":
        return np.zeros(n)
    if kind == "two":
        return rng.integers(0, 2, n)
    if kind == "equal":
        return np.arange(n) % 4096 - 2048
    if kind.startswith("first"):  # that many codes, some of equal counts
        k = int(kind[5:])
        return np.arange(n) % k - k // 2
    if kind == "wide":
        return np.arange(n) % 40000 - 20000
    if kind == "fibonacci":
        f = [1, 1]
        while len(f) < 26:
            f.append(f[-1] + f[-2])
        v = np.repeat(np.arange(1, 27), f)
        return rng.permutation(np.concatenate([v, np.zeros(n - v.size)]))
    if kind == "geometric":
        return rng.permutation(rng.geometric(0.5, n) * rng.choice([-1, 1], n))
    if kind == "unpredictable":
        return np.where(rng.random(n) < 0.01, 1e6, np.rint(rng.laplace(0, 400, n)))
    if kind == "runs":
        return np.where(rng.random(n) < 0.02, rng.integers(-30, 31, n), 0)
    raise ValueError(kind)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind,dims,radius,chunk", [
    ("one", (64, 64, 64), 32768, 32),
    ("two", (64, 64, 64), 32768, 32),
    ("equal", (64, 128, 64), 32768, 32),
    ("first511", (64, 64, 64), 32768, 32),
    ("first512", (64, 64, 64), 32768, 32),
    ("first513", (64, 64, 64), 32768, 32),
    ("first1025", (64, 64, 64), 32768, 32),
    ("wide", (128, 128, 128), 32768, 32),
    ("fibonacci", (128, 128, 192), 32768, 32),
    ("geometric", (128, 64, 64), 32768, 32),
    ("unpredictable", (64, 64, 128), 32768, 32),
    ("runs", (128, 128, 64), 1024, 16),
    ("runs", (64, 64, 64), 20, 32),
    ("unpredictable", (32, 32, 32), 2, 2),
    ("runs", (32, 48, 16), 512, 1),
])
def test_stream_with_a_chosen_histogram_is_the_oracles(ctx, dtype, kind, dims, radius, chunk):
    rng = np.random.default_rng(len(kind) + sum(dims) + radius)
    f = np.zeros(dims, dtype)
    n = f.size // 8
    for si in range(1, 8):
        f[si >> 2 & 1::2, si >> 1 & 1::2, si & 1::2] = _codes(kind, n, rng).reshape(dims[0] // 2, dims[1] // 2, -1)
    low = max(1, chunk // 2)
    s = ctx.compress(torch.from_numpy(f).cuda(), eb=0.5, eb_mode="abs", bound_mode="reference", mult_base=1.0,
                     mult_low=1.0, mult_high=1.0, radius=radius, chunk_high=chunk, chunk_low=low)
    want = po.compress(f, 0.5, radius=radius, chunk_high=chunk, chunk_low=low, mults=(1.0, 1.0, 1.0))
    assert s.to_bytes() == want
    out = ctx.decompress(s)
    assert np.array_equal(out.view(np.uint8), po.decompress(want).view(np.uint8))
