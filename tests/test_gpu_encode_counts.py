"""The encoder's counts of unpredictable values and of codes far from the
centre: containers equal to the oracle's for fields whose every level loses
values (none to all, marker chunks of every edge against the kernels' tiles),
and for a single far code in one stream."""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.float64])  # the type that gathers its counts
@pytest.mark.parametrize("share", [0.001, 0.3, 1.0])
@pytest.mark.parametrize("dims,high,low", [((64, 64, 64), 1, 1), ((96, 96, 96), 3, 3), ((80, 80, 160), 20, 10),
                                           ((128, 128, 64), 32, 16), ((128, 128, 256), 64, 32)])
def test_values_lost_on_every_level(ctx, dtype, share, dims, high, low):
    rng = np.random.default_rng(high)
    f = rng.integers(-40, 41, dims).astype(dtype)
    f += np.where(rng.random(dims) < share, 1e6 * rng.standard_normal(dims), 0).astype(dtype)
    kw = dict(chunk_high=high, chunk_low=low)
    s = ctx.compress(torch.from_numpy(f).cuda(), eb=0.5, eb_mode="abs", bound_mode="reference", mult_base=1.0,
                     mult_low=1.0, mult_high=1.0, radius=64, **kw)
    assert s.to_bytes() == po.compress(f, 0.5, radius=64, mults=(1.0, 1.0, 1.0), **kw)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("far", [2047, 2048, -2048, -2049, 30000])
@pytest.mark.parametrize("at", [(1, 0, 0), (65, 64, 63), (2, 34, 66)])  # on the shell, inside, below the finest level
def test_one_far_code(ctx, dtype, far, at):
    f = np.zeros((128, 128, 128), dtype)
    f[at] = far
    s = ctx.compress(torch.from_numpy(f).cuda(), eb=0.5, eb_mode="abs", bound_mode="reference", mult_base=1.0,
                     mult_low=1.0, mult_high=1.0, chunk_high=32, chunk_low=16)
    assert s.to_bytes() == po.compress(f, 0.5, chunk_high=32, chunk_low=16, mults=(1.0, 1.0, 1.0))
