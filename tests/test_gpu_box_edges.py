"""Boxes and slices whose ends lie beside marker-chunk faces: a window's cells
then hold parities whose own chunks the request does not decode. Equal to the
cut of the oracle's whole decode, with unpredictable values nowhere (a stream
without a list of them), in every chunk, and in a chunk's first and last plane
only; one by one, in one server batch on buffers that nothing has filled, and
after larger requests have."""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint8)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("unpred", ["none", "some", "edges"])
@pytest.mark.parametrize("dims,high,low", [((64, 64, 64), 16, 8), ((40, 40, 40), 5, 5), ((128, 64, 64), 32, 16),
                                           ((256, 128, 128), 64, 32)])
def test_boxes_beside_chunk_faces_are_the_cut(ctx, dtype, unpred, dims, high, low):
    from stz_b200 import Server

    rng = np.random.default_rng(high)
    z, y, x = np.ogrid[: dims[0], : dims[1], : dims[2]]
    f = np.sin(x / 9.0) * np.cos(y / 7.0) + np.sin(z / 5.0) + 0.01 * rng.standard_normal(dims)
    if unpred == "some":
        f[rng.random(dims) < 0.002] += 1e6
    elif unpred == "edges":
        edge = (np.arange(dims[0]) // 2 % high == 0) | (np.arange(dims[0]) // 2 % high == high - 1)
        odd = np.arange(dims[2]) % 2 == 1  # no other sample is predicted from these
        f[(rng.random(dims) < 0.004) & edge[:, None, None] & odd] += 1e6
    s = ctx.compress(torch.from_numpy(f.astype(dtype)).cuda(), eb=1e-3, eb_mode="abs", bound_mode="reference",
                     chunk_high=high, chunk_low=low)
    full = po.decompress(s.to_bytes())
    ctx.upload(s)
    nz, ny, nx = dims
    c = 2 * high  # field planes of a chunk
    ends = {(0, 0), (0, nz - 1), (nz - 1, nz - 1), (nz // 2, nz // 2), (c - 1, c), (c, c + 1), (c - 2, c - 2),
            (1, c - 2), (c // 2 + 1, nz - 2), (c + 3, c + 4)}
    boxes = [((x0, 2, z0), (nx - 1 - x0, ny - 3, z1)) for x0 in (0, 5) for z0, z1 in sorted(ends)]
    fx, fy = min(c, nx // 2), min(c, ny // 2)
    boxes += [((fx - 1, fy - 1, c - 1), (fx, fy, c)), ((fx - 1, 0, 0), (fx + 2, 3, 4)), ((0, fy - 1, 1), (3, fy - 1, 5))]
    want = [full[lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1] for lo, hi in boxes]
    for (lo, hi), w in zip(boxes, want):
        assert np.array_equal(_bits(ctx.decompress_box(s, lo, hi)), _bits(w)), (lo, hi)
    srv = Server(0, arena_bytes=2 << 30, max_batch=32)
    try:
        sid = srv.add_stream(s)
        for whole in (False, True, False):  # cold buffers; then a whole decode in the batch; then what it left
            order = rng.permutation(len(boxes))
            extra = [srv.submit_level(sid, s.info().n_levels)] if whole else []
            tickets = [srv.submit_box(sid, *boxes[i]) for i in order]
            for i, t in zip(order, tickets):
                assert np.array_equal(_bits(srv.copy_out(srv.wait(t), dtype)), _bits(want[i])), boxes[i]
            for t in extra:
                srv.wait(t)
            for t in tickets + extra:
                srv.release(t)
    finally:
        srv.close()
