"""An MMA wait of the learned network that gave up (its error word set from
the host): compress returns the error before any coder kernel is launched,
since the failed level's codes are not all written, and the context goes on to
give the oracle's bytes; decompress returns the error too."""
import numpy as np
import pytest

import pyoracle as po
import stz_b200
from conftest import model_file, random_model

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CODER = ("k_run_stats", "k_codebook", "k_sub_bits", "k_scan_stream", "k_encode", "k_pack_streams", "k_unpred_move")


@pytest.mark.parametrize("flags", [0x7F7F, -1])  # forced, and chosen by the sampled estimate
def test_compress_stops_before_the_coder(flags):
    from stz_b200 import fields

    f = torch.from_numpy(fields.grf((64, 64, 128), 11.0 / 3.0, 31, np.float32)).cuda()
    rng = np.random.default_rng(5)
    recs = (random_model(rng), random_model(rng))
    model = stz_b200.Model.from_bytes(model_file(recs))
    kw = dict(eb=1e-3, eb_mode="rel", chunk_high=16, chunk_low=8)
    with stz_b200.Context(0) as ctx:
        want = ctx.compress(f, model=model, learned_flags=flags, **kw).to_bytes()
        plain = ctx.compress(f, **kw).to_bytes()
        ctx.profile_reset()
        stz_b200._check(ctx.lib.stz_debug_learned_fail(ctx._c))
        with pytest.raises(stz_b200.StzError, match="did not complete in time"):
            ctx.compress(f, model=model, learned_flags=flags, **kw)
        n = {k: v[1] for k, v in ctx.profile_read().items()}
        assert sum(v for k, v in n.items() if k.startswith("k_level_encode")) > 0
        assert not any(n.get(k, 0) for k in CODER), n
        # whatever the failed call had queued, the next calls' results are theirs
        s = ctx.parse(want)
        out = ctx.decompress(s)
        assert np.array_equal(out.view(np.uint32), po.decompress(want).view(np.uint32))
        assert ctx.compress(f, **kw).to_bytes() == plain
        assert ctx.compress(f, model=model, learned_flags=flags, **kw).to_bytes() == want
        if s.info().learned_flags:
            stz_b200._check(ctx.lib.stz_debug_learned_fail(ctx._c))
            with pytest.raises(stz_b200.StzError, match="did not complete in time"):
                ctx.decompress(s)
            assert np.array_equal(ctx.decompress(s).view(np.uint32), out.view(np.uint32))
