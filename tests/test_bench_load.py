"""bench.py's serving load, against a fake server: no collection of Python's
stops the producer while the load runs, and the collector is on again after a
run, an error and an exception."""
import gc
import types

import pytest

import bench


class FakeServer:
    def __init__(self, fail=None):
        self.fail, self.enabled, self.n = fail, [], 0

    def submit_box(self, sid, lo, hi):
        self.enabled.append(gc.isenabled())
        self.n += 1
        return self.n

    def wait(self, t):
        self.enabled.append(gc.isenabled())
        if self.fail == "raise" and t == 5:
            raise RuntimeError("wait")
        return types.SimpleNamespace(status=1 if self.fail == "status" and t == 5 else 0, latency_ms=1.0, queue_ms=0.5,
                                     batch=t, batch_size=1, nbytes=4)

    def release(self, t):
        pass


@pytest.mark.parametrize("fail", [None, "status", "raise"])
def test_no_collection_during_a_load(fail):
    srv = FakeServer(fail)
    gen = lambda rng: ("box", [0, 0, 0], [1, 1, 1])
    assert gc.isenabled()
    if fail == "raise":
        with pytest.raises(RuntimeError):
            bench.serve_load(srv, 0, (8, 8, 8), 2, 1000, 0.05, gen, 1)
    else:
        out = bench.serve_load(srv, 0, (8, 8, 8), 2, 1000, 0.05, gen, 1)
        assert ("error" in out) == (fail is not None)
        if not fail:
            assert out["requests"] == 50 and out["p99_ms"] == 1.0
    assert gc.isenabled()
    assert srv.enabled and not any(srv.enabled)
