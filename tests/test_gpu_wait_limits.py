"""A wait inside an iteration kernel that gives up ends the call with an error, and the next
call is as any other. The limit of 0 polls lets every wait fail at once although what it waits
for is on its way, so nothing hangs and nothing is read that was not written."""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

spec = importlib.util.spec_from_file_location("batch_shapes", os.path.join(os.path.dirname(__file__), "test_gpu_batch_cluster.py"))
shapes = importlib.util.module_from_spec(spec)
spec.loader.exec_module(shapes)


def fails_then_works(engine, call):
    """call() -> (rc, outputs): right before and after, an error with a limit of 0."""
    rc, before = call()
    assert rc == 0, engine.last_error()
    engine.set_wait_limit(0)
    try:
        rc, _ = call()
        assert rc == -1 and "gave up" in engine.last_error()
    finally:
        engine.set_wait_limit(-1)
    rc, after = call()
    assert rc == 0, engine.last_error()
    for a, b in zip(before, after):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind", ["ctas", "clusters"])
def test_batch_on_ctas(engine, instances, kind):
    """Rows of up to 300 entries: a row beyond a chunk takes no copy, its neighbours do."""
    rng = np.random.default_rng(4)
    lps = [shapes.one(instances, rng, 300, 600, [12, 3, 21, 300]) for _ in range(190)]
    if kind == "clusters":
        lps[7:7] = [shapes.one(instances, rng, 1500, 3001, [12, 40, 0, 5]) for _ in range(10)]
    blk, rseg, cseg = engine.block_diagonal(lps)
    A = engine.Matrix.from_instance(blk)
    s = engine.batch_default_settings()
    s.max_iterations, s.primal_tol, s.dual_tol = 61, 1e-13, 1e-13

    def call():
        rc, x, y, _ = engine.batch_pdhg(A, blk, rseg, cseg, s, want_dual=True)
        return rc, (x, y)
    fails_then_works(engine, call)
