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
        assert rc != 0 and "gave up" in engine.last_error()
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


def loop_call(engine, oracle, inst, limit, time_limit=0.0, tol=1e-300):
    """The C core's loop; returns a function for fails_then_works."""
    import ctypes as C
    keep = oracle._Keep()
    model = oracle.build_sk_model(keep, inst, False)

    def call():
        opts = oracle.SkOptions(primal_tol=tol, dual_tol=tol, iteration_limit=limit, threads=1, time_limit=time_limit)
        x, y, act = np.zeros(inst["n"]), np.zeros(inst["m"]), np.zeros(inst["m"])
        res = engine.LoopResult()
        rc = engine.lib().sankhya_b200_pdhg_loop(C.byref(model), C.byref(opts), engine._p(x), engine._p(y),
                                                 engine._p(act), C.byref(res))
        return rc, (x, y, act, res.iterations, res.dual_step, keep is None)
    return call


def fixed_call(engine, inst):
    A = engine.Matrix.from_instance(inst)
    kw = dict(max_iterations=100, check_every=40, tau=0.05, sigma=0.05, tolerance=1e-300)
    return lambda: (lambda rc, x, _, r: (rc, (x, r["objective"])))(*engine.pdhg(A, inst, engine.settings(**kw)))


def pdlp_call(engine, inst, **kw):
    A = engine.Matrix.from_instance(inst)
    s = engine.pdlp_default_settings()
    s.max_iterations, s.eps_optimal, s.ruiz_iterations = 150, 1e-300, 5
    for k, v in kw.items():
        setattr(s, k, v)
    return lambda: (lambda rc, x, y, r: (rc, (x, y)))(*engine.pdlp_solve(A, inst, s))


def solve_call(engine, oracle, inst, entry):
    if entry == "fixed":
        return fixed_call(engine, inst)
    if entry == "loop":
        return loop_call(engine, oracle, inst, 100)
    if entry == "halpern":
        return pdlp_call(engine, inst, algorithm=engine.PDLP_HALPERN)
    return pdlp_call(engine, inst, precision=getattr(engine, entry))


ENTRIES = ["fixed", "loop", "halpern", "FP64", "FP32_REFINE", "BF16_REFINE"]


@pytest.mark.parametrize("entry", ENTRIES)
def test_cooperative_launch(engine, oracle, instances, entry):
    fails_then_works(engine, solve_call(engine, oracle, instances.lp_uniform(6, 8000, 16000, 8), entry))


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("shape", [(40, 31, 3), (2000, 5000, 5)], ids=str)
def test_cluster(engine, oracle, instances, shape, entry):
    fails_then_works(engine, solve_call(engine, oracle, instances.lp_uniform(7, *shape), entry))
