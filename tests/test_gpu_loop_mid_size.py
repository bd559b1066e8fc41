"""The C core's loop at a size that takes the cooperative launch, whose last dual step comes
from one partial per thread block: every row and column has at most 32 entries, so the
iterates are the oracle's bit for bit, at checkpoints, at a limit between two and with a time
limit (which the host looks at between launches)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit,seconds", [(40, 0.0), (61, 0.0), (61, 1e6)])
def test_loop_equals_the_oracle(engine, oracle, instances, limit, seconds):
    inst = instances.lp_uniform(21, 12000, 20000, 3)
    assert max(np.diff(inst["ptr"]).max(), np.bincount(inst["idx"]).max()) <= 32
    x2, y2, act2, out2 = oracle.sk_loop(inst, limit, 1e-300, 1e-300)
    keep = oracle._Keep()
    model = oracle.build_sk_model(keep, inst, False)
    opts = oracle.SkOptions(primal_tol=1e-300, dual_tol=1e-300, iteration_limit=limit, threads=1, time_limit=seconds)
    x, y, act = np.zeros(inst["n"]), np.zeros(inst["m"]), np.zeros(inst["m"])
    res = engine.LoopResult()
    assert engine.lib().sankhya_b200_pdhg_loop(C.byref(model), C.byref(opts), engine._p(x), engine._p(y), engine._p(act),
                                               C.byref(res)) == 0, engine.last_error()
    assert engine.last_timing()["kernel_launches"] == (limit + 19) // 20   # a window each; checks are not counted
    assert res.iterations == out2["iterations"] == limit
    assert np.array_equal(x, x2) and np.array_equal(y, y2) and np.array_equal(act, act2)
    assert res.dual_step == out2["dual_step"]
