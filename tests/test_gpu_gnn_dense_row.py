"""A row with most of the columns: one warp walks it in each aggregation, and the backward
one, which goes through a relu as well, takes hardly longer per entry than the forward one."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def least(call, n=8):
    times = []
    for _ in range(n):
        start = time.perf_counter()
        call()
        times.append(time.perf_counter() - start)
    return min(times)


def test_gradient_against_prediction(engine, instances):
    """The gradient is the forward aggregations and as many backward, which also gather the
    entries' scales: 2.5 times the prediction, 3.0 with a slower chain."""
    rng = np.random.default_rng(1)
    m, n, dense = 9154, 28801, 20000
    key = np.unique(np.concatenate([rng.integers(0, m, 4 * n) * n + np.repeat(np.arange(n), 4),
                                    (m // 2) * n + rng.choice(n, dense, replace=False)]))
    ptr, idx, val = instances._csr_from_entries(m, key // n, key % n, rng.standard_normal(key.shape[0]))
    inst = instances._finish_lp(rng, m, n, ptr, idx, val)
    A, net = engine.Matrix.from_instance(inst), engine.Gnn(seed=1)
    xt, yt = np.zeros(n), np.zeros(m)
    predict, gradient = least(lambda: net.predict(A, inst)), least(lambda: net.gradient(A, inst, xt, yt))
    assert gradient < 2.75 * predict, (predict, gradient)
