"""The windows of a shared-matrix batch between checks replay one captured graph: a second
window costs what a fourth does, without another capture (0.1 to 0.25 ms). And one result for any number of windows, of any parity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(engine, instances, every, iterations, timed=False):
    inst = instances.lp_uniform(3, 2000, 4000, 3)
    A, count = engine.Matrix.from_instance(inst), 8
    cl, cu = np.repeat(inst["cl"][None], count, 0), np.repeat(inst["cu"][None], count, 0)
    cu[:, 3] = np.arange(count) % 5
    s = engine.batch_default_settings()
    s.max_iterations, s.check_every, s.primal_tol, s.dual_tol, s.schedule = iterations, every, 1e-300, 1e-300, 2
    engine.set_timing(1)
    try:
        best = np.inf
        for _ in range(12 if timed else 1):
            rc, x, y, res = engine.shared_batch_pdhg(A, count, inst["c"], inst["rl"], inst["ru"], cl, cu, s, want_dual=True)
            assert rc == 0, engine.last_error()
            best = min(best, engine.last_timing()["loop_ms"])
    finally:
        engine.set_timing(0)
    return best, x, y, res


def test_a_second_window_needs_no_second_graph(engine, instances):
    one, two, three, four = (batch(engine, instances, 60, 60 * k, timed=True)[0] for k in (1, 2, 3, 4))
    second, fourth = two - one, four - three
    assert second - fourth < 0.06, (one, two, three, four)


@pytest.mark.parametrize("every", [1, 2, 3, 7, 64, 65, 130])
def test_windows_of_any_length_give_the_same_point(engine, instances, every):
    _, x, y, res = batch(engine, instances, every, 131)
    _, x2, y2, res2 = batch(engine, instances, 131, 131)
    assert np.array_equal(x, x2) and np.array_equal(y, y2)
    assert res == res2   # the last check is at 131 in both, with the dual step of that iteration


def test_few_lps_with_a_dense_row_gather_far_ahead(engine):
    """Up to 64 LPs the first schedule has 8 entries of a row in flight: a row with most of
    the columns is a chain of gathers (4,000 of 8,000 columns, 31 LPs: 235 us against 431 with three in
    flight, 387 with six).
    The points of all schedules are the same."""
    rng, m, n, count = np.random.default_rng(5), 2000, 4000, 31
    ptr, idx = [0], []
    for i in range(m):
        idx.append(np.sort(rng.choice(n, 3500 if i == 7 else 3, replace=False)))
        ptr.append(ptr[-1] + len(idx[-1]))
    idx = np.concatenate(idx).astype(np.int32)
    A = engine.Matrix(m, n, ptr, idx, rng.uniform(0.1, 1, len(idx)))
    cl, cu = np.zeros((count, n)), np.full((count, n), 10.0)
    cu[:, 0] = np.arange(count) % 7
    c, rl, ru = rng.normal(size=n), np.full(m, -1e30), rng.uniform(1, 5, m)
    ms, points = {}, {}
    engine.set_timing(1)
    try:
        for schedule in (1, 2, 3) * 3:
            s = engine.batch_default_settings()
            s.max_iterations, s.check_every, s.primal_tol, s.dual_tol, s.schedule = 60, 60, 1e-300, 1e-300, schedule
            rc, x, y, _ = engine.shared_batch_pdhg(A, count, c, rl, ru, cl, cu, s, want_dual=True)
            assert rc == 0, engine.last_error()
            ms[schedule] = min(ms.get(schedule, np.inf), engine.last_timing()["loop_ms"])
            points[schedule] = (x, y)
    finally:
        engine.set_timing(0)
    for schedule in (2, 3):
        assert all(np.array_equal(a, b) for a, b in zip(points[1], points[schedule]))
    assert ms[1] < 0.75 * ms[3], ms
