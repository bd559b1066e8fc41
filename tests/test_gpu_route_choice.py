"""Which path a solve takes, seen by the launches it reports, at the edges of the rules that
choose it; and that products of a mid-size matrix are not slower than a larger one's."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def lp_with_row(instances, m, n, per_col, row_len=0, seed=0):
    """Uniform columns, and row m // 2 with row_len further entries."""
    rng = np.random.default_rng(seed)
    col = np.repeat(np.arange(n), per_col)
    row = rng.integers(0, m, n * per_col)
    if row_len:
        col = np.concatenate([col, rng.choice(n, row_len, replace=False)])
        row = np.concatenate([row, np.full(row_len, m // 2)])
    key = np.unique(row.astype(np.int64) * n + col)
    ptr, idx, val = instances._csr_from_entries(m, key // n, key % n, rng.standard_normal(key.shape[0]))
    return instances._finish_lp(rng, m, n, ptr, idx, val)


def pair_us(engine, A, n, m):
    """Least time of A x and A'y by turns."""
    x, y = torch.randn(n, dtype=torch.float64, device="cuda"), torch.randn(m, dtype=torch.float64, device="cuda")
    x2, y2, L, h = torch.empty_like(x), torch.empty_like(y), engine.lib(), C.byref(A.handle)
    best = np.inf
    for _ in range(12):
        torch.cuda.synchronize()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        for _ in range(100):
            assert L.sankhya_cuda_spmv_device_f64(h, x.data_ptr(), y2.data_ptr()) == 0
            assert L.sankhya_cuda_spmv_transpose_device_f64(h, y.data_ptr(), x2.data_ptr()) == 0
        t1.record()
        torch.cuda.synchronize()
        best = min(best, t0.elapsed_time(t1) * 10)
    return best


def test_products_of_a_mid_size_matrix_are_not_slower_than_a_larger_ones(engine, instances):
    """Four sizes of 60 to 260 thread blocks a product against one of 340 (they took twice its
    time when the next product's blocks were let in as each began)."""
    larger = lp_with_row(instances, 40000, 70000, 10)
    limit = 1.3 * pair_us(engine, engine.Matrix.from_instance(larger), 70000, 40000)
    for m, n, per_col in [(8000, 16000, 8), (15000, 30000, 8), (25000, 45000, 8), (30000, 65000, 8)]:
        inst = lp_with_row(instances, m, n, per_col)
        assert pair_us(engine, engine.Matrix.from_instance(inst), n, m) < limit, (m, n)


def rows_of(instances, m, n, short, longer, share, seed=0):
    """Rows of `short` entries, a share of them of `longer`."""
    rng = np.random.default_rng(seed)
    deg = np.where(rng.random(m) < share, longer, short)
    key = np.unique(np.repeat(np.arange(m), deg).astype(np.int64) * n + rng.integers(0, n, deg.sum()))
    ptr, idx, val = instances._csr_from_entries(m, key // n, key % n, rng.standard_normal(key.shape[0]))
    return instances._finish_lp(rng, m, n, ptr, idx, val)


def transposed(instances, inst):
    rows = np.repeat(np.arange(inst["m"]), np.diff(inst["ptr"]))
    ptr, idx, val = instances._csr_from_entries(inst["n"], inst["idx"], rows, inst["val"])
    return instances._finish_lp(np.random.default_rng(0), inst["n"], inst["m"], ptr, idx, val)


def launches_of(engine, inst, iterations, **kw):
    A = engine.Matrix.from_instance(inst)
    engine.set_timing(1)
    try:
        rc, *_ = engine.pdhg(A, inst, engine.settings(max_iterations=iterations, check_every=iterations, tau=1e-3, sigma=1e-3,
                                                      tolerance=1e-300, **kw))
        assert rc == 0, engine.last_error()
        return engine.last_timing()["kernel_launches"]
    finally:
        engine.set_timing(0)


# (cooperative launch or not, instance): where it loses time, the launches stay
SIZES = {
    "mid-size": (True, lambda i: lp_with_row(i, 8000, 16000, 8)),
    "a row of 700": (True, lambda i: lp_with_row(i, 8000, 16000, 8, 700)),
    "a dense row": (False, lambda i: lp_with_row(i, 20000, 40000, 5, 40000)),
    "half in rows of 60, light ones beside": (True, lambda i: rows_of(i, 90000, 50000, 2, 60, 0.04)),
    "half in columns of 60, light ones beside": (True, lambda i: transposed(i, rows_of(i, 90000, 50000, 2, 60, 0.04))),
    "two rounds of light rows": (False, lambda i: rows_of(i, 150000, 40000, 1, 36, 0.04)),
    "four fifths in rows of 40": (False, lambda i: rows_of(i, 76000, 30000, 1, 40, 0.1)),
    "light rows and columns, two thirds in rows of 100": (False, lambda i: rows_of(i, 100000, 80000, 1, 100, 0.02)),
    "long rows beside two rounds of columns": (False, lambda i: lp_with_row(i, 15000, 90000, 5)),
    "a few long rows beside two rounds of columns": (True, lambda i: lp_with_row(i, 25000, 100000, 5)),
    "a dense row, 5,000 x 12,000": (False, lambda i: lp_with_row(i, 5000, 12000, 5, 12000)),
    "one chunk a warp, rows of 45": (True, lambda i: lp_with_row(i, 12000, 27000, 20)),
    "two chunks a warp, rows of 40": (False, lambda i: rows_of(i, 40000, 60000, 6, 40, 0.4)),
    "a fifth in rows of 100": (True, lambda i: rows_of(i, 100000, 100000, 8, 100, 0.02)),
    "most elements": (True, lambda i: lp_with_row(i, 250000, 300000, 4)),
    "too many elements": (False, lambda i: lp_with_row(i, 300000, 500000, 3)),
    "wide, 120 a row": (True, lambda i: lp_with_row(i, 800, 24000, 4)),
    "wide, 400 a row": (False, lambda i: lp_with_row(i, 800, 80000, 4)),
    "wide, 250 a row": (False, lambda i: lp_with_row(i, 1200, 75000, 4)),
    "tall, 180 a column": (False, lambda i: transposed(i, lp_with_row(i, 2000, 90000, 4))),
    "a quarter in rows of 400": (True, lambda i: rows_of(i, 20000, 30000, 10, 400, 0.007)),
    "half in rows of 400": (False, lambda i: rows_of(i, 20000, 30000, 6, 400, 0.018)),
    "a fifth in rows beyond 32, many elements": (False, lambda i: rows_of(i, 150000, 200000, 6, 40, 0.05)),
}


@pytest.mark.parametrize("name", SIZES)
def test_cooperative_launch_where_it_pays(engine, instances, name):
    cooperative, make = SIZES[name]
    launches = launches_of(engine, make(instances), 60)
    assert launches < 60 if cooperative else launches >= 120


@pytest.mark.parametrize("m,n,per_col,every,limit,one_launch_a_window", [
    (2000, 5000, 5, 3, 1e6, False), (2000, 5000, 5, 4, 1e6, True), (2000, 5000, 5, 3, 0.0, True),
    (130000, 180000, 4, 9, 0.0, False), (130000, 180000, 4, 10, 0.0, True), (100000, 150000, 4, 1, 0.0, True)])
def test_short_windows_stay_on_the_launches(engine, instances, m, n, per_col, every, limit, one_launch_a_window):
    """Iterations between checkpoints that the host judges; the same point either way."""
    inst = lp_with_row(instances, m, n, per_col)
    A = engine.Matrix.from_instance(inst)
    got = []
    for level in (1, 2):
        engine.set_timing(level)
        try:
            rc, x, _, r = engine.pdhg(A, inst, engine.settings(max_iterations=5 * every, check_every=every, tau=1e-3, sigma=1e-3,
                                                               tolerance=1e-300, time_limit=limit))
            assert rc == 0, engine.last_error()
            got.append((x, r, engine.last_timing()["kernel_launches"]))
        finally:
            engine.set_timing(0)
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]
    checks = 5 * 4   # launches of the checkpoints the host judges
    assert got[0][2] <= checks + 5 if one_launch_a_window else got[0][2] == checks + 2 * 5 * every


def test_a_solve_of_few_iterations_is_a_short_window(engine, instances):
    inst = lp_with_row(instances, 2000, 5000, 5)
    A = engine.Matrix.from_instance(inst)
    engine.set_timing(1)
    try:
        for iterations, launches in ((3, 6), (4, 1)):
            rc, *_ = engine.pdhg(A, inst, engine.settings(max_iterations=iterations, check_every=100, tau=1e-3, sigma=1e-3,
                                                          tolerance=1e-300, time_limit=1e6))
            assert rc == 0 and engine.last_timing()["kernel_launches"] == launches + 4
    finally:
        engine.set_timing(0)


def test_anchored_windows_of_one_iteration_stay_on_the_launches(engine, instances):
    inst = lp_with_row(instances, 200, 300, 3)
    A = engine.Matrix.from_instance(inst)
    launches = []
    for period in (1, 2):
        s = engine.pdlp_default_settings()
        s.max_iterations, s.restart_period, s.algorithm, s.eps_optimal = 20 * period, period, engine.PDLP_HALPERN, 1e-300
        rc, *_ = engine.pdlp_solve(A, inst, s)
        assert rc == 0, engine.last_error()
        launches.append(engine.last_timing()["kernel_launches"])
    assert launches[0] > launches[1]   # two launches an iteration, then one a window; 20 windows each


@pytest.mark.parametrize("count,m,every,on_ctas", [(512, 30, 20, False), (512, 30, 100, False), (40, 60, 20, True),
                                                   (300, 60, 20, True), (300, 250, 20, True), (296, 500, 20, True)])
def test_batches_of_small_lps(engine, instances, count, m, every, on_ctas):
    """Several tiny LPs a CTA take longer than two launches over all of them."""
    lps = [lp_with_row(instances, m, 2 * m, 4, seed=k) for k in range(count)]
    blk, rseg, cseg = engine.block_diagonal(lps)
    s = engine.batch_default_settings()
    s.max_iterations, s.check_every, s.primal_tol, s.dual_tol = 100, every, 1e-300, 1e-300
    engine.set_timing(1)
    try:
        rc, *_ = engine.batch_pdhg(engine.Matrix.from_instance(blk), blk, rseg, cseg, s)
        assert rc == 0 and (engine.last_timing()["kernel_launches"] < 100) == on_ctas
    finally:
        engine.set_timing(0)
