"""Iterations of a small LP on one thread-block cluster, and of a mid-size one in one
cooperative launch, against the two fused launches per iteration (the path that per-kernel
timing, level 2, takes). Both sum every row in the same
order and use the same elementwise arithmetic, so their iterates are equal bit for bit; where
every row has at most 32 entries they equal the oracle's serial sums too (tests/test_gpu_parity.py
runs config 0 there). The shapes are the edges: one entry, empty rows and columns, rows of 32 /
33 / 256 / 257 entries (owner, warp tree, streamed), fewer chunks than CTAs, chunk counts at and
above the cluster's 256, more chunks than the cooperative launch has warps, and long rows there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lp(instances, m, n, lens, seed=0):
    """Row i has lens[i % len(lens)] entries in distinct random columns."""
    rng = np.random.default_rng(seed)
    deg = np.minimum(np.resize(np.asarray(lens), m), n)
    row = np.repeat(np.arange(m), deg)
    col = np.concatenate([rng.choice(n, size=k, replace=False) for k in deg] or [np.zeros(0, int)])
    val = rng.standard_normal(col.shape[0])
    ptr, idx, val = instances._csr_from_entries(m, row, col, val)
    return instances._finish_lp(rng, m, n, ptr, idx, val)


def steps(inst):
    rows = np.repeat(np.arange(inst["m"]), np.diff(inst["ptr"]))
    rm = np.bincount(rows, np.abs(inst["val"]), inst["m"])
    cm = np.bincount(inst["idx"], np.abs(inst["val"]), inst["n"])
    return 0.9 / (1 + cm), 0.9 / (1 + rm)


def scaled_steps(engine, **kw):
    s = engine.pdlp_default_settings()
    s.eps_optimal, s.ruiz_iterations = 1e-14, 10
    for k, v in kw.items():
        setattr(s, k, v)
    return s


SHAPES = [
    (1, 1, [1]), (3, 2, [0, 2, 1]), (40, 31, [0, 1, 31]), (257, 300, [32, 33, 0]), (64, 700, [256, 257, 300, 5]),
    (1200, 900, [1, 40, 3]), (15, 6000, [9]), (6000, 15, [2]), (4000, 9000, [7, 3, 11]), (9000, 17500, [4]),
    (9000, 20500, [4]), (8192, 8192, [1]), (8193, 5000, [6]), (500, 7000, [300, 12, 0, 64]), (42000, 30000, [5, 17, 0, 9]),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("entry", ["lp", "with_dual", "diagonal"])
def test_cluster_equals_launches(engine, instances, shape, entry):
    inst = lp(instances, *shape)
    ps, ds = steps(inst)
    kw = dict(max_iterations=47, check_every=19, theta=0.5 if entry == "with_dual" else 1.0, tolerance=1e-13)
    extra = {}
    if entry == "with_dual":
        extra = dict(primal_steps=ps, dual_steps=ds, want_dual=True)
    else:
        norm = np.sqrt(max((0.9 / ps - 1).max() * (0.9 / ds - 1).max(), 1e-3))
        kw.update(tau=0.9 / norm, sigma=0.9 / norm)
    if entry == "diagonal":
        extra = dict(qdiag=np.random.default_rng(3).uniform(0, 2, inst["n"]))
    A = engine.Matrix.from_instance(inst)
    got = []
    for level in (0, 2):
        engine.set_timing(level)
        try:
            rc, x, y, r = engine.pdhg(A, inst, engine.settings(**kw), **extra)
        finally:
            engine.set_timing(0)
        assert rc == 0
        got.append((x, y, r))
    assert np.array_equal(got[0][0], got[1][0])
    if got[0][1] is not None:
        assert np.array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2]


@pytest.mark.parametrize("check_every,limit", [(1, 300), (7, 9001), (4096, 8193), (4097, 8195)])
@pytest.mark.parametrize("tolerance", [0.3, 1e-3, 1e-300])
def test_checkpoints_in_the_kernel_equal_the_hosts(engine, instances, check_every, limit, tolerance):
    """Without a time limit a cluster judges its checkpoints itself, over launches of 4096
    iterations at most; a limit that never runs out leaves them to the host. The same
    residuals and the same stop, bit for bit."""
    inst = lp(instances, 257, 300, [3, 5, 0], seed=2)
    A = engine.Matrix.from_instance(inst)
    ps, ds = steps(inst)
    norm = np.sqrt((0.9 / ps - 1).max() * (0.9 / ds - 1).max())
    got = []
    for seconds in (0.0, 1e9):
        rc, x, _, r = engine.pdhg(A, inst, engine.settings(max_iterations=limit, check_every=check_every, tau=0.9 / norm,
                                                           sigma=0.9 / norm, tolerance=tolerance, time_limit=seconds))
        assert rc == 0
        got.append((x, r))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1] == got[1][1]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE", "BF16_REFINE"])
def test_adaptive_cluster_equals_launches(engine, instances, shape, precision):
    """A QP whose diagonal Hessian is zero is the same LP on the launches: x - tau g over
    1 + tau 0 = 1, so every step and every decision has the same bits (only the objective's
    sums are formed differently). 150 iterations: windows of 64 and a tail of 22."""
    inst = lp(instances, *shape, seed=5)
    s = scaled_steps(engine, max_iterations=150, precision=getattr(engine, precision))
    A = engine.Matrix.from_instance(inst)
    rc, x, y, r = engine.pdlp_solve(A, inst, s)
    rc2, x2, y2, r2 = engine.pdlp_solve_qp(A, inst, s, qdiag=np.zeros(inst["n"]))
    assert rc == rc2 == 0
    assert np.array_equal(x, x2) and np.array_equal(y, y2)
    for k in ("iterations", "restarts", "rejected_steps", "final_step_size", "primal_weight"):
        assert r[k] == r2[k], k


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_halpern_cluster_equals_numpy(engine, instances, shape):
    """64 anchored steps and T(z), the point the window's restart takes, against numpy FP64
    without scaling. The anchored iteration is non-expansive, so a step's rounding (a few
    ulps over rows of up to 300 entries) adds up at most linearly: 64 x 300 x 2^-52 = 4e-12
    of the largest entry."""
    inst = lp(instances, *shape, seed=9)
    s = scaled_steps(engine, max_iterations=64, scaling=0, algorithm=engine.PDLP_HALPERN, initial_primal_weight=1.0)
    rc, x, y, r = engine.pdlp_solve(engine.Matrix.from_instance(inst), inst, s)
    assert rc == 0 and r["iterations"] == 64
    import scipy.sparse as sp
    A = sp.csr_matrix((inst["val"], inst["idx"], inst["ptr"]), shape=(inst["m"], inst["n"]))
    eta = 0.9 / r["matrix_norm"]
    clip = lambda v, lo, hi: np.minimum(np.maximum(v, lo), hi)
    u, v = np.zeros(inst["n"]), np.zeros(inst["m"])
    for k in range(65):
        xp = clip(u - eta * (inst["c"] + A.T @ v), inst["cl"], inst["cu"])
        w = v + eta * (A @ (2 * xp - u))
        yp = w - eta * clip(w / eta, inst["rl"], inst["ru"])
        if k == 64:
            break
        lam = (k + 1.0) / (k + 2.0)
        u, v = lam * (2 * xp - u), lam * (2 * yp - v)
    if r["restarts"] == 0:
        xp, yp = u, v
    assert np.abs(x - xp).max() <= 4e-12 * max(1.0, np.abs(xp).max())
    assert np.abs(y - yp).max() <= 4e-12 * max(1.0, np.abs(yp).max())
