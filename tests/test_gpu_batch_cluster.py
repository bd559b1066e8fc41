"""A batch on clusters (each LP by one CTA or by a whole cluster) against the same LPs on the
launches over the whole batch. An LP whose vectors no CTA holds puts its batch on the launches;
every row is summed in the same order on both, so the other LPs' results are equal bit for bit.
The LPs are the edges: no rows, no columns, one entry, rows of 32 / 33 / 256 / 257 entries, chunks
that hold rows of several LPs, LPs of more and of fewer chunks than a CTA has warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def one(instances, rng, m, n, lens):
    deg = np.minimum(np.resize(np.asarray(lens), m), n)
    row = np.repeat(np.arange(m), deg)
    col = np.concatenate([rng.choice(n, size=k, replace=False) for k in deg] or [np.zeros(0, int)]).astype(int)
    ptr, idx, val = instances._csr_from_entries(m, row, col, rng.standard_normal(col.shape[0]))
    return instances._finish_lp(rng, m, n, ptr, idx, val)


def empty(rng, m, n):
    return dict(m=m, n=n, ptr=np.zeros(m + 1, np.int32), idx=np.zeros(0, np.int32), val=np.zeros(0), c=rng.standard_normal(n),
                rl=-rng.random(m), ru=rng.random(m), cl=np.zeros(n), cu=np.ones(n))


def solve(engine, lps, **kw):
    blk, rseg, cseg = engine.block_diagonal(lps)
    s = engine.batch_default_settings()
    for k, v in kw.items():
        setattr(s, k, v)
    engine.set_timing(1)
    try:
        rc, x, y, res = engine.batch_pdhg(engine.Matrix.from_instance(blk), blk, rseg, cseg, s, want_dual=True)
        launches = engine.last_timing()["kernel_launches"]
    finally:
        engine.set_timing(0)
    assert rc == 0, engine.last_error()
    return x, y, res, launches, rseg, cseg


@pytest.mark.parametrize("kind", ["edges", "pairs"])
@pytest.mark.parametrize("limit,every,tol,seconds", [(61, 20, 1e-13, 0.0), (5000, 7, 2e-2, 0.0), (60, 20, 1e-3, 1e9)])
def test_clusters_equal_launches(engine, instances, kind, limit, every, tol, seconds):
    rng = np.random.default_rng(11)
    if kind == "edges":
        lps = [one(instances, rng, m, n, lens) for m, n, lens in
               [(1, 1, [1]), (3, 2, [0, 2, 1]), (40, 31, [0, 1, 31]), (70, 300, [32, 33, 0]), (64, 700, [256, 257, 300, 5]),
                (7, 900, [3]), (800, 5, [2, 0, 1]), (1200, 900, [1, 4, 3])]]
        lps[2:2] = [empty(rng, 0, 5), empty(rng, 4, 0), empty(rng, 37, 33)]
    else:   # many LPs and a few large ones: these by whole clusters
        lps = [one(instances, rng, 300, 600, [12, 3, 21]) for _ in range(190)]
        lps[7:7] = [one(instances, rng, 1500, 3001, [12, 40, 0, 5]) for _ in range(10)]
    kw = dict(max_iterations=limit, check_every=every, primal_tol=tol, dual_tol=tol, time_limit=seconds)
    x, y, res, launches, rseg, cseg = solve(engine, lps, **kw)
    huge = empty(rng, 20000, 9000)
    x2, y2, res2, launches2, _, _ = solve(engine, lps + [huge], **kw)
    assert launches < 2 * res[0]["iterations"] <= launches2   # on clusters, and not
    assert np.array_equal(x, x2[:cseg[-1]]) and np.array_equal(y, y2[:rseg[-1]])
    for a, b in zip(res, res2):
        assert a == b
