"""The scaling's row and column maxima at the edges of their chunks: no entries, one, rows of
32 / 33 (owner lane, whole warp) and 256 / 257 (a chunk, a streamed row). A maximum does not
depend on the order, so the factors equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,lens", [(1, 1, [1]), (40, 31, [0, 1, 31]), (70, 300, [32, 33, 0]), (64, 700, [256, 257, 300, 5]),
                                      (700, 64, [3]), (5000, 3000, [1, 40, 0, 7])])
def test_ruiz_bit_exact_at_chunk_edges(engine, oracle, instances, m, n, lens):
    rng = np.random.default_rng(4)
    deg = np.minimum(np.resize(np.asarray(lens), m), n)
    row = np.repeat(np.arange(m), deg)
    col = np.concatenate([rng.choice(n, size=k, replace=False) for k in deg]).astype(int)
    ptr, idx, val = instances._csr_from_entries(m, row, col, rng.standard_normal(col.shape[0]) * 10.0 ** rng.uniform(-3, 3, col.shape[0]))
    inst = instances._finish_lp(rng, m, n, ptr, idx, val)
    rc, r, c = engine.scale_factors(engine.Matrix.from_instance(inst), engine.SCALE_RUIZ, 30, 1e-3)
    ro, co, conv = oracle.ruiz(inst, 30, 1e-3)
    assert rc == 0
    assert np.array_equal(r, ro) and np.array_equal(c, co)
