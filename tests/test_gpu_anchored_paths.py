"""The anchored (Halpern) iteration on a cluster, in one cooperative launch and on the launches
gives the same bits. Rows without entries or bounds move an LP from path to path (their chunks
fill the cluster, and 700,000 of them are too many elements for the cooperative launch) and
touch nothing else: their duals stay zero, and the matrix norm is a sum over the columns. The
start is a warm one, since a zero anchor has no rounding of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def with_empty_rows(inst, count):
    m = inst["m"] + count
    return dict(inst, m=m, ptr=np.concatenate([inst["ptr"], np.full(count, inst["ptr"][-1], np.int32)]).astype(np.int32),
                rl=np.concatenate([inst["rl"], np.full(count, -np.inf)]), ru=np.concatenate([inst["ru"], np.full(count, np.inf)]))


@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
@pytest.mark.parametrize("shape", [(40, 31, 3), (2000, 5000, 5)], ids=str)
def test_three_paths_give_the_same_bits(engine, instances, shape, precision):
    base = instances.lp_uniform(8, *shape)
    rng = np.random.default_rng(3)
    x0, y0 = rng.uniform(0, 10, shape[1]), rng.standard_normal(shape[0])
    got, launches = [], []
    for empty in (0, 20000, 700000):
        inst = with_empty_rows(base, empty)
        s = engine.pdlp_default_settings()
        s.max_iterations, s.algorithm, s.eps_optimal, s.ruiz_iterations = 60, engine.PDLP_HALPERN, 1e-300, 3
        s.precision = getattr(engine, precision)
        rc, x, y, r = engine.pdlp_solve(engine.Matrix.from_instance(inst), inst, s, x0=x0, y0=np.r_[y0, np.zeros(empty)])
        assert rc == 0, engine.last_error()
        got.append((x, y[:shape[0]], r["final_step_size"]))
        launches.append(engine.last_timing()["kernel_launches"])
    assert launches[0] == launches[1] < launches[2] - 100   # one launch a window; two an iteration
    for x, y, step in got[1:]:
        assert step == got[0][2]
        assert np.array_equal(x, got[0][0]) and np.array_equal(y, got[0][1])
