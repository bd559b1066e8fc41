"""The shapes at which the cluster and the cooperative launch are compared with the launches take
those paths: a comparison of the launches with themselves would pass as well."""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

spec = importlib.util.spec_from_file_location("cluster_shapes", os.path.join(os.path.dirname(__file__), "test_gpu_cluster.py"))
shapes = importlib.util.module_from_spec(spec)
spec.loader.exec_module(shapes)
COOPERATIVE = {(4000, 9000), (9000, 17500), (9000, 20500), (8193, 5000), (42000, 30000)}


@pytest.mark.parametrize("shape", shapes.SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_paths(engine, instances, shape):
    inst = shapes.lp(instances, *shape)
    A = engine.Matrix.from_instance(inst)
    engine.set_timing(1)
    try:
        rc, *_ = engine.pdhg(A, inst, engine.settings(max_iterations=47, check_every=19, tau=1e-3, sigma=1e-3, tolerance=1e-300))
        launches = engine.last_timing()["kernel_launches"]
    finally:
        engine.set_timing(0)
    assert rc == 0, engine.last_error()
    # one for all on a cluster; a window's one and a checkpoint's four otherwise; the launches 94 + 12
    assert launches == (15 if shape[:2] in COOPERATIVE else 1)
    counts = []
    for call in (lambda s: engine.pdlp_solve(A, inst, s), lambda s: engine.pdlp_solve_qp(A, inst, s, qdiag=np.zeros(shape[1]))):
        s = shapes.scaled_steps(engine, max_iterations=150)
        rc, *_, result = call(s)
        assert rc == 0, engine.last_error()
        counts.append((engine.last_timing()["kernel_launches"], result["iterations"]))
    # the QP's three launches an iteration against one a window, of 64
    saved = 3 * counts[0][1] - 3
    assert counts[0][1] == counts[1][1] and counts[0][0] <= counts[1][0] - saved
    s = shapes.scaled_steps(engine, max_iterations=150, algorithm=engine.PDLP_HALPERN)
    rc, *_, result = engine.pdlp_solve(A, inst, s)
    # the same setup and as many windows as the adaptive solve, where the launches would take 300 more
    assert rc == 0 and engine.last_timing()["kernel_launches"] < counts[0][0] + result["iterations"]
