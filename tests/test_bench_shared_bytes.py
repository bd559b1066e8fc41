"""The byte count behind the shared-matrix batch's reported bandwidth: column bounds are one
pair per column and slab of 32 LPs, and the LPs' own only where a slab's differ."""
import importlib.util
import os

import numpy as np

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_bounds_are_counted_by_slab():
    spec = importlib.util.spec_from_file_location("bench_bytes", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    m, n, nnz, batch = 50, 100, 600, 70   # three slabs, the last of 6 LPs, stored as 96
    cl, cu = np.zeros((batch, n)), np.ones((batch, n))
    matrix = 24 * nnz + 4 * (m + 1) + 4 * (n + 1)
    vectors = 8 * 96 * (n + 2 * m) + 8 * 96 * (m + 3 * n) + 16 * n + 24 * m
    assert bench.shared_iteration_bytes(m, n, nnz, cl, cu) == matrix + vectors + 3 * 16 * n
    cl[40, 7] = cu[40, 7] = 1.0    # a node fixes a variable: one slab of one column differs
    cu[69, 9] = 0.0
    assert bench.shared_iteration_bytes(m, n, nnz, cl, cu) == matrix + vectors + 3 * 16 * n + 2 * 16 * 32
