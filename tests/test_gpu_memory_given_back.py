"""Device memory that solves keep for the next one goes back when the last matrix handle is
destroyed, and on request; each case in a process of its own, whose other allocations stand
still meanwhile."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
PROGRAM = """
import importlib.util, sys
import numpy as np
import torch
def load(name, path):
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod
E = load("sankhya_b200", "the-solver_b200/__init__.py")
I = load("inst", "the-solver_b200/instances.py")
MB = 1 << 20
def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
def solve(A, inst):
    s = E.pdlp_default_settings()
    s.max_iterations, s.eps_optimal, s.ruiz_iterations = 64, 1e-300, 2
    assert E.pdlp_solve(A, inst, s)[0] == 0, E.last_error()
tiny = I.lp_uniform(1, 30, 40, 3)
T = E.Matrix.from_instance(tiny)
solve(T, tiny)                      # modules, streams and the pool itself exist
inst = I.lp_uniform(2, 300000, 600000, 4)
"""


def run(body):
    out = subprocess.run([sys.executable, "-c", PROGRAM + body], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr


def test_the_last_handle_gives_it_back():
    run("""
T.close()
before = free()
A = E.Matrix.from_instance(inst)
solve(A, inst)
A.close()
assert before - free() <= 72 * MB, (before - free()) / MB   # 64 MiB stay for small solves
""")


def test_given_back_on_request():
    run("""
A = E.Matrix.from_instance(inst)
before = free()
solve(A, inst)
kept = before - free()
E.release_memory()
assert kept >= 64 * MB, kept / MB   # or this shows nothing
assert before - free() <= 8 * MB, (before - free()) / MB
solve(A, inst)
""")


def test_a_matrix_holds_no_numbered_copies_on_the_launches():
    """900,000 rows and columns are beyond the cooperative launch: a fixed-step solve's cached
    workspace is 16 vectors of 8 bytes, without the 16 bytes more each that the launch numbers."""
    run("""
A = E.Matrix.from_instance(inst)
before = free()
assert E.pdhg(A, inst, E.settings(max_iterations=5, check_every=5, tau=1e-3, sigma=1e-3, tolerance=1e-300))[0] == 0
kept = before - free()
vectors = 8 * (10 * 600000 + 6 * 300000)
assert vectors <= kept <= vectors + 8 * MB, kept / MB
""")


def test_a_handle_may_outlive_the_threads_streams():
    """The last handle destroyed by another thread than the one that solved, which has ended."""
    run("""
import threading
T.close()
A = E.Matrix.from_instance(inst)
t = threading.Thread(target=solve, args=(A, inst))
t.start()
t.join()
t = threading.Thread(target=A.close)
t.start()
t.join()
A = E.Matrix.from_instance(tiny)
solve(A, tiny)
import atexit
atexit.register(A.close)
""")
