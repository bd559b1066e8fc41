"""Solves from several host threads at once, each on a matrix of its own or all on one: the same
bits as alone, and mid-size ones do not queue for the whole chip (a cooperative launch holds
every SM, so that eight of them would take eight times as long as one)."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def together(calls, rounds=1):
    """Runs the calls from a thread each; outputs and the least time of a round."""
    out, errors, times = [None] * len(calls), [], []
    barrier = threading.Barrier(len(calls) + 1)

    def work(k):
        for _ in range(rounds):
            barrier.wait()
            try:
                out[k] = calls[k]()
            except Exception as e:   # noqa: BLE001 (the barrier must not be left waiting)
                errors.append(e)
            barrier.wait()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for _ in range(rounds):
        barrier.wait()
        start = time.perf_counter()
        barrier.wait()
        times.append(time.perf_counter() - start)
    for t in threads:
        t.join()
    assert not errors, errors
    return out, min(times)


def fixed(engine, A, inst, iterations=400):
    def call():
        rc, x, _, r = engine.pdhg(A, inst, engine.settings(max_iterations=iterations, check_every=100, tau=0.02, sigma=0.02,
                                                           tolerance=1e-300))
        assert rc == 0, engine.last_error()
        return x, np.array(r["objective"])
    return call


def restarted(engine, A, inst, **kw):
    s = engine.pdlp_default_settings()
    s.max_iterations, s.eps_optimal, s.ruiz_iterations = 200, 1e-300, 5
    for k, v in kw.items():
        setattr(s, k, v)

    def call():
        rc, x, y, _ = engine.pdlp_solve(A, inst, s)
        assert rc == 0, engine.last_error()
        return x, y
    return call


@pytest.mark.parametrize("shape", [(2000, 5000, 5), (8000, 16000, 8), (50000, 100000, 8)], ids=str)
@pytest.mark.parametrize("one_matrix", [False, True])
def test_threads_give_the_same_bits(engine, instances, shape, one_matrix):
    inst = instances.lp_uniform(9, *shape)
    A = engine.Matrix.from_instance(inst)
    kinds = [lambda m: fixed(engine, m, inst), lambda m: restarted(engine, m, inst),
             lambda m: restarted(engine, m, inst, algorithm=engine.PDLP_HALPERN),
             lambda m: restarted(engine, m, inst, precision=engine.FP32_REFINE)]
    alone = [make(A)() for make in kinds]
    for count in (1, 2):   # 4 and 8 threads
        got, _ = together([make(A if one_matrix else engine.Matrix.from_instance(inst)) for make in kinds * count])
        for k, out in enumerate(got):
            for a, b in zip(alone[k % len(kinds)], out):
                assert np.array_equal(a, b), k


def test_eight_mid_size_solves_share_the_chip(engine, instances):
    """One takes 4.6 ms; eight took 34 ms on cooperative launches and 17 on the two launches an
    iteration, which fill the chip together."""
    inst = instances.lp_uniform(9, 8000, 16000, 8)
    calls = [fixed(engine, engine.Matrix.from_instance(inst), inst, 1000) for _ in range(8)]
    _, one = together(calls[:1], rounds=4)
    _, eight = together(calls, rounds=6)
    assert eight < 6 * one, (one, eight)
