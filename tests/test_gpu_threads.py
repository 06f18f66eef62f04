"""Handles stepped from several host threads at once: multi-step cooperative
launches of small grids, plain launches of larger ones and a batch, each with
the results it has alone."""
import threading

import numpy as np
import pytest

import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu


def params(nx, ny, precision):
    return e2d.make_params(nx, ny, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8, implode_shape=1,
                           precision=precision)


def steps(p):
    with e2d.HydroRun(p) as h:
        t, ns = 0.0, 0
        for n in (300, 1, 299):
            t, ns, _ = h.step_n(n, 1e9, t, ns)
        return t, h.current(ns)


def host_loop(p):
    with e2d.HydroRun(p) as h:
        t = 0.0
        for n in range(60):
            dt = h.compute_dt(n % 2)
            h.godunov_unsplit(n, dt)
            t += dt
        return t, h.current(60)


def batch(p):
    with e2d.Batch("hllc", pool_bytes=1 << 28) as b:
        ids = [b.admit(q, 1e9) for q in (p, params(150, 70, e2d.PRECISION_FP64))]
        for _ in range(6):
            assert b.run(50) == 2
        return b.query(ids[0])[0], np.concatenate([b.get_state(i).ravel() for i in ids])


def test_threads_do_not_change_results(gpu_lib):
    jobs = [(steps, params(640, 420, e2d.PRECISION_FP64)), (steps, params(90, 70, e2d.PRECISION_FP64)),
            (steps, params(700, 400, e2d.PRECISION_FP32C)), (steps, params(128, 128, e2d.PRECISION_FP32C)),
            (steps, params(1500, 900, e2d.PRECISION_FP32C)), (host_loop, params(300, 200, e2d.PRECISION_FP64)),
            (batch, params(200, 160, e2d.PRECISION_FP32C))]
    want = [f(p) for f, p in jobs]
    got = [None] * len(jobs)

    def work(k):
        try:
            got[k] = jobs[k][0](jobs[k][1])
        except Exception as e:  # reported by the assertion below
            got[k] = e

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, (g, w) in enumerate(zip(got, want)):
        assert not isinstance(g, Exception), (k, g)
        assert g[0] == w[0] and np.array_equal(g[1], w[1]), k
