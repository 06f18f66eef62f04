"""Short strips (FP32C) and multi-step launches (both precisions): the bits of
16-row strips and of one launch per step, at the sizes where they can differ."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)


def run(monkeypatch, prec, nx, ny, bc, steps, *, loop, strip=None, riemann="hllc", t_end=10.0, slope=2.0):
    monkeypatch.setenv("E2D_LOOP", loop)
    if strip:
        monkeypatch.setenv("E2D_F32C_STRIP_H", strip)
    else:
        monkeypatch.delenv("E2D_F32C_STRIP_H", raising=False)
    p = e2d.make_params(nx, ny, problem="implode", riemann=riemann, gamma0=1.4, cfl=0.8, slope_type=slope, bc=bc,
                        precision=prec)
    u0 = C.smooth_state(nx, ny, G14, seed=nx + 3 * ny)
    with e2d.HydroRun(p, init_problem=False) as h:
        h.set_state(0, u0)
        h.set_state(1, u0)
        t, ns, tr = 0.0, 0, []
        for n in steps:
            t, ns, d = h.step_n(n, t_end, t, ns)
            tr.append(d)
        return [h.get_state(0), h.get_state(1), np.concatenate(tr), np.array([t, ns])]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# one unit and less; a strip's last columns at every offset of a 16-byte chunk; heights around a unit's; > 2 waves
FP32C_GRIDS = [(2, 2, (1, 1, 1, 1)), (3, 5, (3, 3, 3, 3)), (58, 16, (2, 1, 1, 2)), (59, 17, (1, 2, 3, 3)),
               (60, 15, (3, 3, 2, 1)), (61, 31, (1, 1, 2, 2)), (62, 33, (2, 2, 1, 1)), (121, 130, (3, 3, 3, 3)),
               (300, 200, (1, 2, 1, 2))]


@pytest.mark.parametrize("strip", [None, "2", "4", "8"])
@pytest.mark.parametrize("loop", ["0", "1"])
def test_fp32c_short_strips_give_the_bits_of_a_unit(gpu_lib, monkeypatch, strip, loop):
    for k, (nx, ny, bc) in enumerate(FP32C_GRIDS):
        riemann = ("hllc", "hll", "approx")[k % 3]
        want = run(monkeypatch, e2d.PRECISION_FP32C, nx, ny, bc, [5, 6], loop="0", strip="16", riemann=riemann)
        got = run(monkeypatch, e2d.PRECISION_FP32C, nx, ny, bc, [5, 6], loop=loop, strip=strip, riemann=riemann)
        assert same(got, want), (nx, ny, bc, strip, loop)


@pytest.mark.parametrize("strip", ["2", "4", "8"])
def test_fp32c_loop_with_several_units_a_block(gpu_lib, monkeypatch, strip):
    """More units than blocks that fit the GPU at once."""
    nx, ny = {"2": (700, 400), "4": (900, 500), "8": (1400, 900)}[strip]
    want = run(monkeypatch, e2d.PRECISION_FP32C, nx, ny, (1, 1, 1, 1), [7], loop="0", strip="16")
    got = run(monkeypatch, e2d.PRECISION_FP32C, nx, ny, (1, 1, 1, 1), [7], loop="1", strip=strip)
    assert same(got, want)


@pytest.mark.parametrize("nx,ny,bc", [(2, 3, (1, 1, 1, 1)), (65, 33, (3, 3, 3, 3)), (222, 140, (1, 2, 3, 3)),
                                      (640, 420, (2, 2, 1, 1))])
@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP64_FAST])
def test_fp64_loop_equals_a_launch_per_step(gpu_lib, monkeypatch, nx, ny, bc, precision):
    want = run(monkeypatch, precision, nx, ny, bc, [5, 1, 7], loop="0", slope=1.0)
    got = run(monkeypatch, precision, nx, ny, bc, [5, 1, 7], loop="1", slope=1.0)
    assert same(got, want)


@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP32C])
def test_loop_stops_at_t_end_and_takes_many_steps(gpu_lib, monkeypatch, precision):
    """t_end inside a launch, resuming after it, and more steps than one launch takes."""
    a = run(monkeypatch, precision, 40, 24, (1, 1, 1, 1), [3, 50, 50], loop="0", t_end=0.05)
    b = run(monkeypatch, precision, 40, 24, (1, 1, 1, 1), [3, 50, 50], loop="1", t_end=0.05)
    assert same(a, b) and b[3][0] == 0.05
    a = run(monkeypatch, precision, 24, 16, (3, 3, 3, 3), [1300], loop="0", t_end=1e9)
    b = run(monkeypatch, precision, 24, 16, (3, 3, 3, 3), [1300], loop="1", t_end=1e9)
    assert same(a, b) and b[3][1] == 1300


def test_loop_barrier_wait_runs_out_with_etimeout(gpu_lib, monkeypatch):
    """With E2D_TEST_WAIT_TIMEOUT=1 the barrier of a multi-step launch waits
    for one block more than there are; the wait gives up after its 1 s limit,
    step_n returns E2D_ETIMEOUT and the context stays usable."""
    p = e2d.make_params(128, 96, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8, implode_shape=1,
                        precision=e2d.PRECISION_FP32C)
    monkeypatch.setenv("E2D_TEST_WAIT_TIMEOUT", "1")
    with e2d.HydroRun(p) as h:
        with pytest.raises(e2d.E2DError) as ei:
            h.step_n(3, 10.0, 0.0, 0)
        assert ei.value.status == 4  # E2D_ETIMEOUT
    monkeypatch.delenv("E2D_TEST_WAIT_TIMEOUT")
    with e2d.HydroRun(p) as h:
        t, ns, _ = h.step_n(3, 10.0, 0.0, 0)
        assert ns == 3 and np.isfinite(h.current(ns)).all()


@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP32C])
def test_loop_reports_a_nonfinite_state(gpu_lib, precision):
    p = e2d.make_params(64, 48, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8, precision=precision)
    with e2d.HydroRun(p) as h:
        u = h.U
        u[0, 20, 20] = np.nan
        h.set_state(0, u)
        with pytest.raises(e2d.E2DError) as ei:
            h.step_n(10, 10.0, 0.0, 0)
        assert ei.value.status == 3  # E2D_ENUMERIC
