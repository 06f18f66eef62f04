"""The FP64 march of large grids (segments of 32-column strips in chunks of 15
rows): the bits of the tiled step at the edges of chunks, segments and
strips, and its bounded wait."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)


def run(monkeypatch, p, march, steps=(3, 4)):
    monkeypatch.setenv("E2D_LOOP", "0")
    monkeypatch.setenv("E2D_F64_MARCH", str(march))
    u0 = C.smooth_state(p.nx, p.ny, G14, seed=p.nx + 2 * p.ny)
    with e2d.HydroRun(p, init_problem=False) as h:
        h.set_state(0, u0)
        h.set_state(1, u0)
        t, ns, tr = 0.0, 0, []
        for n in steps:
            t, ns, d = h.step_n(n, 10.0, t, ns)
            tr.append(d)
        return [h.get_state(0), h.get_state(1), np.concatenate(tr), np.array([t])]


# segment rows: one chunk (13), two, not a whole number of chunks, the grid's height and more
@pytest.mark.parametrize("rows", [1, 13, 14, 28, 43, 58, 300])
@pytest.mark.parametrize("riemann,precision", [("hllc", "fp64"), ("hll", "fp64"), ("approx", "fp64"), ("hllc", "fast")])
def test_march_equals_tiles(gpu_lib, monkeypatch, rows, riemann, precision):
    # smaller than a strip, odd pitch (gathered), interior chunks by TMA, every boundary type
    for nx, ny, bc in [(2, 2, (1, 1, 1, 1)), (33, 17, (3, 3, 1, 2)), (157, 96, (2, 2, 2, 2)), (200, 131, (1, 2, 3, 3))]:
        p = e2d.make_params(nx, ny, problem="implode", riemann=riemann, gamma0=1.4, cfl=0.8,
                            slope_type=1.0 if rows == 28 else 2.0, bc=bc,
                            precision=e2d.PRECISION_FP64_FAST if precision == "fast" else e2d.PRECISION_FP64)
        want, got = run(monkeypatch, p, 0), run(monkeypatch, p, rows)
        assert all(np.array_equal(a, b) for a, b in zip(want, got)), (nx, ny, rows, riemann)


def test_march_is_what_a_large_grid_runs(gpu_lib, monkeypatch):
    p = e2d.make_params(1100, 1024, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8)
    want = run(monkeypatch, p, 0, (3,))
    monkeypatch.delenv("E2D_F64_MARCH")
    u0 = C.smooth_state(p.nx, p.ny, G14, seed=p.nx + 2 * p.ny)
    with e2d.HydroRun(p, init_problem=False) as h:
        h.set_state(0, u0)
        h.set_state(1, u0)
        t, ns, tr = h.step_n(3, 10.0, 0.0, 0)
        assert np.array_equal(tr, want[2]) and np.array_equal(h.get_state(1), want[1])


def test_march_wait_runs_out_with_etimeout(gpu_lib, monkeypatch):
    """With E2D_TEST_WAIT_TIMEOUT=1 block (1, 0) never copies its second
    chunk: its bounded wait gives up after 1 s, waits (bounded) once more and
    flags the step; step_n returns E2D_ETIMEOUT and the context stays usable."""
    p = e2d.make_params(256, 256, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8)
    monkeypatch.setenv("E2D_F64_MARCH", "58")
    monkeypatch.setenv("E2D_TEST_WAIT_TIMEOUT", "1")
    with e2d.HydroRun(p) as h:
        with pytest.raises(e2d.E2DError) as ei:
            h.step_n(1, 10.0, 0.0, 0)
        assert ei.value.status == 4  # E2D_ETIMEOUT
    monkeypatch.delenv("E2D_TEST_WAIT_TIMEOUT")
    with e2d.HydroRun(p) as h:
        t, ns, _ = h.step_n(2, 10.0, 0.0, 0)
        assert ns == 2 and np.isfinite(h.current(ns)).all()
