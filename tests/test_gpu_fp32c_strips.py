"""FP32C strips of two heights on one grid (tall ones that fill whole waves,
shorter ones after them): the bits of strips of one height, where the rows of
one height end inside the other's, at odd sizes and with every staging."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)


def run(p, u0):
    with e2d.HydroRun(p, init_problem=False) as h:
        h.set_state(0, u0)
        t, ns, tr = h.step_n(3, 10.0, 0.0, 0)
        return [h.get_state(ns % 2), tr, np.array([t])]


# 60-column strips, 1824 of them a wave: 32-row strips just over one wave, with 16-row ones after them;
# 64 or 128 rows with a last strip of one row; a grid of one column strip
@pytest.mark.parametrize("nx,ny,riemann", [(6000, 641, "hllc"), (2048, 2048, "hll"), (9000, 1703, "hllc"),
                                           (2896, 2897, "approx"), (60, 59000, "hllc")])
@pytest.mark.parametrize("variant", [None, "6", "7"])
def test_two_heights_equal_one(gpu_lib, monkeypatch, nx, ny, riemann, variant):
    if variant and riemann != "hllc":
        pytest.skip("one solver per staging")
    p = e2d.make_params(nx, ny, problem="implode", riemann=riemann, gamma0=1.4, cfl=0.8, slope_type=2.0,
                        bc=(1, 2, 3, 3), precision=e2d.PRECISION_FP32C)
    u0 = C.smooth_state(nx, ny, G14, seed=nx)
    if variant:
        monkeypatch.setenv("E2D_F32C_VARIANT", variant)
    got = run(p, u0)
    monkeypatch.setenv("E2D_F32C_STRIP_H", "48")
    want = run(p, u0)
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


# the chunks with ghost columns: first, last and last but one of the grid, all three in one strip (57 columns and
# less), none of a chunk's own (nx + 2 a multiple of 4), the grid's edge at a strip's; against rows kept in registers
@pytest.mark.parametrize("nx", [2, 5, 33, 57, 58, 59, 60, 61, 62, 117, 121])
@pytest.mark.parametrize("riemann", ["hllc", "approx"])
@pytest.mark.parametrize("bc", [(1, 2, 1, 1), (3, 3, 2, 1)])
def test_edge_columns_equal_register_rows(gpu_lib, monkeypatch, nx, riemann, bc):
    p = e2d.make_params(nx, 37, problem="implode", riemann=riemann, gamma0=1.4, cfl=0.8, slope_type=2.0, bc=bc,
                        precision=e2d.PRECISION_FP32C)
    u0 = C.smooth_state(nx, 37, G14, seed=nx)
    monkeypatch.setenv("E2D_F32C_VARIANT", "2")
    want = run(p, u0)
    for variant, height in (("4", "16"), ("4", "32"), (None, "2"), (None, "8")):
        monkeypatch.delenv("E2D_F32C_VARIANT")
        if variant:
            monkeypatch.setenv("E2D_F32C_VARIANT", variant)
        monkeypatch.setenv("E2D_F32C_STRIP_H", height)
        got = run(p, u0)
        monkeypatch.delenv("E2D_F32C_STRIP_H")
        monkeypatch.setenv("E2D_F32C_VARIANT", "2")
        assert all(np.array_equal(a, b) for a, b in zip(want, got)), (variant, height)
