"""Every tile shape of the fused FP64 step, at its smallest and largest number
of rows and as chosen for the grid, on grids at the edges of tiles: dt
sequence and whole state bit for bit the oracle's."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)
# smaller than a tile, one cell more or less than whole tiles, odd pitch (tiles gathered), several waves of tiles
GRIDS = [(2, 2, (1, 1, 1, 1)), (9, 7, (3, 3, 1, 2)), (33, 17, (1, 2, 3, 3)), (64, 48, (1, 1, 1, 1)),
         (127, 65, (2, 2, 2, 2)), (230, 196, (3, 3, 3, 3))]
# 100 rows + shape: 32, 16 and 8 columns
TILES = [None, "0", "300", "700", "1300", "1", "301", "1101", "2", "302", "502"]


@pytest.mark.parametrize("tile", TILES)
def test_every_tile_gives_the_oracle_bits(gpu_lib, monkeypatch, tile):
    if tile is not None:
        monkeypatch.setenv("E2D_F64_TILE", tile)
    for k, (nx, ny, bc) in enumerate(GRIDS):
        riemann = ("hllc", "hll", "approx")[k % 3]
        slope = (2.0, 1.0)[k % 2]
        p = e2d.make_params(nx, ny, problem="implode", riemann=riemann, gamma0=1.4, cfl=0.8, slope_type=slope, bc=bc)
        u0 = C.smooth_state(nx, ny, G14, seed=7 * nx + ny)
        with e2d.HydroRun(p, init_problem=False) as h:
            h.set_state(0, u0)
            h.set_state(1, u0)
            t, ns, trace = h.step_n(9, 10.0, 0.0, 0)
            got = h.current(ns)
            # the host-driven step (two launches) takes the same tiles
            h.set_state(0, u0)
            h.godunov_unsplit(0, float(trace[0]))
            first = h.get_state(1)
        op = po.make_params(nx, ny, gamma0=1.4, cfl=0.8, slope_type=slope, bc=bc, riemann=riemann)
        want, dts, _, n = po.run(op, u0, 9, 10.0)
        assert ns == n == 9
        assert np.array_equal(trace, dts), (nx, ny, tile)
        assert np.array_equal(got, want), (nx, ny, tile)
        assert np.array_equal(first, po.run(op, u0, 1, 10.0)[0]), (nx, ny, tile)
