"""A state written through an address that was asked for once: the device loop
steps from what is there, whatever it left in a call before."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)


class View:
    def __init__(self, h, which):
        self.__cuda_array_interface__ = {"shape": h.shape, "typestr": "<f8", "data": (h.device_state(which), False),
                                         "version": 3}


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP64_FAST])
@pytest.mark.parametrize("nx,ny,march,loop", [(75, 44, "0", "1"), (75, 44, "0", "0"), (200, 190, "58", "0")])
def test_step_n_after_a_write_through_a_kept_address(gpu_lib, monkeypatch, nx, ny, march, loop, precision, steps):
    import torch

    monkeypatch.setenv("E2D_F64_MARCH", march)
    monkeypatch.setenv("E2D_LOOP", loop)
    ua, ub = (C.smooth_state(nx, ny, G14, seed=s) for s in (1, 2))
    p = e2d.make_params(nx, ny, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8, bc=(1, 2, 3, 3),
                        precision=precision)
    with e2d.HydroRun(p, init_problem=False) as h, e2d.HydroRun(p, init_problem=False) as want:
        h.set_state(0, ua)
        views = [torch.as_tensor(View(h, k), device="cuda") for k in (0, 1)]
        t, ns, _ = h.step_n(steps, 10.0, 0.0, 0)
        views[ns % 2].copy_(torch.from_numpy(ub))
        torch.cuda.synchronize()
        got = h.step_n(3, 10.0, t, ns)
        want.set_state(ns % 2, ub)
        ref = want.step_n(3, 10.0, t, ns)
        assert got[:2] == ref[:2] and np.array_equal(got[2], ref[2])
        assert np.array_equal(h.current(got[1]), want.current(got[1]))
