"""The host-driven step reuses the primitives compute_dt formed only while
nothing can have changed the state between the two calls."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)
NX, NY, BC = 75, 44, (1, 2, 3, 3)


def handle(u0):
    p = e2d.make_params(NX, NY, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8, bc=BC)
    h = e2d.HydroRun(p, init_problem=False)
    h.set_state(0, u0)
    h.set_state(1, u0)
    return h


def step_alone(u0, dt, nstep=0):
    with handle(u0) as h:
        h.godunov_unsplit(nstep, dt)
        return h.U, h.U2


def test_step_after_compute_dt_equals_the_step_alone(gpu_lib):
    ua = C.smooth_state(NX, NY, G14, seed=1)
    with handle(ua) as h:
        dt = h.compute_dt(0)
        assert h.compute_dt(0) == dt
        h.godunov_unsplit(0, dt)
        got = h.U, h.U2
        want = step_alone(ua, dt)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        # the other state's primitives are not this one's
        h.compute_dt(0)
        dt1 = h.compute_dt(1)
        h.godunov_unsplit(1, dt1)
        with handle(ua) as f:
            f.godunov_unsplit(0, dt)
            f.godunov_unsplit(1, dt1)
            assert np.array_equal(h.U, f.U) and np.array_equal(h.U2, f.U2)


@pytest.mark.parametrize("change", ["set_state", "other_state", "step_n", "address_before", "address_between", "godunov"])
def test_a_changed_state_is_not_stepped_from_old_primitives(gpu_lib, change):
    import torch

    ua, ub = (C.smooth_state(NX, NY, G14, seed=s) for s in (1, 2))
    dt = 1e-3

    class View:
        def __init__(self, h, which):
            self.__cuda_array_interface__ = {"shape": h.shape, "typestr": "<f8", "data": (h.device_state(which), False),
                                             "version": 3}

    with handle(ua) as h:
        if change == "address_before":
            t = torch.as_tensor(View(h, 0), device="cuda")
        h.compute_dt(0)
        nstep, want = 0, step_alone(ub, dt)[1]
        if change == "set_state":
            h.set_state(0, ub)
        elif change == "other_state":
            h.set_state(1, ub)
            nstep, want = 1, step_alone(ub, dt, 1)[0]
        elif change == "step_n":
            _, ns, _ = h.step_n(2, 10.0, 0.0, 0)
            with handle(ua) as f:
                f.step_n(2, 10.0, 0.0, 0)
                f.godunov_unsplit(0, dt)
                want = f.U2
        elif change == "godunov":
            h.godunov_unsplit(1, 2e-3)  # rewrites state 0
            with handle(ua) as f:
                f.godunov_unsplit(1, 2e-3)
                f.godunov_unsplit(0, dt)
                want = f.U2
        else:
            if change == "address_between":
                t = torch.as_tensor(View(h, 0), device="cuda")
            t.copy_(torch.from_numpy(ub))
            torch.cuda.synchronize()
        h.godunov_unsplit(nstep, dt)
        got = h.get_state(1 - nstep)
        assert np.array_equal(got, want)


def test_compute_dt_reports_a_nonfinite_state_and_recovers(gpu_lib):
    ua = C.smooth_state(NX, NY, G14, seed=1)
    bad = ua.copy()
    bad[0, 20, 20] = np.nan
    with handle(ua) as h:
        dt = h.compute_dt(0)
        h.set_state(0, bad)
        with pytest.raises(e2d.E2DError) as ei:
            h.compute_dt(0)
        assert ei.value.status == 3  # E2D_ENUMERIC
        h.set_state(0, ua)
        assert h.compute_dt(0) == dt
