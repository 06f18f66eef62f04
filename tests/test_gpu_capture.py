"""godunov_unsplit captured into a CUDA graph: a replay steps the states as they
are then, whatever was called before the capture or between replays."""
import numpy as np
import pytest

import _cases as C
import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

G14 = C.f32(1.4)
NX, NY, BC = 75, 44, (1, 2, 3, 3)
DT = 1e-3


def handle(u0, precision):
    p = e2d.make_params(NX, NY, problem="implode", riemann="hllc", gamma0=1.4, cfl=0.8, bc=BC, precision=precision)
    h = e2d.HydroRun(p, init_problem=False)
    h.set_state(0, u0)
    h.set_state(1, u0)
    return h


class Captured:
    """The steps 0 and 1 of a handle as a graph on its own stream."""

    def __init__(self, h):
        import torch

        self.torch, self.stream = torch, torch.cuda.ExternalStream(h.stream())
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(self.stream):
            self.graph.capture_begin()
            h.godunov_unsplit(0, DT)
            h.godunov_unsplit(1, DT)
            self.graph.capture_end()

    def replay(self):
        with self.torch.cuda.stream(self.stream):
            self.graph.replay()
        self.torch.cuda.synchronize()


@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP32C])
def test_replay_after_compute_dt_and_a_new_state(gpu_lib, precision):
    ua, ub = (C.smooth_state(NX, NY, G14, seed=s) for s in (1, 2))
    with handle(ua, precision) as h, handle(ub, precision) as want:
        h.compute_dt(0)
        g = Captured(h)
        h.set_state(0, ub)
        g.replay()
        want.godunov_unsplit(0, DT)
        want.godunov_unsplit(1, DT)
        assert np.array_equal(h.U, want.U) and np.array_equal(h.U2, want.U2)


@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP32C])
@pytest.mark.parametrize("call", ["compute_dt", "step_n"])
def test_a_replay_between_calls_is_seen(gpu_lib, precision, call):
    ua = C.smooth_state(NX, NY, G14, seed=1)
    with handle(ua, precision) as h, handle(ua, precision) as want:
        g = Captured(h)
        g.replay()
        want.godunov_unsplit(0, DT)
        want.godunov_unsplit(1, DT)
        if call == "compute_dt":
            assert h.compute_dt(0) == want.compute_dt(0)
            g.replay()
            want.godunov_unsplit(0, DT)
            want.godunov_unsplit(1, DT)
            h.godunov_unsplit(0, DT)
            want.set_state(0, want.U)
            want.godunov_unsplit(0, DT)
        else:
            t, ns, _ = h.step_n(2, 10.0, 0.0, 0)
            assert want.step_n(2, 10.0, 0.0, 0)[:2] == (t, ns)
            g.replay()
            want.godunov_unsplit(0, DT)
            want.godunov_unsplit(1, DT)
            want.set_state(0, want.U)
            got, ref = h.step_n(3, 10.0, t, ns), want.step_n(3, 10.0, t, ns)
            assert got[:2] == ref[:2] and np.array_equal(got[2], ref[2])
        assert np.array_equal(h.U, want.U) and np.array_equal(h.U2, want.U2)
