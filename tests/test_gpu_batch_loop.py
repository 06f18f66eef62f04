"""The batches' multi-iteration launches (k_batch_loop_f64, k_batch_loop_f32c): a
wait that runs out, and the same bits whatever the list and its launches are."""
import numpy as np
import pytest

import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu

POOL = 1 << 30


def implosion(nx, ny, precision, riemann="hllc", **kw):
    return e2d.make_params(nx, ny, problem="implode", riemann=riemann, gamma0=1.4, cfl=0.8, implode_shape=1,
                           precision=precision, **kw)


@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP32C])
def test_batch_barrier_wait_runs_out_with_etimeout(gpu_lib, monkeypatch, precision):
    """With E2D_TEST_WAIT_TIMEOUT=2 the barrier between two iterations waits for
    one block more than there are: the wait gives up after its 1 s limit, every
    instance whose units the blocks had reports E2D_ETIMEOUT, and none is
    stepped again."""
    p = [implosion(n, 96, precision) for n in (128, 70)]
    monkeypatch.setenv("E2D_TEST_WAIT_TIMEOUT", "2")
    with e2d.Batch(pool_bytes=POOL) as b:
        ids = [b.admit(q, 10.0) for q in p]
        assert b.run(3) == 0
        before = [b.poll(i) for i in ids]
        for i, (t, ns, active, ok) in zip(ids, before):
            assert ns == 1 and not active and not ok
            with pytest.raises(e2d.E2DError) as ei:
                b.query(i)
            assert ei.value.status == 4  # E2D_ETIMEOUT
        assert b.run(3) == 0 and [b.poll(i) for i in ids] == before
    monkeypatch.delenv("E2D_TEST_WAIT_TIMEOUT")
    with e2d.Batch(pool_bytes=POOL) as b:
        ids = [b.admit(q, 10.0) for q in p]
        assert b.run(3) == 2
        assert all(b.query(i)[1] == 3 and np.isfinite(b.get_state(i)).all() for i in ids)


def test_fp64_loop_barrier_wait_runs_out_with_etimeout(gpu_lib, monkeypatch):
    p = implosion(128, 96, e2d.PRECISION_FP64)
    monkeypatch.setenv("E2D_TEST_WAIT_TIMEOUT", "2")
    with e2d.HydroRun(p) as h:
        with pytest.raises(e2d.E2DError) as ei:
            h.step_n(3, 10.0, 0.0, 0)
        assert ei.value.status == 4  # E2D_ETIMEOUT
    monkeypatch.delenv("E2D_TEST_WAIT_TIMEOUT")
    with e2d.HydroRun(p) as h:
        t, ns, _ = h.step_n(3, 10.0, 0.0, 0)
        assert ns == 3 and np.isfinite(h.current(ns)).all()


def test_strip_heights_alone_are_a_tuning(gpu_lib, monkeypatch):
    """Heights without a variant keep a short list in strips of them, and an
    autotune that has nothing to time leaves them: strips have no grid barrier,
    so E2D_TEST_WAIT_TIMEOUT=2 does not stop the solve."""
    p = implosion(128, 96, e2d.PRECISION_FP32C)
    monkeypatch.setenv("E2D_TEST_WAIT_TIMEOUT", "2")
    for autotune in (False, True):
        with e2d.Batch(pool_bytes=POOL) as b:
            b.set_tuning(strip_h=[32, 48, 64])
            i = b.admit(p, 10.0)
            if autotune:
                b.autotune(2)
            assert b.run(3) == 1 and b.query(i)[1] == 3
            assert b.get_tuning()[1] == [32, 48, 64]


def alone(p, steps):
    with e2d.HydroRun(p) as h:
        t, ns, _ = h.step_n(steps, 1e9, 0.0, 0)
        return t, h.current(ns)


# lists whose FP64 tiles are chosen 8, 16 and 32 columns wide
LISTS = [[(96, 80), (40, 33), (2, 2)], [(300, 200), (64, 64)], [(500, 300), (301, 257), (64, 48)]]
WALLS = [(1, 1, 1, 1), (3, 3, 2, 1), (2, 1, 3, 3)]


@pytest.mark.parametrize("loop", ["0", "1"])
@pytest.mark.parametrize("grids", LISTS)
@pytest.mark.parametrize("riemann", ["approx", "hll", "hllc"])
@pytest.mark.parametrize("precision", [e2d.PRECISION_FP64, e2d.PRECISION_FP32C])
def test_a_list_ends_where_each_grid_alone_does(gpu_lib, monkeypatch, precision, riemann, grids, loop):
    """Also without cooperative launches (E2D_LOOP=0): a launch per iteration."""
    monkeypatch.setenv("E2D_LOOP", loop)
    params = [implosion(nx, ny, precision, riemann, bc=bc) for (nx, ny), bc in zip(grids, WALLS)]
    with e2d.Batch(riemann, pool_bytes=POOL) as b:
        ids = [b.admit(p, 1e9) for p in params]
        assert b.run(4) == len(ids) and b.run(3) == len(ids)
        got = [(b.query(i)[0], b.get_state(i)) for i in ids]
    for p, (t, u) in zip(params, got):
        want = alone(p, 7)
        assert t == want[0] and np.array_equal(u, want[1])


def test_a_reused_slot_copies_by_its_own_tensor_map(gpu_lib):
    """Instances of other sizes one after another in the same table slot, rows
    staged by TMA (variant 6): each ends where the grid alone does."""
    with e2d.Batch(pool_bytes=POOL) as b:
        b.set_tuning(6, [32, 32, 32])
        for k, (nx, ny) in enumerate([(300, 96), (421, 130), (200, 64), (700, 200), (301, 97)]):
            p = implosion(nx, ny, e2d.PRECISION_FP32C, bc=WALLS[k % 3])
            i = b.admit(p, 1e9)
            assert i == 0 and b.run(5) == 1
            want = alone(p, 5)
            assert b.query(i)[0] == want[0] and np.array_equal(b.get_state(i), want[1])
            b.release(i)


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("riemann", ["hllc", "approx"])
def test_a_long_list_that_gets_short(gpu_lib, riemann, autotune):
    """More than 1100 fold units (strips, one launch an iteration, timed by an
    autotune), then 449 and 65 as the larger solves end (short strips, many
    iterations a launch): each solve ends where its grid alone does."""
    params = [implosion(nx, ny, e2d.PRECISION_FP32C, riemann, bc=bc)
              for (nx, ny), bc in zip([(1100, 700), (700, 500), (300, 200)], WALLS)]
    want = [alone(p, 50 + 10 * k) for k, p in enumerate(params)]
    with e2d.Batch(riemann, pool_bytes=POOL) as b:
        ids = [b.admit(p, t) for p, (t, _) in zip(params, want)]
        if autotune:
            b.autotune(2)
            assert 0 < b.query(ids[0])[1] < 50 and b.get_tuning()[0] in (4, 5, 6)
        while b.run(7) > 0:
            pass
        got = [(b.query(i), b.get_state(i)) for i in ids]
    for k, ((t, ns, active), u) in enumerate(got):
        assert not active and ns == 50 + 10 * k and t == want[k][0] and np.array_equal(u, want[k][1])
