"""FP64 Riemann solvers where intermediate values overflow though inputs and
fluxes are finite: the oracle's bits."""
import numpy as np
import pytest

import euler2d_kokkos_gb300 as e2d

pytestmark = pytest.mark.gpu


def wide(rng, n, lo, hi):
    x = np.exp2(rng.uniform(lo, hi, (n, 8))) * rng.uniform(1, 2, (n, 8)) * rng.choice([-1.0, 1.0], (n, 8))
    x[:, [0, 1, 4, 5]] = np.abs(x[:, [0, 1, 4, 5]])
    return x


@pytest.mark.parametrize("gamma0", [1.4, 3.0])
def test_hll_kinetic_energy_near_overflow(gpu_lib, gamma0):
    """Half of r u^2 is finite where r u^2 is not; and ordinary, tiny and still states."""
    from oracle import pyoracle as O

    rng = np.random.default_rng(7)
    x = np.concatenate([wide(rng, 2000, -20, 20), wide(rng, 2000, -300, 300), wide(rng, 2000, -20, 20)])
    big = x[4000:]  # supersonic, r u^2 of the upwind side about 2^1024
    s = rng.choice([-1.0, 1.0], 2000)
    big[:, [1, 5]] = 1e-10
    big[:, [2, 6]] = s[:, None] * rng.uniform(0.9, 1.4, (2000, 2))
    big[:, [3, 7]] *= 1e-20
    for side in (0, 1):
        m, r, u = (s < 0) == side, 4 * side, 4 * side + 2
        with np.errstate(over="ignore"):
            big[m, r] = np.minimum(np.exp2(1023.0 + rng.uniform(-0.5, 1.2, m.sum())) / big[m, u] ** 2, 1.7e308)
    x[:500, 2] = 0.0
    x[250:750, 7] = -0.0
    out = e2d.eval_device(e2d.make_params(64, 64, gamma0=gamma0, riemann="hll"), "riemann_hll", x)
    want = O.riemann(O.make_params(64, 64, gamma0=O.f32(gamma0)), "hll", x[:, :4], x[:, 4:])
    ok = np.isfinite(want)
    assert ok[4000:, 1].sum() > 200
    assert np.array_equal(out[ok], want[ok])
    assert not np.isfinite(out[~ok]).any()
