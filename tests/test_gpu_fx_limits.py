"""Where the fixed-point columns' arithmetic ends and the FP64 evaluation takes
over (adg_fx.cuh), through whole steps."""
import numpy as np
import pytest

from parity import G
from test_gpu_plain_predictor import pair

pytestmark = pytest.mark.gpu

CELLS = {2: (6, 5, 1), 3: (4, 3, 3)}
FLOOR = 10 * 2.0 ** -52  # of the pressure


def low_pressure(shape, D, seed):
    """Densities about 1e-13, no momentum, positive pressures below the floor
    (two fifths of the energy) that vary within the elements."""
    r = np.random.RandomState(seed)
    U = np.zeros(shape)
    n = len(U)
    U[:, 0, 0] = r.uniform(1e-13, 2e-13, n)
    U[:, D + 1, 0] = r.uniform(2e-15, 4e-15, n)
    U[:, D + 1, 1] = 0.3 * U[:, D + 1, 0]
    assert 0.4 * 1.3 * U[:, D + 1, 0].max() < FLOOR
    return U


@pytest.mark.parametrize("D,P", [(2, 1), (2, 3), (2, 5), (3, 2)])
def test_step_below_the_pressure_floor_matches_oracle(D, P):
    """The floored pressure is uniform, so the momentum stays at zero; the
    unfloored one's gradient gives it 1e-3 of the density.  Tolerance as in
    test_gpu_plain_predictor."""
    o, g = pair(D, P, CELLS[D], "vortex" if D == 2 else "blast3d")
    U = low_pressure(o.get_uw().shape, D, P)
    o.set_uw(U, 0)
    g.set_U_w(U)
    o.dt = g.Dt = 1e-2
    o.ader()
    g.ADER()
    a, b = g.get_U_w(), o.get_uw()
    assert np.max(np.abs(a - b)) < 1e-13 * np.max(np.abs(b[:, 0, 0]))


@pytest.mark.parametrize("D,P", [(2, 2), (2, 3), (3, 2)])
def test_seeded_step_below_the_pressure_floor_matches_its_fallback(D, P):
    """Every element's time-independent part from the fixed-point kernel, and
    every element recomputed by the FP64 fallback.  The FP32 changes and the
    untrained seed matter in the second order of Dt/dx = 1e-6; an unfloored
    pressure would change the momentum by Dt/dx times a part of the floor."""
    _, g = pair(D, P, CELLS[D], "vortex" if D == 2 else "blast3d")
    U = low_pressure(g.get_U_w().shape, D, P)
    dx = max(np.subtract(g.cfg.prob_hi[:D], g.cfg.prob_lo[:D]) / np.array(CELLS[D][:D]))
    seed = G.PredictorSeed(D, P, hidden=128, rng_seed=5)
    out = []
    for tol in (1e30, 1e-300):
        seed.attach(g, mode=2, sweeps=P, tol=tol)
        g.set_U_w(U)
        g.Dt = 1e-6 * dx
        g.ADER()
        out.append(g.get_U_w())
        fallbacks, predicted = G.seed_stats(g)
        assert fallbacks == (0 if tol > 1 else predicted)
    assert np.max(np.abs(out[0] - out[1])[:, 1:D + 1]) < 1e-3 * 1e-6 * FLOOR
