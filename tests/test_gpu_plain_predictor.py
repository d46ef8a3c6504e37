"""The plain predictor's fixed-point operators (adg_predictor_fx.cuh) where
they can go wrong: element counts around a block's, every (D, P), columns that
are zero or far apart in magnitude, and values that are not finite.

Tolerance against the oracle: the fixed-point operators carry 2^-60 of a
column's bound times at most N^(D+1) = 343, 3e-16, and the oracle's dense sums
of up to 343 terms round to about 343 * 2^-53 = 4e-14; 1e-13 covers one step."""
import numpy as np
import pytest

import oracle_ffi as O
from parity import G

pytestmark = pytest.mark.gpu


def pair(D, P, n, ic, periodic=1, E=0):
    hi = tuple(float(k) / max(n) * (10.0 if ic == "vortex" else 1.0) for k in n)
    kw = dict(seed=11, noise_amp=1e-3) if ic == "kh_noise" else dict(u_inf=1.0, v_inf=0.5)
    o = O.OracleSim(O.make_cfg(D=D, P=P, n=n, hi=hi, periodic=(periodic,) * 3, ic=ic, c_dt=0.5, **kw))
    o.init()
    g = G.AmrDG(P=P, D=D)
    g.setGeometrySettings(prob_lo=(0, 0, 0), prob_hi=hi, n_cell=n, periodic=(periodic,) * 3)
    g.settings(c_dt=0.5, elems_per_block=E)
    g.init(G.Compressible_Euler().settings("isentropic_vortex" if ic == "vortex" else ic, **kw))
    g.set_U_w(o.get_uw())
    g.Dt = o.dt
    return o, g


# element counts 1, a block less one, a block plus one, several blocks and a rest
@pytest.mark.parametrize("D,P,n,ic,E", [
    (2, 1, (1, 1, 1), "vortex", 0), (2, 1, (17, 1, 1), "vortex", 16), (2, 2, (5, 3, 1), "kh_noise", 16),
    (2, 2, (11, 3, 1), "kh_noise", 32), (2, 3, (1, 7, 1), "kh_noise", 8), (2, 3, (17, 3, 1), "kh_noise", 16),
    (2, 4, (3, 3, 1), "vortex", 0), (2, 5, (7, 5, 1), "kh_noise", 0), (2, 6, (3, 5, 1), "vortex", 0),
    (3, 1, (5, 1, 1), "blast3d", 4), (3, 1, (7, 3, 2), "blast3d", 16), (3, 2, (1, 7, 1), "blast3d", 8),
    (3, 2, (3, 3, 2), "blast3d", 4), (3, 3, (3, 1, 3), "blast3d", 0), (3, 3, (5, 2, 2), "blast3d", 0)])
def test_step_matches_oracle(D, P, n, ic, E):
    o, g = pair(D, P, n, ic, periodic=0 if ic == "blast3d" else 1, E=E)
    o.ader()
    g.ADER()
    a, b = g.get_U_w(), o.get_uw()
    assert np.max(np.abs(a - b)) < 1e-13 * np.max(np.abs(b[:, :, 0]))


@pytest.mark.parametrize("D,P", [(2, 1), (2, 3), (2, 4), (3, 1), (3, 2)])
@pytest.mark.parametrize("slope", [0.5, 0.98])
def test_steep_densities_and_low_pressures_match_oracle(D, P, slope):
    """Densities up to 100 apart within an element, and pressures down to the
    floor beside ordinary ones: both flux evaluations and their border."""
    o, g = pair(D, P, (6, 5, 1) if D == 2 else (4, 3, 3), "vortex" if D == 2 else "blast3d")
    r = np.random.RandomState(P)
    U = np.zeros_like(o.get_uw())
    n = len(U)
    lin = 1  # the first mode of degree one
    U[:, 0, 0] = r.uniform(1, 2, n)
    U[::2, 0, lin] = slope * U[::2, 0, 0]
    U[:, 1:D + 1, 0] = 0.02 * r.uniform(-1, 1, (n, D))
    U[:, D + 1, 0] = np.where(np.arange(n) % 3 == 0, 1e-14, 1.0)
    o.set_uw(U, 0)
    g.set_U_w(U)
    o.dt = g.Dt = 1e-4
    o.ader()
    g.ADER()
    a, b = g.get_U_w(), o.get_uw()
    assert np.isfinite(b).all()
    assert np.max(np.abs(a - b)) < 1e-13 * np.max(np.abs(b[:, :, 0]))


@pytest.mark.parametrize("D,P", [(2, 1), (2, 2), (2, 3), (2, 6), (3, 2), (3, 3)])
def test_step_scales_with_the_state(D, P):
    """The Euler fluxes are homogeneous of degree one where the pressure is above
    its floor: a state times a power of two steps to the result times it, bit
    for bit (column exponents only)."""
    _, g = pair(D, P, (5, 4, 3)[:D] + (1,) * (3 - D), "vortex" if D == 2 else "blast3d")
    r = np.random.RandomState(D + P)
    U = 0.02 * r.uniform(-1, 1, g.get_U_w().shape)
    U[:, 0, 0] = r.uniform(1, 2, len(U))
    U[:, 1:D + 1, 0] = r.uniform(-0.3, 0.3, (len(U), D))
    U[:, D + 1, 0] = r.uniform(4, 6, len(U))  # pressure above 1.4
    dt = 1e-3
    g.set_U_w(U)
    g.Dt = dt
    g.ADER()
    ref = g.get_U_w()
    for k in (-16, 40, 300):
        g.set_U_w(np.ldexp(U, k))
        g.Dt = dt
        g.ADER()
        assert np.array_equal(g.get_U_w(), np.ldexp(ref, k)), k


@pytest.mark.parametrize("D,P", [(2, 1), (2, 3), (2, 5), (3, 2)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_that_are_not_finite_stay_in_their_neighbourhood(D, P, bad):
    n = (9, 7, 1) if D == 2 else (5, 4, 6)
    o, g = pair(D, P, n, "kh_noise" if D == 2 else "blast3d")
    U = o.get_uw()
    g.ADER()
    ref = g.get_U_w()
    k = n[0] * (n[1] // 2) + 3
    V = U.copy()
    V[k, D + 1, 0] = bad  # the energy's mean
    g.set_U_w(V)
    g.Dt = o.dt
    g.ADER()
    out = g.get_U_w()
    xyz = np.stack(np.unravel_index(np.arange(len(U)), n[:D][::-1])[::-1], 1)
    gap = np.abs(xyz - xyz[k])
    gap = np.minimum(gap, np.array(n[:D]) - gap).sum(1)
    finite = np.isfinite(out).all(axis=(1, 2))
    assert not finite[gap <= 1].any()
    assert np.array_equal(out[gap > 1], ref[gap > 1])
    g.set_Dt()
    assert g.status() & 1
