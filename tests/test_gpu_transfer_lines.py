"""The projections between levels as chains of fixed-point lines
(adg_transfer.cuh) where they can go wrong: batch sizes around a block's, every
(D, P), columns of zeros, at the ends of the range of doubles, and values that
are not finite.

Tolerance, relative to the sum of |coefficient x value| of a column: a column
with the dense FP64 operators sums up to 2^D Np_s = 160 terms, 160 * 2^-53 =
1.8e-14; the fixed-point lines keep 2^-54 of the column's bound and round once.
Among subnormal numbers every term may round by one unit, times the row sums
of the operators' two factors (at most 3^D (2P + 1)^D)."""
import numpy as np
import pytest

import oracle_ffi as O
from parity import G

pytestmark = pytest.mark.gpu
TOL = 2e-14
ALL = [(2, p) for p in range(1, 7)] + [(3, p) for p in range(1, 4)]


def sim(D, P):
    s = G.AmrDG(P=P, D=D)
    s.setGeometrySettings(prob_lo=(0, 0, 0), prob_hi=(1, 1, 1), n_cell=(4, 4, 1 if D == 2 else 4), periodic=(1, 1, 1))
    s.settings(c_dt=0.5)
    s.init(G.Compressible_Euler().settings("isentropic_vortex" if D == 2 else "blast3d"))
    return s


def matrices(D, P):
    """Scatter and gather of every child, [2^D, Np, Np]."""
    Minv, nov = O.matrix(D, P, "Minv"), 1 << D
    return (np.stack([Minv @ O.matrix(D, P, "P_cf", l) for l in range(nov)]),
            np.stack([Minv @ O.matrix(D, P, "P_fc", l) for l in range(nov)]) / nov)


def check(got, mats, src, tiny=0.0):
    """got[i, q] = sum_k mats[i, k] src[i, k, q], to TOL of the column's terms and tiny."""
    top = np.max(np.abs(src), axis=(1, 3), keepdims=True)  # [i, 1, q, 1]
    unit = src / np.where(top > 0, top, 1.0)
    want = np.einsum("iknm,ikqm->iqn", mats, unit)
    bound = np.max(np.einsum("iknm,ikqm->iqn", np.abs(mats), np.abs(unit)), axis=2, keepdims=True)
    top = np.where(top > 0, top, 1.0)[:, 0]
    assert np.all(np.abs(got / top - want) <= TOL * bound + tiny / top)


@pytest.mark.parametrize("D,P", ALL)
@pytest.mark.parametrize("n", [1, 7, 33, 300])  # less than a block's, several blocks and a rest
def test_batches_match_the_dense_matrices(D, P, n):
    s = sim(D, P)
    down, up = matrices(D, P)
    r = np.random.default_rng(100 * D + 10 * P + n)
    coarse = r.standard_normal((n, s.Q, s.Np_s)) * 10.0 ** r.uniform(-6, 6, (n, s.Q, s.Np_s))
    child = r.integers(0, 1 << D, n).astype(np.int8)
    check(s.amr_scatter(coarse, child), down[child][:, None], coarse[:, None])
    kids = r.standard_normal((n, 1 << D, s.Q, s.Np_s)) * 10.0 ** r.uniform(-6, 6, (n, 1 << D, s.Q, s.Np_s))
    check(s.amr_gather(kids), np.broadcast_to(up, (n,) + up.shape), kids)


@pytest.mark.parametrize("D,P", [(2, 1), (2, 3), (2, 6), (3, 2)])
def test_columns_at_the_ends_of_the_range(D, P):
    s = sim(D, P)
    down, up = matrices(D, P)
    r = np.random.default_rng(D + P)
    tiny = 2.0 ** -1074 * (2 << D) * s.Np_s * 3 ** D * (2 * P + 1) ** D
    scale = np.array([1e-320, 1e-309, 1e-300, 1e-270, 1e-269, 1e-200, 0.0, -0.0, 1.0, 1e200, 1e298, 1e303, 1e305])
    n = 40
    c = scale[r.integers(0, len(scale), (n, 1, s.Q, 1))]
    coarse = (c * r.uniform(-1, 1, (n, 1, s.Q, s.Np_s)))[:, 0]
    child = r.integers(0, 1 << D, n).astype(np.int8)
    check(s.amr_scatter(coarse, child), down[child][:, None], coarse[:, None], tiny)
    kids = c * r.uniform(-1, 1, (n, 1 << D, s.Q, s.Np_s))
    check(s.amr_gather(kids), np.broadcast_to(up, (n,) + up.shape), kids, tiny)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite_stay_in_their_column(bad):
    s = sim(2, 3)
    r = np.random.default_rng(3)
    n = 21
    coarse = r.standard_normal((n, s.Q, s.Np_s))
    child = r.integers(0, 4, n).astype(np.int8)
    kids = r.standard_normal((n, 4, s.Q, s.Np_s))
    a, b = s.amr_scatter(coarse, child), s.amr_gather(kids)
    coarse[5, 2, 0] = bad  # the mean reaches mode 0 only
    kids[9, 3, 1, 0] = bad  # a child's mean reaches every mode
    a2, b2 = s.amr_scatter(coarse, child), s.amr_gather(kids)
    rest = np.ones((n, s.Q), bool)
    rest[5, 2] = False
    assert np.array_equal(a2[rest], a[rest]) and not np.isfinite(a2[5, 2, 0])
    assert np.all(np.isfinite(a2[5, 2, 1:]))
    rest[5, 2], rest[9, 1] = True, False
    assert np.array_equal(b2[rest], b[rest]) and not np.isfinite(b2[9, 1, 0])
