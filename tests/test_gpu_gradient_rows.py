"""The weight gradients split over the samples (mlp::k_sgemm, EPI_SLICE): one
sample at a time carries the whole gradient, so a sample lost or counted twice
at the end of a K step, of a slice or of the batch is an error of order one."""
import numpy as np
import pytest

from parity import G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,n", [(100, 129), (128, 1000), (128, 8229), (130, 20001)])
def test_every_sample_counts_once(hidden, n):
    """Targets equal to the outputs but in one row: every sum over the samples
    has one term that is not zero, so the gradient is the same bits wherever the
    row stands.  Slices end at multiples of 16 samples."""
    s = G.PredictorSeed(2, 1, hidden=hidden, rng_seed=3)
    r = np.random.default_rng(n)
    X = r.standard_normal((n, s.n_in)).astype(np.float32)
    Y = s.forward(X)
    first = None
    ends = r.choice(np.arange(16, n - 1, 16), 24, replace=n < 400)
    for row in sorted({0, 1, 15, n // 2, n - 2, n - 1, *ends, *(ends - 1), 16 * ((n - 1) // 16)}):
        at = np.arange(n)
        at[[0, row]] = row, 0  # sample 0 stands in this row
        T = Y[at]
        T[row] += 1.0
        g, loss = s.gradients(X[at], T)
        if first is None:
            first = g, loss
            assert np.isfinite(g).all() and np.count_nonzero(g) > 0.9 * g.size
            assert abs(loss * n - 1.0) < 1e-6
        assert np.array_equal(g, first[0]) and loss == first[1], row
