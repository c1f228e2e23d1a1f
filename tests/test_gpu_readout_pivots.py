"""A matrix that is not positive definite, found while many blocks work on the
panel: the fits' second try, or their zeros, equal the oracle's bit for bit."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column", [1, 40, 500])
def test_binary_pivot_fails_in_an_early_and_a_late_panel(column):
    rng = np.random.default_rng(column)
    x = rng.poisson(1.5, (900, 640)).astype(np.float32)
    x[:, column] = x[:, 0]
    y = rng.integers(0, 2, 900).astype(np.float32)
    w, ref = nb.fit_ridge(x, y, 0.0), O.fit_ridge(x, y, 0.0)
    assert np.array_equal(np.nan_to_num(w).view(np.uint64), np.nan_to_num(ref).view(np.uint64))


@pytest.mark.parametrize("lam", [-20000.0, -20.0])
def test_multi_pivot_fails(lam):
    """A negative ridge: the first pivot fails, or one in the middle; the dual
    weights are then zeros and the biases the class means."""
    rng = np.random.default_rng(5)
    x = rng.poisson(1.5, (700, 300)).astype(np.float32)
    lab = rng.integers(0, 3, 700).astype(np.uint32)
    w, ref = nb.fit_ridge_multi(x, lab, 3, lam), O.fit_ridge_multi(x, lab, 3, lam)
    assert np.array_equal(w.view(np.uint64), ref.view(np.uint64))
    assert not w[:, :-1].any() and w[:, -1].all()
