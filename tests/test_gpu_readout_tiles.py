"""The tiled readout kernels at the edges of their tiles (32 x 32 Gram and
normal tiles, chunks of 32 terms, Cholesky panels of 32 rows, trailing tiles
of 64), a failed factorization inside a panel, and more classes than a host
solve takes side by side: weights equal the oracle's bit for bit."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu


def design(t, f, seed):
    rng = np.random.default_rng(seed)
    return rng.poisson(1.5, (t, f)).astype(np.float32), rng.integers(0, 1 << 30, t)


@pytest.mark.parametrize("t, f, k", [(2, 1, 2), (31, 3, 2), (32, 33, 3), (33, 32, 4), (65, 129, 5), (96, 31, 2),
                                     (161, 66, 9), (225, 700, 4)])
def test_multi_at_tile_edges(t, f, k):
    x, r = design(t, f, t * 7 + f)
    lab = r % k
    w = nb.fit_ridge_multi(x, lab, k, 0.7)
    ref = O.fit_ridge_multi(x, lab, k, 0.7)
    assert np.array_equal(w.view(np.uint64), ref.view(np.uint64))


@pytest.mark.parametrize("t, f", [(1, 1), (5, 30), (32, 31), (33, 32), (64, 33), (100, 63), (31, 95), (130, 200)])
def test_binary_at_tile_edges(t, f):
    x, r = design(t, f, t * 5 + f)
    y = (r % 2).astype(np.float32)
    w = nb.fit_ridge(x, y, 0.5)
    ref = O.fit_ridge(x, y, 0.5)
    assert np.array_equal(w.view(np.uint64), ref.view(np.uint64))


@pytest.mark.parametrize("t, f", [(40, 70), (20, 33)])
def test_failed_factorization_falls_back(t, f):
    """No regularisation and fewer rows than features: a pivot fails in a
    later row of some panel, and the retry or the zeros follow the oracle."""
    x, r = design(t, f, 3)
    x[:, f // 2] = x[:, 0]
    y = (r % 2).astype(np.float32)
    w = nb.fit_ridge(x, y, 0.0)
    ref = O.fit_ridge(x, y, 0.0)
    assert np.array_equal(np.nan_to_num(w).view(np.uint64), np.nan_to_num(ref).view(np.uint64))
