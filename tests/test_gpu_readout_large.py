"""A factor larger than the pinned buffer that the fits keep (64 MB): its copy
is pageable, the weights equal the oracle's bit for bit."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu


def test_multi_with_a_pageable_factor():
    rng = np.random.default_rng(8)
    t = 2901  # 2901^2 doubles: 67.3 MB
    x = rng.poisson(1.5, (t, 40)).astype(np.float32)
    lab = rng.integers(0, 3, t).astype(np.uint32)
    w, ref = nb.fit_ridge_multi(x, lab, 3, 0.5), O.fit_ridge_multi(x, lab, 3, 0.5)
    assert np.array_equal(w.view(np.uint64), ref.view(np.uint64))
