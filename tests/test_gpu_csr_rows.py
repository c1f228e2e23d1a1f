"""The device CSR build's two ways of bringing a row into list order, at the
edges of what each takes: rows of up to 128 synapses (in registers), up to
512 and 2048 (staged passes), one more than the limit (the scatter), empty
rows, lists in source order and reversed: equal to the host build."""
import numpy as np
import pytest

import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["source", "reversed", "shuffled"])
@pytest.mark.parametrize("longest", [1, 127, 128, 129, 511, 513, 2048, 2049])
def test_rows_of_every_length_class(longest, order):
    n = 150
    rng = np.random.default_rng(longest)
    lens = rng.integers(0, longest + 1, n)
    lens[[3, 149]] = longest
    lens[[0, 70]] = 0
    src = np.repeat(np.arange(n), lens).astype(np.uint32)
    if order == "reversed":
        src = src[::-1].copy()
    elif order == "shuffled":
        rng.shuffle(src)
    e = len(src)
    tgt = rng.integers(0, n, e).astype(np.uint32)
    w = rng.uniform(-1.0, 1.0, e).astype(np.float32)
    # a long delay in half of the cases: the wide record
    d = rng.uniform(0.0, 40.0 if longest % 2 else 20.0, e).astype(np.float32)
    kind = (rng.random(n) < 0.2).astype(np.uint8)
    params = np.tile(np.array([0.02, 0.2, -65.0, 8.0], np.float32), (n, 1))
    cfg = nb.default_config(int_weights=1)
    host = nb.B200Sim(nb.from_synapses(np.zeros(n, np.uint8), params, kind, src, tgt, w, d, dt_ms=cfg.dt_ms), cfg)
    dev = nb.B200Sim.from_synapses(np.zeros(n, np.uint8), params, kind, src, tgt, w, d, cfg)
    for x, y, what in zip(host.read_csr(), dev.read_csr(), ("rowptr", "tgt", "w", "delay")):
        assert np.array_equal(x, y), what
