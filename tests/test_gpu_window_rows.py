"""spike_counts over windows of every kind of length (more rows than a byte
counts, a window that wraps the record ring, one row, none) and ragged sizes
around the 1024 neurons of a block, against sums of the rows themselves."""
import numpy as np
import pytest

import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 1024, 1025, 2100])
def test_windows_equal_the_sum_of_their_rows(n):
    rng = np.random.default_rng(n)
    e = 4 * n
    net = nb.from_synapses(np.zeros(n, np.uint8), np.tile(np.float32([0.02, 0.2, -65.0, 8.0]), (n, 1)),
                           np.zeros(n, np.uint8), rng.integers(0, n, e), rng.integers(0, n, e),
                           rng.uniform(0, 2, e), rng.uniform(0.1, 5.0, e))
    s = nb.B200Sim(net, nb.default_config(int_weights=1, record_spikes=1, spike_record_steps=700, seed=3,
                                          noise_rate_hz=2000.0, noise_kick_mv=30.0))
    s.run_steps(950)  # the ring has wrapped
    bits = np.stack([np.unpackbits(s.spike_row(b).view(np.uint8), bitorder="little")[:n] for b in range(700)])
    assert bits.sum() > 0
    for rows in (0, 1, 2, 31, 32, 33, 255, 256, 257, 508, 699, 700):
        assert np.array_equal(s.spike_counts(rows), bits[:rows].sum(axis=0)), rows
