"""Spike lists of the cluster kernel that no ring word goes with: networks
whose spikes come from kicks alone, on clusters of several blocks with hops
longer than one step, against the C oracle."""
import numpy as np
import pytest

import pyoracle as O
from helpers import assert_state_bits_equal, lockstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, lo, hi", [(2000, 3, 4), (4100, 6, 40), (3000, 16, 17)])
@pytest.mark.parametrize("heard", [0.0, 0.01])
def test_kicked_spikes_are_delivered(n, lo, hi, heard):
    """Synapses of weight 0 leave every ring word 0 (`heard` of them have a
    weight, so an entry lost or stale would show in the targets)."""
    net = O.ONet()
    rng = np.random.default_rng(n + lo)
    for i in range(n):
        net.add_neuron(0.0, 0.0, 0.0, O.EXC)
    for i in range(n):
        for t, d, h in zip(rng.integers(0, n, 6), rng.integers(lo, hi + 1, 6), rng.random(6)):
            net.push_synapse(i, int(t), 4.0 if h < heard else 0.0, 0.1 * float(d))
    g, o, first = lockstep(net, 600, int_weights=True, chunk=100, noise_rate_hz=500.0, noise_kick_mv=40.0, seed=n)
    assert first < 0, f"raster diverged at step {first}"
    assert o.spikes_total() > n
    assert_state_bits_equal(g, o)
