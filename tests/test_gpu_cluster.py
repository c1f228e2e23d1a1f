"""The cluster kernel (one thread-block cluster per net, several steps per
barrier where the shortest delay allows) against the C oracle: with the int
ring every raster row and every state bit is equal, at the edges of its
shapes (one warp, one block, two blocks, sixteen, more neurons than threads),
for hops of one step, of a few and of the cap, at delays up to the ring
depth, and across windows that cut hops short."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb
from helpers import assert_state_bits_equal, lockstep

pytestmark = pytest.mark.gpu


def net_with_delays(n, k, lo_ms, hi_ms, seed):
    net = O.ONet()
    rng = np.random.default_rng(seed)
    for i in range(n):
        net.add_neuron(0.0, 0.0, 0.0, O.EXC if i < 0.8 * n else O.INH)
    for i in range(n):
        for t, w, d in zip(rng.integers(0, n, k), rng.uniform(0.5, 3.0, k), rng.uniform(lo_ms, hi_ms, k)):
            net.push_synapse(i, int(t), float(w), float(d))
    return net


@pytest.mark.parametrize("n, k, lo_ms, hi_ms", [
    (1, 1, 0.1, 0.1),       # a neuron alone on a ring of two slots
    (33, 8, 0.1, 1.5),      # a ragged warp, hop 1
    (256, 12, 0.3, 0.7),    # one block, hop 3, delays near the ring depth
    (257, 12, 0.6, 4.0),    # two blocks, hop 6
    (1100, 20, 2.0, 3.0),   # hop cut at its cap of 16, delay 16 more than the cap
    (5000, 12, 0.2, 0.9),   # sixteen blocks, hop 2
])
def test_rasters_and_state_equal_the_oracle(n, k, lo_ms, hi_ms):
    onet = net_with_delays(n, k, lo_ms, hi_ms, n)
    g, o, first = lockstep(onet, 400, int_weights=True, chunk=50, noise_rate_hz=400.0, noise_kick_mv=20.0, seed=3)
    assert first < 0, f"raster diverged at step {first}"
    assert o.spikes_total() > 0
    assert_state_bits_equal(g, o)


@pytest.mark.parametrize("mode", [nb.KERNEL_AUTO, nb.KERNEL_STREAM])
def test_windows_cut_hops_and_many_nets_share_launches(mode):
    """Uneven nets, windows of 7 steps (not a multiple of any hop), launches
    of 1, 5 and 64 steps: every window count and state equals the oracle's."""
    sizes = [(40, 0.1), (300, 0.6), (1500, 0.6), (2600, 0.3), (700, 2.5)]
    onets = [net_with_delays(n, 10, lo, lo + 1.0, n) for n, lo in sizes]
    kw = dict(int_weights=1, noise_rate_hz=400.0, noise_kick_mv=20.0, window_steps=7, max_windows=40)
    b = nb.Batch([x.flat() for x in onets], [nb.default_config(seed=5 + j, **kw) for j in range(len(onets))])
    b.set_kernel_mode(mode)
    for steps in (1, 5, 64, 210):
        b.run_steps(steps)
    for j, x in enumerate(onets):
        o = O.OSim(x, O.cfg(seed=5 + j, int_weights=1, noise_rate_hz=400.0, noise_kick_mv=20.0, record_spikes=1,
                            spike_record_steps=512, exp_mode=1))
        for w in range(40):
            o.run_steps(7)
            assert np.array_equal(b.window_counts(j, w), o.spike_counts(7)), f"net {j} window {w}"
        assert b.spikes_total(j) == o.spikes_total() > 0
        for slot in (0, 1):
            assert np.array_equal(b.state(j, slot).view(np.uint32), o.state(slot).view(np.uint32))
