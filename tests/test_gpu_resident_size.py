"""The largest net that the resident kernel holds in 256 x 2 tiles: 27 tiles
of 512 neurons in each block's shared memory, on every SM."""
import numpy as np
import pytest
import torch

import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu


def test_twenty_seven_tiles_per_sm_fit():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 27 * 512 - 5000
    rng = np.random.default_rng(3)
    e = 1000
    src, tgt = (rng.integers(0, n, e).astype(np.uint32) for _ in range(2))
    args = (np.zeros(n, np.uint8), np.tile(np.array([0.02, 0.2, -65.0, 8.0], np.float32), (n, 1)),
            np.zeros(n, np.uint8), src, tgt, np.full(e, 3.0, np.float32), np.full(e, 0.3, np.float32),
            nb.default_config(int_weights=1, noise_rate_hz=400.0, noise_kick_mv=30.0, seed=2))
    got = []
    for mode in (nb.KERNEL_RESIDENT, nb.KERNEL_STREAM):
        with nb.B200Sim.from_synapses(*args) as sim:
            sim.set_kernel_mode(mode)
            assert sim.kernel_mode()[1] == (mode == nb.KERNEL_RESIDENT)
            sim.run_steps(40)
            got.append((sim.spikes_total(), sim.v(), sim.state(1), sim.syn_current(), sim.trace()))
    assert got[0][0] == got[1][0] > 0
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("tiles, share", [(1, 8), (27, 20)])
def test_custom_currents_with_and_without_their_buffer(tiles, share):
    """Synapses with their own tau, at a size where the buffer of their
    currents fits beside the state and at one where it does not."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * tiles * 512 - 5000 if tiles == 27 else 5003
    rng = np.random.default_rng(tiles)
    e = 40 * 3000
    src, tgt = (rng.integers(0, min(n, 3000), e).astype(np.uint32) for _ in range(2))
    tau = np.where(rng.random(e) < share / 40.0, rng.uniform(1.0, 30.0, e), 0.0).astype(np.float32)
    net = nb.from_synapses(np.zeros(n, np.uint8), np.tile(np.array([0.02, 0.2, -65.0, 8.0], np.float32), (n, 1)),
                           np.zeros(n, np.uint8), src, tgt, rng.random(e).astype(np.float32),
                           rng.uniform(0.1, 2.0, e).astype(np.float32), tau_ms=tau)
    cfg = nb.default_config(int_weights=1, noise_rate_hz=400.0, noise_kick_mv=30.0, seed=2)
    got = []
    for mode in (nb.KERNEL_RESIDENT, nb.KERNEL_STREAM):
        with nb.B200Sim(net, cfg) as sim:
            sim.set_kernel_mode(mode)
            sim.run_steps(60)
            got.append((sim.spikes_total(), sim.v(), sim.state(1), sim.syn_current(), sim.trace()))
    assert got[0][0] == got[1][0] > 0
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
