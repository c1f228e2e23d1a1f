"""Recorded nets run on instances of the streaming kernel with and without the
custom-tau pass, by whether a net has such synapses: both against the oracle
in small and large tiles, alone and side by side in a batch."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb
from helpers import assert_state_bits_equal, configs, rows_equal
from test_gpu_xsyn import mixed_tau_net

pytestmark = pytest.mark.gpu
KW = dict(noise_rate_hz=400.0, noise_kick_mv=20.0, seed=5)


def net(share):
    return mixed_tau_net(1500, 30, 3, share)


@pytest.mark.parametrize("share", [0.0, 0.5])
@pytest.mark.parametrize("block, npt", [(64, 4), (128, 1), (256, 8), (512, 4)])
def test_recorded_net_in_every_kind_of_tile(share, block, npt):
    onet = net(share)
    gc, oc = configs(True, 100, 1, **KW)
    g, o = nb.B200Sim(onet.flat(), gc), O.OSim(onet, oc)
    g.set_tile_shape(block, npt)
    for _ in range(3):
        g.run_steps(100)
        o.run_steps(100)
        assert rows_equal(g, o, 100) < 0
    assert o.spikes_total() > 0
    assert_state_bits_equal(g, o)


@pytest.mark.parametrize("shares", [(0.0, 0.0), (0.0, 0.5)])
def test_recorded_nets_of_a_batch(shares):
    onets = [net(s) for s in shares]
    b = nb.Batch([x.flat() for x in onets], [configs(True, 100, 1, **KW)[0] for _ in onets])
    b.set_kernel_mode(nb.KERNEL_STREAM)
    b.run_steps(300)
    for j, x in enumerate(onets):
        o = O.OSim(x, configs(True, 100, 1, **KW)[1])
        o.run_steps(300)
        assert b.spikes_total(j) == o.spikes_total() > 0
        for slot in (0, 1):
            assert np.array_equal(b.state(j, slot).view(np.uint32), o.state(slot).view(np.uint32))
