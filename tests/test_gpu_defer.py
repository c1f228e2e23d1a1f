"""Deferred delivery (AUTO mode, one net past the cluster kernel's size or
with custom-tau synapses): against the oracle where a step's spikes wait for
the next launch: delays of 1 (delivered at once), of 2 and up to the ring
depth, launch groups of every small length (each ends with a flush), bursts
in which every neuron spikes, a switch of the kernel between groups, and the
fall-back when many neurons have a delay of 1."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb
from helpers import assert_state_bits_equal, configs, rows_equal

pytestmark = pytest.mark.gpu

N = 16500  # past 16 blocks of 1024 neurons


def big_net(lo_ms, hi_ms, k=6, ones=0, seed=4):
    net = O.ONet()
    rng = np.random.default_rng(seed)
    for i in range(N):
        net.add_neuron(0.0, 0.0, 0.0, O.EXC if i < 0.8 * N else O.INH)
    for i in range(N):
        for t, w, d in zip(rng.integers(0, N, k), rng.uniform(0.5, 3.0, k), rng.uniform(lo_ms, hi_ms, k)):
            net.push_synapse(i, int(t), float(w), float(d))
    for i in rng.integers(0, N, ones):
        net.push_synapse(int(i), int(rng.integers(0, N)), 2.0, 0.1)
    return net


@pytest.mark.parametrize("lo_ms, hi_ms, ones", [(0.2, 1.0, 0), (0.2, 1.0, 300), (0.1, 0.3, 0), (1.0, 30.0, 40)])
def test_groups_of_every_length(lo_ms, hi_ms, ones):
    onet = big_net(lo_ms, hi_ms, ones=ones)
    gc, oc = configs(True, 300, 1, noise_rate_hz=300.0, noise_kick_mv=20.0, seed=9)
    g, o = nb.B200Sim(onet.flat(), gc), O.OSim(onet, oc)
    done = 0
    for i, steps in enumerate((1, 2, 3, 4, 5, 256, 17, 1, 1, 257)):
        if i == 6:
            g.set_kernel_mode(nb.KERNEL_STREAM)
        if i == 7:
            g.set_kernel_mode(nb.KERNEL_AUTO)
        g.run_steps(steps)
        o.run_steps(steps)
        done += steps
        assert rows_equal(g, o, min(steps, 300)) < 0, f"raster differs in the {steps} steps to {done}"
    assert g.spikes_total() == o.spikes_total() > 0
    assert_state_bits_equal(g, o)
    g.reset_state()
    o.reset_state()
    g.run_steps(40)
    o.run_steps(40)
    assert rows_equal(g, o, 40) < 0
    assert_state_bits_equal(g, o)


def test_every_neuron_spikes_at_once():
    onet = big_net(0.1, 1.2)
    gc, oc = configs(True, 120, 1, seed=2)
    g, o = nb.B200Sim(onet.flat(), gc), O.OSim(onet, oc)
    g.set_external_all(np.full(N, 60.0, np.float32))
    for i in range(N):
        o.set_external(i, 60.0)
    g.run_steps(120)
    o.run_steps(120)
    assert rows_equal(g, o, 120) < 0
    assert g.spikes_total() == o.spikes_total() >= N
    assert_state_bits_equal(g, o)
