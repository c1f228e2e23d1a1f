"""The kernel that runs is the one that is reported: by a sim's size and
synapses, after a tile shape, a kernel or autotuning was asked for, and for
batches and servers.  (What each computes is compared elsewhere.)"""
import numpy as np
import pytest

import neuro_edit_v2_b200 as nb
from neuro_edit_v2_b200 import workloads as W

pytestmark = pytest.mark.gpu
IZH = np.array([0.02, 0.2, -65.0, 8.0], np.float32)


def sparse(n, tau=0.0, seed=1):
    rng = np.random.default_rng(seed)
    e = 500
    return nb.from_synapses(np.zeros(n, np.uint8), np.tile(IZH, (n, 1)), np.zeros(n, np.uint8), rng.integers(0, n, e),
                            rng.integers(0, n, e), rng.random(e), rng.uniform(0.1, 3.0, e),
                            tau_ms=np.full(e, tau, np.float32) if tau else None)


@pytest.mark.parametrize("n, tau, runs", [(300, 0.0, "cluster"), (16384, 0.0, "cluster"), (16400, 0.0, "deferred"),
                                          (2000, 5.0, "deferred"), (150000, 0.0, "stream")])
def test_a_sim_by_its_size(n, tau, runs):
    s = nb.B200Sim(sparse(n, tau), int_weights=1)
    assert s.tiling()["runs"] == s.running_kernel() == runs
    s.run_steps(30)
    assert s.running_kernel() == runs
    s.set_kernel_mode(nb.KERNEL_RESIDENT)
    assert s.running_kernel() == "resident"
    s.set_kernel_mode(nb.KERNEL_AUTO)
    assert s.running_kernel() == runs
    s.set_tile_shape(128, 1)
    assert s.tiling()["runs"] == "stream" and s.tiling()["block"] == 128


def test_a_batch_and_a_server():
    b = nb.Batch([sparse(400), sparse(3000)], [nb.default_config(int_weights=1, seed=k) for k in range(2)])
    assert b.running_kernel() == "cluster"
    b.set_kernel_mode(nb.KERNEL_STREAM)
    assert b.running_kernel() == "stream"
    b = nb.Batch([sparse(400), sparse(3000, tau=4.0)], [nb.default_config(int_weights=1, seed=k) for k in range(2)])
    assert b.running_kernel() == "stream"
    srv = nb.Server(neuron_capacity=1 << 16, synapse_capacity=1 << 20, ring_capacity=1 << 24, max_requests=2)
    cfg = nb.default_config(int_weights=1, window_steps=100, max_windows=2)
    net = W.with_inputs(sparse(900), 2, 10, 5.0, np.random.default_rng(0))
    assert srv.submit(net, cfg, np.zeros((200, 2), np.float32), 200) is not None
    assert srv.running_kernel() == "cluster"
    srv.set_tile_shape(128, 1)
    assert srv.running_kernel() == "stream"
