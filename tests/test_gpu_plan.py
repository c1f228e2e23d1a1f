"""The choice between clusters and the streaming kernel for several nets, and
a server whose choice changes while requests run: the same results."""
import numpy as np
import pytest

import neuro_edit_v2_b200 as nb
from neuro_edit_v2_b200 import workloads as W

pytestmark = pytest.mark.gpu
IZH = np.array([0.02, 0.2, -65.0, 8.0], np.float32)


def net(n, lo_ms, hi_ms, seed=1, k=8, tau=0.0):
    rng = np.random.default_rng(seed)
    e = n * k
    return nb.from_synapses(np.zeros(n, np.uint8), np.tile(IZH, (n, 1)), np.zeros(n, np.uint8),
                            np.repeat(np.arange(n), k), rng.integers(0, n, e), rng.random(e),
                            rng.uniform(lo_ms, hi_ms, e), tau_ms=np.full(e, tau, np.float32) if tau else None)


@pytest.mark.parametrize("sizes, lo_ms, runs", [
    ((8000, 8000), 0.1, "cluster"),
    ((60000, 60000), 0.1, "stream"),   # four passes on 32 of the SMs
    ((60000, 60000), 0.6, "cluster"),  # six steps per barrier
    ((66000, 300), 0.6, "stream"),     # past what a cluster holds
])
def test_a_batch_runs_where_it_is_faster_and_the_same(sizes, lo_ms, runs):
    nets = [net(n, lo_ms, 5.0, seed=j) for j, n in enumerate(sizes)]
    cfgs = [nb.default_config(int_weights=1, noise_rate_hz=200.0, seed=j) for j in range(len(sizes))]
    a, b = nb.Batch(nets, cfgs), nb.Batch(nets, cfgs)
    assert a.running_kernel() == runs
    b.set_kernel_mode(nb.KERNEL_STREAM)
    for x in (a, b):
        x.run_steps(150)
    for j in range(len(sizes)):
        assert a.spikes_total(j) == b.spikes_total(j) > 0
        for slot in (0, 1):
            assert np.array_equal(a.state(j, slot).view(np.uint32), b.state(j, slot).view(np.uint32))


def test_a_server_changes_kernels_between_steps():
    rng = np.random.default_rng(4)
    reqs = {"small": (net(3000, 0.1, 5.0, seed=1), 900), "tau": (net(1200, 0.1, 5.0, seed=2, tau=6.0), 200),
            "large": (net(70000, 0.6, 5.0, seed=3, k=4), 150), "late": (net(2100, 0.8, 5.0, seed=4), 300)}
    reqs = {k: (W.with_inputs(x, 2, 40, 12.0, rng), s) for k, (x, s) in reqs.items()}
    cfg = {k: nb.default_config(int_weights=1, window_steps=50, max_windows=20, noise_rate_hz=200.0, seed=11 + j)
           for j, k in enumerate(reqs)}
    inputs = {k: (rng.random((s, 2)) < 0.1).astype(np.float32) for k, (_, s) in reqs.items()}

    def serve(forced):
        srv = nb.Server(neuron_capacity=1 << 18, synapse_capacity=1 << 22, ring_capacity=1 << 26, max_requests=4,
                        steps_per_launch=50)
        if forced:
            srv.set_tile_shape(128, 1)
        ids, seen = {}, []
        for after, k in ((0, "small"), (2, "tau"), (8, "large"), (12, "late")):
            while len(seen) < after:
                seen.append(srv.running_kernel())
                srv.step()
            ids[k] = srv.submit(reqs[k][0], cfg[k], inputs[k], reqs[k][1])
        while srv.stats()["active"]:
            seen.append(srv.running_kernel())
            srv.step()
        return {k: srv.take(i) for k, i in ids.items()}, seen

    got, seen = serve(False)
    assert seen[:2] == ["cluster"] * 2 and seen[2:6] == ["stream"] * 4  # custom tau comes
    assert seen[6:8] == ["cluster"] * 2 and seen[8:11] == ["stream"] * 3  # ... and goes; the large net comes
    assert set(seen[12:18]) == {"cluster"}
    ref, forced = serve(True)
    assert set(forced) == {"stream"}
    for k in reqs:
        assert got[k][1] == ref[k][1] > 0
        assert np.array_equal(got[k][0], ref[k][0]), k
