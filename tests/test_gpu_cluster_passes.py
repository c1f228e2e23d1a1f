"""The cluster kernel where a block has more neurons than threads (the state
waits in shared memory between the passes of a hop): hops of one step and of
several, AdEx rows, input streams, windows that cut hops short, records, the
last pass ragged; and more nets than the device holds at once.  Every window
count and state bit against the oracle."""
import numpy as np
import pytest

import pyoracle as O
import neuro_edit_v2_b200 as nb

pytestmark = pytest.mark.gpu
ADEX = np.array([281.0, 30.0, -70.6, -50.4, 2.0, 4.0, 144.0, 80.5, -70.6, 20.0], np.float32)


def net(n, lo_ms, hi_ms, adex, k=5):
    onet = O.ONet()
    rng = np.random.default_rng(n)
    for i in range(n):
        onet.add_neuron(0.0, 0.0, 0.0, O.EXC if i < 0.8 * n else O.INH)
        if adex and i % 3 == 0:
            onet.set_model(i, O.ADEX, ADEX)
    tgt, w, d = rng.integers(0, n, (n, k)), rng.uniform(0.5, 3.0, (n, k)), rng.uniform(lo_ms, hi_ms, (n, k))
    for i in range(n):
        for q in range(k):
            onet.push_synapse(i, int(tgt[i, q]), float(w[i, q]), float(d[i, q]))
    for _ in range(2):
        onet.add_input([(int(t), 30.0) for t in rng.integers(0, n, 200)])
    return onet


def check(b, j, onet, kw, stream, windows, win):
    o = O.OSim(onet, O.cfg(record_spikes=1, spike_record_steps=win, exp_mode=1, **kw))
    for i in range(2):
        o.play_input(i, stream[:, i])
    for w in range(windows):
        o.run_steps(win)
        assert np.array_equal(b.window_counts(j, w), o.spike_counts(win)), f"net {j} window {w}"
    assert b.spikes_total(j) == o.spikes_total() > 0
    for slot in (0, 1):
        assert np.array_equal(b.state(j, slot).view(np.uint32), o.state(slot).view(np.uint32)), f"net {j}"


@pytest.mark.parametrize("record", [0, 1])
@pytest.mark.parametrize("sizes, lo_ms, hi_ms, adex", [
    ((17013, 20005), 0.1, 1.5, False),  # hop 1, two passes
    ((17013, 17500), 0.1, 1.5, True),
    ((17013, 33005), 0.6, 4.0, True),   # hop 6, two and three passes
])
def test_more_neurons_than_threads(sizes, lo_ms, hi_ms, adex, record):
    onets = [net(n, lo_ms, hi_ms, adex) for n in sizes]
    kw = [dict(int_weights=1, noise_rate_hz=400.0, noise_kick_mv=20.0, seed=5 + j) for j in range(2)]
    b = nb.Batch([x.flat() for x in onets],
                 [nb.default_config(window_steps=7, max_windows=30, record_spikes=record, **c) for c in kw])
    streams = [(np.random.default_rng(j).random((210, 2)) < 0.1).astype(np.float32) for j in range(2)]
    for j, x in enumerate(streams):
        for i in range(2):
            b.play_input(j, i, x[:, i])
    assert b.running_kernel() == "cluster"
    for steps in (1, 5, 64, 140):
        b.run_steps(steps)
    for j, x in enumerate(onets):
        check(b, j, x, kw[j], streams[j], 30, 7)


def test_more_nets_than_the_device_holds():
    onet = net(8003, 0.6, 4.0, False)
    count, kw = 170, [dict(int_weights=1, noise_rate_hz=400.0, noise_kick_mv=20.0, seed=3 + j) for j in range(170)]
    flat = onet.flat()
    b = nb.Batch([flat] * count, [nb.default_config(window_steps=10, max_windows=12, **c) for c in kw])
    assert b.running_kernel() == "cluster"
    for steps in (3, 117):
        b.run_steps(steps)
    zero = np.zeros((1, 2), np.float32)
    for j in (0, 84, 169):
        check(b, j, onet, kw[j], zero, 12, 10)
