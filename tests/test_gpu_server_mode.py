"""NE2B_KERNEL=resident in the environment does not reach a server: a request
past what the resident kernel holds is served, with the same counts."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import hashlib
import numpy as np
import neuro_edit_v2_b200 as nb
from neuro_edit_v2_b200 import workloads as W

n, steps = 2_300_000, 40
rng = np.random.default_rng(1)
net = nb.from_synapses(np.zeros(n, np.uint8), np.tile(np.array([0.02, 0.2, -65.0, 8.0], np.float32), (n, 1)),
                       np.zeros(n, np.uint8), rng.integers(0, n, 5000), rng.integers(0, n, 5000),
                       rng.random(5000) * 3.0, rng.uniform(0.1, 0.5, 5000))
net = W.with_inputs(net, 2, 24, 12.0, rng)
srv = nb.Server(neuron_capacity=1 << 22, synapse_capacity=1 << 20, ring_capacity=1 << 26, max_requests=2,
                steps_per_launch=20)
cfg = nb.default_config(int_weights=1, window_steps=20, max_windows=2, noise_rate_hz=400.0, noise_kick_mv=30.0)
rid = srv.submit(net, cfg, np.ones((steps, 2), np.float32), steps)
while srv.stats()["active"]:
    srv.step()
counts, total = srv.take(rid)
assert total > 0
print(total, hashlib.sha256(counts.tobytes()).hexdigest())
"""


def test_a_server_does_not_take_the_resident_mode():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for mode in (None, "resident"):
        env = {k: v for k, v in os.environ.items() if k != "NE2B_KERNEL"}
        if mode:
            env["NE2B_KERNEL"] = mode
        r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, env=env, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        out.append(r.stdout.split())
    assert out[0] == out[1]
