"""Builds from a synapse list when the device has no room for what only the
quicker way needs.  A preloaded allocator refuses allocations of given sizes
(so many times each); the network is the one that the host builds."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REFUSER = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
typedef int (*alloc_fn)(void **, size_t, void *);
/* REFUSE="bytes:times:after,..." : so many, after so many that are served */
int cudaMallocAsync(void **p, size_t n, void *st) {
    static alloc_fn real;
    static size_t size[8];
    static int left[8], after[8], count = -1;
    if (!real) real = (alloc_fn)dlsym(RTLD_NEXT, "cudaMallocAsync");
    if (count < 0) {
        count = 0;
        const char *s = getenv("REFUSE");
        while (s && *s && count < 8 && sscanf(s, "%zu:%d:%d", &size[count], &left[count], &after[count]) >= 2) {
            ++count;
            s = strchr(s, ',');
            if (s) ++s;
        }
    }
    for (int k = 0; k < count; ++k)
        if (size[k] == n && after[k] > 0) --after[k];
        else if (size[k] == n && left[k] > 0) {
            --left[k];
            fprintf(stderr, "refused %zu\n", n);
            return 2; /* cudaErrorMemoryAllocation */
        }
    return real(p, n, st);
}
"""
CHILD = r"""
import numpy as np, torch
import neuro_edit_v2_b200 as nb
n, e = 3000, 70001
rng = np.random.default_rng(1)
src, tgt = (rng.integers(0, n, e).astype(np.uint32) for _ in range(2))
w = rng.uniform(-1.0, 1.0, e).astype(np.float32)
d = rng.uniform(0.1, 15.0, e).astype(np.float32)
kind = (rng.random(n) < 0.2).astype(np.uint8)
params = np.tile(np.array([0.02, 0.2, -65.0, 8.0], np.float32), (n, 1))
cfg = nb.default_config(int_weights=1)
on_gpu = [torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).cuda() for x in (src, tgt, w, d)]
on_gpu = [x.view(torch.uint32) if x.dtype == torch.int32 else x for x in on_gpu]
dev = nb.B200Sim.from_synapses(np.zeros(n, np.uint8), params, kind, *on_gpu, cfg)
host = nb.B200Sim(nb.from_synapses(np.zeros(n, np.uint8), params, kind, src, tgt, w, d, dt_ms=cfg.dt_ms), cfg)
for x, y in zip(host.read_csr(), dev.read_csr()):
    assert np.array_equal(x, y)
print("ok")
"""
E = 70001


@pytest.fixture(scope="module")
def refuser(tmp_path_factory):
    d = tmp_path_factory.mktemp("refuse")
    (d / "refuse.c").write_text(REFUSER)
    subprocess.run(["gcc", "-shared", "-fPIC", str(d / "refuse.c"), "-o", str(d / "refuse.so"), "-ldl"], check=True)
    return str(d / "refuse.so")


@pytest.mark.parametrize("sizes", [
    [4 * E],            # the places
    [16 * E],           # the scratch of the records
    [8 * E],            # the net's own records, as long as the places are held
])
def test_the_net_is_built_without_the_optional_memory(refuser, sizes):
    # an allocation is tried twice: what the fits keep is given back in between
    env = dict(os.environ, LD_PRELOAD=refuser, REFUSE=",".join(f"{s}:2" for s in sizes))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
    assert all(f"refused {s}" in r.stderr for s in sizes)


TUNE = r"""
import torch
import numpy as np
import neuro_edit_v2_b200 as nb
net = nb.random_kout(5000, 20, 3)
sims = [nb.B200Sim(net, int_weights=1, noise_rate_hz=300.0) for _ in range(2)]
for s in sims:
    s.run_steps(50)
a = sims[1]
a.set_tile_shape(256, 4)
try:
    a.autotune(64)
except nb.Ne2bError as e:
    assert "ENOMEM" in str(e)
    print("refused")
t = a.tiling()
assert (t["runs"], t["block"], t["neurons_per_thread"]) == ("stream", 256, 4), t
for s in sims:
    s.run_steps(300)
assert np.array_equal(a.v().view(np.uint32), sims[0].v().view(np.uint32)) and a.spikes_total() > 0
print("ok")
"""


def test_autotune_without_room_for_its_snapshot_keeps_the_tile_shape(refuser):
    # 8 bytes per neuron: the lifetime counts, allocated with each sim and then by the snapshot
    env = dict(os.environ, LD_PRELOAD=refuser, REFUSE=f"{8 * 5056}:2:2")  # 5000 neurons in whole words of 64
    r = subprocess.run([sys.executable, "-c", TUNE], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["refused", "ok"], r.stdout + r.stderr
