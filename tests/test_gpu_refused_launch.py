"""A cluster launch that the runtime refuses: the launches already made on
other streams are still joined to the engine's stream, the error is reported,
and the batch runs on afterwards.  A preloaded runtime refuses the launch
before it reaches the device."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
REFUSER = r"""
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
#define REAL(name) ((decltype(&name))dlsym(RTLD_NEXT, #name))
static bool noisy() { return getenv("REFUSE_LAUNCH") != nullptr; }
extern "C" {
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    static int clusters = 0;
    if (noisy() && c->numAttrs == 1 && c->attrs[0].id == cudaLaunchAttributeClusterDimension) {
        if (++clusters == atoi(getenv("REFUSE_LAUNCH"))) {
            fprintf(stderr, "refused\n");
            return cudaErrorLaunchOutOfResources;
        }
        fprintf(stderr, "launch %p\n", (void *)c->stream);
    }
    return REAL(cudaLaunchKernelExC)(c, f, args);
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (noisy()) fprintf(stderr, "record %p %p\n", (void *)e, (void *)s);
    return REAL(cudaEventRecord)(e, s);
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
    if (noisy()) fprintf(stderr, "wait %p %p\n", (void *)s, (void *)e);
    return REAL(cudaStreamWaitEvent)(s, e, f);
}
}
"""
CHILD = r"""
import sys
import torch  # loads the runtime for every library of the process
import numpy as np
import neuro_edit_v2_b200 as nb
nets = [nb.liquid(s, seed=k) for k, s in enumerate((6, 12, 17, 25))]
cfgs = [nb.default_config(int_weights=1, noise_rate_hz=200.0, seed=k) for k in range(4)]
a, b = nb.Batch(nets, cfgs), nb.Batch(nets, cfgs)
b.set_kernel_mode(nb.KERNEL_STREAM)
assert a.running_kernel() == "cluster"
print("stream", a.stream_handle(), file=sys.stderr, flush=True)
try:
    a.run_steps(20)
except nb.Ne2bError as e:
    print("error", flush=True)
print("end", file=sys.stderr, flush=True)
a.reset_state()
for x in (a, b):
    x.run_steps(100)
for j in range(4):
    assert a.spikes_total(j) == b.spikes_total(j) > 0
    assert np.array_equal(a.state(j, 0).view(np.uint32), b.state(j, 0).view(np.uint32))
print("ok")
"""


@pytest.mark.parametrize("which", [1, 2, 3, 4])
def test_the_launches_made_are_joined(which, tmp_path):
    (tmp_path / "refuse.cpp").write_text(REFUSER)
    subprocess.run(["g++", "-shared", "-fPIC", "-I", CUDA, str(tmp_path / "refuse.cpp"), "-o",
                    str(tmp_path / "refuse.so"), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(tmp_path / "refuse.so"), REFUSE_LAUNCH=str(which))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["error", "ok"], r.stdout + r.stderr
    log = r.stderr[: r.stderr.index("end\n")]
    main = int(re.search(r"stream (\d+)", log).group(1))
    made = [int(x, 16) for x in re.findall(r"launch (\S+)", log)]
    assert len(made) == which - 1
    after = log[log.index("refused"):]
    joined = {int(e, 16): int(s, 16) for e, s in re.findall(r"record (\S+) (\S+)", after)}
    waited = {int(e, 16) for s, e in re.findall(r"wait (\S+) (\S+)", after) if int(s, 16) == main}
    for s in made:
        assert s == main or any(joined[e] == s for e in waited if e in joined)
