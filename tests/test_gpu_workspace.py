"""The fits leave the device's default memory pool as it was, and give their
own memory back."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C
import numpy as np
import neuro_edit_v2_b200 as nb

rt = C.CDLL("libcudart.so.12")
pool, keep = C.c_void_p(), C.c_uint64()
THRESHOLD = 4


def kept():
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, THRESHOLD, C.byref(keep)) == 0
    return keep.value


def free():
    a, b = C.c_size_t(), C.c_size_t()
    assert rt.cudaMemGetInfo(C.byref(a), C.byref(b)) == 0
    return a.value


before = kept()
rng = np.random.default_rng(0)
x = rng.poisson(1.5, (600, 5000)).astype(np.float32)
lab = rng.integers(0, 2, 600).astype(np.uint32)
nb.fit_ridge_multi(x[:40, :40], lab[:40], 2, 1.0)
nb.release_workspaces()
room = free()
w = nb.fit_ridge_multi(x, lab, 2, 1.0)
nb.fit_ridge(x[:, :300], lab.astype(np.float32), 1.0)
assert kept() == before, (kept(), before)
held = room - free()
assert 0 < held <= 256 << 20, held
nb.release_workspaces()
assert room - free() < 8 << 20, (room, free())
assert np.array_equal(nb.fit_ridge_multi(x, lab, 2, 1.0), w)
print("ok")
"""


def test_fits_keep_to_their_own_pool():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", "import torch\n" + CHILD], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
