"""The fits' device workspaces against a fake runtime: they come from a pool
of their own, the default pool when that has no room, and are given back when
asked and when another allocation of the library finds no room."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neuro_edit_v2_b200", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
SOURCE = r"""
#include "ne2b_workspace.cpp"
// a device of `room` bytes; what the fits' pool has been given stays its own
// until it is trimmed
static size_t room, pool_held;
static int pools, last, trims;
static uint64_t threshold;
static cudaError_t fail(cudaError_t e) { last = e; return e; }
extern "C" {
cudaError_t cudaGetLastError() { const cudaError_t e = (cudaError_t)last; last = 0; return e; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *q) {
    if (q->location.id > 7) return fail(cudaErrorNotSupported);
    ++pools;
    *p = (cudaMemPool_t)(uintptr_t)(0x100 + q->location.id);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *v) { threshold = *(uint64_t *)v; return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep) {
    ++trims;
    room += pool_held - keep;
    pool_held = keep;
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) {
    if (n > room) return fail(cudaErrorMemoryAllocation);
    room -= n;
    *p = (void *)1;
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
    if (n > room) return fail(cudaErrorMemoryAllocation);
    room -= n;
    pool_held += n;
    *p = (void *)2;
    return cudaSuccess;
}
void set_room(size_t n) { room = n; }
int pool_count() { return pools; }
int trim_count() { return trims; }
int last_error() { return last; }
size_t keeps() { return threshold; }
int fit_alloc(size_t n, int device, uintptr_t *where) {
    void *p = nullptr;
    const cudaError_t e = ne2b::workspace_alloc(&p, n, device, nullptr);
    *where = (uintptr_t)p;
    return e;
}
int net_alloc(size_t n) { void *p; return ne2b::device_alloc(&p, n, nullptr); }
void release() { ne2b::release_workspaces(); }
}
"""
NO_ROOM = 2


@pytest.fixture()
def lib(tmp_path):
    (tmp_path / "fake.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", CUDA,
                    str(tmp_path / "fake.cpp"), "-o", str(tmp_path / "libfake.so")], check=True)
    L = C.CDLL(str(tmp_path / "libfake.so"))
    L.set_room.argtypes = L.net_alloc.argtypes = [C.c_size_t]
    L.fit_alloc.argtypes = [C.c_size_t, C.c_int, C.POINTER(C.c_size_t)]
    L.keeps.restype = C.c_size_t
    return L


def fit(lib, n, device=0):
    where = C.c_size_t()
    return lib.fit_alloc(n, device, C.byref(where)), where.value


def test_a_pool_of_their_own_that_is_bounded_and_given_back(lib):
    lib.set_room(1000)
    assert fit(lib, 100) == (0, 2) and fit(lib, 100) == (0, 2) and fit(lib, 100, 1) == (0, 2)
    assert lib.pool_count() == 2 and lib.keeps() == 256 << 20
    lib.release()
    assert lib.trim_count() == 2


def test_default_pool_when_theirs_cannot_serve(lib):
    lib.set_room(1000)
    assert fit(lib, 100, 9) == (0, 1)  # no pool on this device
    assert lib.last_error() == 0


def test_a_net_gets_the_memory_that_fits_kept(lib):
    lib.set_room(1000)
    assert fit(lib, 900) == (0, 2)
    assert lib.net_alloc(500) == 0  # 100 left: what the fits kept is given back first
    assert lib.trim_count() == 1 and lib.last_error() == 0
    assert lib.net_alloc(600) == NO_ROOM
