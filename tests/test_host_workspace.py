"""The fits' host memory against a fake runtime whose pinning fails: a fit is
served pageable memory when pinning is refused or the factor is larger than
what is kept pinned, leaves no error behind, and one pinned buffer goes from
fit to fit."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neuro_edit_v2_b200", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
SOURCE = r"""
#include "ne2b_workspace.cpp"
static bool refuse;
static int pinned, last;
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (refuse) { last = cudaErrorMemoryAllocation; return cudaErrorMemoryAllocation; }
    ++pinned;
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { --pinned; free(p); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = (cudaError_t)last; last = 0; return e; }
void set_refuse(int r) { refuse = r; }
int pinned_buffers() { return pinned; }
int last_error() { return last; }
void *make() { return new ne2b::HostWorkspace; }
void drop(void *w) { delete (ne2b::HostWorkspace *)w; }
void *get(void *w, size_t n) { return ((ne2b::HostWorkspace *)w)->get(n); }
int is_pinned(void *w) { return ((ne2b::HostWorkspace *)w)->pinned(); }
size_t keep() { return ne2b::kPinnedKeep; }
}
"""


@pytest.fixture()
def lib(tmp_path):
    (tmp_path / "fake.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", CUDA,
                    str(tmp_path / "fake.cpp"), "-o", str(tmp_path / "libfake.so")], check=True)
    L = C.CDLL(str(tmp_path / "libfake.so"))
    L.make.restype = L.get.restype = C.c_void_p
    L.keep.restype = C.c_size_t
    L.get.argtypes = [C.c_void_p, C.c_size_t]
    L.drop.argtypes = L.is_pinned.argtypes = [C.c_void_p]
    return L


def test_refused_pinning_falls_back_to_pageable_memory(lib):
    lib.set_refuse(1)
    w = lib.make()
    p = lib.get(w, 1 << 20)
    assert p and not lib.is_pinned(w) and lib.last_error() == 0
    C.memset(p, 1, 1 << 20)
    lib.drop(w)
    assert lib.pinned_buffers() == 0


def test_a_large_factor_is_not_pinned(lib):
    w = lib.make()
    p = lib.get(w, lib.keep() + 1)
    assert p and not lib.is_pinned(w) and lib.pinned_buffers() == 0
    lib.drop(w)


def test_one_buffer_is_kept(lib):
    a, b = lib.make(), lib.make()
    pa, pb = lib.get(a, 4096), lib.get(b, 1 << 16)  # two fits at once
    assert pa != pb and lib.pinned_buffers() == 2
    lib.drop(b)
    lib.drop(a)
    assert lib.pinned_buffers() == 1
    lib.set_refuse(1)
    c = lib.make()
    assert lib.get(c, 1 << 16) == pb and lib.is_pinned(c)  # the larger one stayed
    d = lib.make()
    assert lib.get(d, 1 << 16) and not lib.is_pinned(d)
    lib.drop(d)
    lib.drop(c)
    assert lib.pinned_buffers() == 1
