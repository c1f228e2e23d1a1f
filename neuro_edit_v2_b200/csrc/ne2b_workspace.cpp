// ne2b_workspace.cpp — see ne2b_workspace.h.
#include "ne2b_workspace.h"

#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>

namespace ne2b {
namespace {

struct Kept {
    std::mutex mu;
    std::map<int, cudaMemPool_t> pools;  // by device
    void *pin = nullptr;
    size_t pin_cap = 0;
};
Kept &kept() {
    static Kept *k = new Kept;  // never destroyed: a fit may end after the statics
    return *k;
}

cudaMemPool_t fit_pool(int device) {
    Kept &k = kept();
    std::lock_guard<std::mutex> lk(k.mu);
    auto it = k.pools.find(device);
    if (it != k.pools.end()) return it->second;
    cudaMemPoolProps props;
    memset(&props, 0, sizeof props);
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    uint64_t keep = kPoolKeep;
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) cudaGetLastError();
    k.pools[device] = pool;
    return pool;
}

}  // namespace

cudaError_t device_alloc(void **p, size_t bytes, cudaStream_t st) {
    cudaError_t e = cudaMallocAsync(p, bytes, st);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    release_workspaces();
    return cudaMallocAsync(p, bytes, st);
}

cudaError_t workspace_alloc(void **p, size_t bytes, int device, cudaStream_t st) {
    if (cudaMemPool_t pool = fit_pool(device)) {
        if (cudaMallocFromPoolAsync(p, bytes, pool, st) == cudaSuccess) return cudaSuccess;
        cudaGetLastError();
    }
    return device_alloc(p, bytes, st);
}

void release_workspaces() {
    Kept &k = kept();
    std::lock_guard<std::mutex> lk(k.mu);
    for (auto &e : k.pools)
        if (cudaMemPoolTrimTo(e.second, 0) != cudaSuccess) cudaGetLastError();
    if (k.pin && cudaFreeHost(k.pin) != cudaSuccess) cudaGetLastError();
    k.pin = nullptr;
    k.pin_cap = 0;
}

void *HostWorkspace::get(size_t bytes) {
    if (bytes <= kPinnedKeep) {
        Kept &k = kept();
        {
            std::lock_guard<std::mutex> lk(k.mu);
            if (k.pin_cap >= bytes) {
                std::swap(p_, k.pin);
                std::swap(cap_, k.pin_cap);
            }
        }
        if (!p_) {
            if (cudaHostAlloc(&p_, bytes, cudaHostAllocPortable) == cudaSuccess) {
                cap_ = bytes;
            } else {
                cudaGetLastError();
                p_ = nullptr;
            }
        }
        pinned_ = p_ != nullptr;
    }
    if (!p_) p_ = malloc(bytes);
    return p_;
}

HostWorkspace::~HostWorkspace() {
    if (!pinned_) {
        free(p_);
        return;
    }
    {
        Kept &k = kept();
        std::lock_guard<std::mutex> lk(k.mu);
        if (cap_ >= k.pin_cap) {
            std::swap(p_, k.pin);
            std::swap(cap_, k.pin_cap);
        }
    }
    if (p_ && cudaFreeHost(p_) != cudaSuccess) cudaGetLastError();
}

}  // namespace ne2b
