// ne2b_workspace.cpp — see ne2b_workspace.h.
#include "ne2b_workspace.h"

#include <stdlib.h>

#include <algorithm>
#include <mutex>

namespace ne2b {
namespace {

struct Kept {
    std::mutex mu;
    void *pin = nullptr;
    size_t pin_cap = 0;
};
Kept &kept() {
    static Kept *k = new Kept;  // never destroyed: a fit may end after the statics
    return *k;
}

}  // namespace

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
