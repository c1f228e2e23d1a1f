// ne2b_workspace.h — memory that the readout fits keep from one call to the
// next (ne2b_workspace.cpp): a memory pool per device, apart from the default
// pool, which keeps up to kPoolKeep, and one pinned host buffer of up to
// kPinnedKeep.  Both are given back by release_workspaces, which the library
// also calls itself when a device allocation of its own finds no room.
// Without them each fit maps its workspaces and pins its host copy anew:
// 5.6 instead of 3.6 ms at 1000 x 4320, 3.8 instead of 2.4 ms at 1200 x 1080.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace ne2b {

constexpr uint64_t kPoolKeep = (uint64_t)256 << 20;
constexpr size_t kPinnedKeep = (size_t)64 << 20;

// Device memory of the default pool on `st`; with no room, once more after
// release_workspaces.
cudaError_t device_alloc(void **p, size_t bytes, cudaStream_t st);
// Device memory for a fit on `device`: of the fits' own pool, or with no room
// there of the default pool.  Freed with cudaFreeAsync.
cudaError_t workspace_alloc(void **p, size_t bytes, int device, cudaStream_t st);
// Gives back what no running fit uses (any thread, any time).
void release_workspaces();

// A fit's host copy of its factor: pinned up to kPinnedKeep, so that the copy
// runs at the link's rate and no fresh pages are faulted in; pageable past
// that (pinning takes 0.25 ms per MB, more than the copy gains) and where
// pinning is refused.  A fit that finds the kept buffer taken (another
// thread's) or too small pins its own.
class HostWorkspace {
  public:
    HostWorkspace() = default;
    HostWorkspace(const HostWorkspace &) = delete;
    HostWorkspace &operator=(const HostWorkspace &) = delete;
    ~HostWorkspace();
    void *get(size_t bytes);  // once; null when the host has no memory
    bool pinned() const { return pinned_; }

  private:
    void *p_ = nullptr;
    size_t cap_ = 0;
    bool pinned_ = false;
};

}  // namespace ne2b
