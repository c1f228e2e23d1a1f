// ne2b_workspace.h — the readout fits' host memory (ne2b_workspace.cpp): one
// pinned buffer of up to kPinnedKeep stays for the next fit.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace ne2b {

constexpr size_t kPinnedKeep = (size_t)64 << 20;

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
