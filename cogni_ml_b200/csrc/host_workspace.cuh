// Device memory of the host-buffer call (host_workspace.cu), lent to one call at a time.
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>

namespace cogni {

struct HostSlot;
struct HostWorkspace {
  void *p;
  HostSlot *slot;  // nullptr: not kept
};
cudaError_t host_workspace_take(size_t bytes, HostWorkspace &w);
void host_workspace_return(HostWorkspace &w, bool keep);
int host_workspace_release_idle();

}  // namespace cogni
