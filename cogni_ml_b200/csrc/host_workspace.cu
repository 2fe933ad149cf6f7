// Device memory of the one-shot host-buffer call, kept between calls.
//
// A call needs one block for weights, activations, bias and outputs.  cudaMalloc + cudaFree of it cost
// 0.7 ms at best and several where other work is in flight (cudaFree waits for the whole device),
// against 0.55 ms for the copy of a 9.4 MB weight: blocks are therefore kept, up to kKeepBytes and
// kSlots in all, and handed from call to call.  A block belongs to one call at a time (several
// threads get several blocks) and to the CUDA context that it was allocated in; nothing of its content
// is ever read by a later call.  cogni_qmm_release_host_workspaces gives the idle ones back, and so does
// a call for which the device has no memory left.
//
// Host code only (no kernels, nothing but the runtime's C API): tests/cpp runs it on a CPU against a
// device that is made up.
#include "host_workspace.cuh"

#include <cuda.h>
#include <mutex>


namespace cogni {
namespace {

constexpr int kSlots = 8;
constexpr size_t kKeepBytes = (size_t)256 << 20;  // idle and lent blocks of all contexts together
constexpr size_t kGrain = (size_t)2 << 20;

struct Slot {
  void *p;
  size_t bytes;
  unsigned long long ctx;
  bool lent;
};
std::mutex g_mutex;
Slot g_slots[kSlots];

// An id that no other context of the process ever has (a later context can reuse a handle); 0 if
// there is none.
unsigned long long context_id() {
  typedef CUresult (*GetCurrentFn)(CUcontext *);
  typedef CUresult (*GetIdFn)(CUcontext, unsigned long long *);
  auto entry = [](const char *name) {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return f;
  };
  static const GetCurrentFn get_current = reinterpret_cast<GetCurrentFn>(entry("cuCtxGetCurrent"));
  static const GetIdFn get_id = reinterpret_cast<GetIdFn>(entry("cuCtxGetId"));
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// Gives the idle blocks of context `ctx` (the current one) back; their number in *count.
cudaError_t release_idle(unsigned long long ctx, int *count) {
  void *idle[kSlots];
  int n = 0;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (Slot &s : g_slots)
      if (s.bytes && !s.lent && s.ctx == ctx) {
        idle[n++] = s.p;
        s = Slot{};
      }
  }
  cudaError_t first = cudaSuccess;
  for (int i = 0; i < n; i++) {
    const cudaError_t e = cudaFree(idle[i]);
    if (first == cudaSuccess) first = e;
  }
  if (count) *count = n;
  return first;
}

}  // namespace

cudaError_t host_workspace_take(size_t bytes, HostWorkspace &w) {
  w = HostWorkspace{nullptr, -1};
  cudaError_t e = cudaFree(nullptr);  // the runtime's context, where none is current yet
  if (e != cudaSuccess) return e;
  const size_t want = (bytes + kGrain - 1) / kGrain * kGrain;
  const unsigned long long ctx = context_id();
  void *old = nullptr;  // too small a block that makes room for this one
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    int fit = -1, small = -1, empty = -1;
    size_t held = 0;
    for (int i = 0; i < kSlots; i++) {
      const Slot &s = g_slots[i];
      held += s.bytes;
      if (!s.bytes) empty = i;
      else if (!s.lent && s.ctx == ctx && s.bytes >= want && (fit < 0 || s.bytes < g_slots[fit].bytes)) fit = i;
      else if (!s.lent && s.ctx == ctx && s.bytes < want) small = i;
    }
    if (ctx && fit >= 0) {
      g_slots[fit].lent = true;
      w = HostWorkspace{g_slots[fit].p, fit};
      return cudaSuccess;
    }
    const int slot = small >= 0 ? small : empty;
    if (ctx && slot >= 0 && held - g_slots[slot].bytes + want <= kKeepBytes) {
      old = g_slots[slot].p;
      g_slots[slot] = Slot{nullptr, want, ctx, true};  // reserved; the pointer is set on return
      w.slot = slot;
    }
  }
  if (old) cudaFree(old);
  const size_t size = w.slot >= 0 ? want : bytes;
  e = cudaMalloc(&w.p, size);
  if (e == cudaErrorMemoryAllocation) {  // what lies idle here may be what is missing
    int freed = 0;
    release_idle(ctx, &freed);
    cudaGetLastError();  // the next launch must not report this one
    if (freed) e = cudaMalloc(&w.p, size);
  }
  if (e != cudaSuccess) {
    if (w.slot >= 0) {
      std::lock_guard<std::mutex> lock(g_mutex);
      g_slots[w.slot] = Slot{};
    }
    w = HostWorkspace{nullptr, -1};
  }
  return e;
}

// keep = false: the call failed, its block is not lent again
void host_workspace_return(HostWorkspace &w, bool keep) {
  if (!w.p) return;
  if (w.slot >= 0) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (keep) {
      g_slots[w.slot].p = w.p;
      g_slots[w.slot].lent = false;
    } else {
      g_slots[w.slot] = Slot{};
    }
  }
  if (w.slot < 0 || !keep) cudaFree(w.p);
  w = HostWorkspace{nullptr, -1};
}

int host_workspace_release_idle() { return (int)release_idle(context_id(), nullptr); }

}  // namespace cogni
