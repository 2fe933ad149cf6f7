// Device memory of the one-shot host-buffer call, kept between calls.
//
// A call needs one block for weights, activations, bias and outputs.  cudaMalloc + cudaFree of it cost
// 0.7 ms at best and several where other work is in flight (cudaFree waits for the whole device),
// against 0.55 ms for the copy of a 9.4 MB weight: blocks are therefore kept, up to kKeepBytes and
// kSlots in a CUDA context, and handed from call to call.  A block belongs to one call at a time (several
// threads get several blocks) and to the context that it was allocated in; nothing of its content
// is ever read by a later call.  cogni_qmm_release_host_workspaces gives the idle ones back, and so does
// a call for which the device has no memory left.
//
// Host code only (no kernels, nothing but the runtime's C API): tests/cpp runs it on a CPU against a
// device that is made up.
#include "host_workspace.cuh"

#include <cuda.h>
#include <mutex>
#include <new>

namespace cogni {

// The entries form a list that only grows; one whose block has been given back is used again.  What a
// destroyed context leaves behind is its entries alone, a few words of host memory: its blocks went with it,
// they are never touched again (its id never comes back), and they count against no other context's limits.
struct HostSlot {
  void *p;
  size_t bytes;  // 0: free entry
  unsigned long long ctx;
  bool lent;
  HostSlot *next;
};

namespace {

constexpr int kSlots = 8;
constexpr size_t kKeepBytes = (size_t)256 << 20;  // idle and lent blocks of a context together
constexpr size_t kGrain = (size_t)2 << 20;

std::mutex g_mutex;
HostSlot *g_slots = nullptr;

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
    for (HostSlot *s = g_slots; ctx && s; s = s->next)
      if (s->bytes && !s->lent && s->ctx == ctx && n < kSlots) {
        idle[n++] = s->p;
        s->bytes = 0;
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
  w = HostWorkspace{nullptr, nullptr};
  cudaError_t e = cudaFree(nullptr);  // the runtime's context, where none is current yet
  if (e != cudaSuccess) return e;
  const size_t want = (bytes + kGrain - 1) / kGrain * kGrain;
  const unsigned long long ctx = context_id();
  void *old = nullptr;  // too small a block that makes room for this one
  if (ctx) {
    std::lock_guard<std::mutex> lock(g_mutex);
    HostSlot *fit = nullptr, *small = nullptr, *empty = nullptr;
    size_t held = 0;
    int own = 0;
    for (HostSlot *s = g_slots; s; s = s->next) {
      if (!s->bytes) {
        empty = s;
      } else if (s->ctx == ctx) {
        held += s->bytes;
        own++;
        if (s->lent) continue;
        if (s->bytes < want) small = s;
        else if (!fit || s->bytes < fit->bytes) fit = s;
      }
    }
    if (fit) {
      fit->lent = true;
      w = HostWorkspace{fit->p, fit};
      return cudaSuccess;
    }
    if (held - (small ? small->bytes : 0) + want <= kKeepBytes && (small || own < kSlots)) {
      HostSlot *slot = small ? small : empty;
      if (!slot && (slot = new (std::nothrow) HostSlot{})) {
        slot->next = g_slots;
        g_slots = slot;
      }
      if (slot) {
        if (small) old = small->p;
        slot->p = nullptr;  // reserved; the pointer is set on return
        slot->bytes = want;
        slot->ctx = ctx;
        slot->lent = true;
        w.slot = slot;
      }
    }
  }
  if (old) cudaFree(old);
  const size_t size = w.slot ? want : bytes;
  e = cudaMalloc(&w.p, size);
  if (e == cudaErrorMemoryAllocation) {  // what lies idle here may be what is missing
    int freed = 0;
    release_idle(ctx, &freed);
    cudaGetLastError();  // the next launch must not report this one
    if (freed) e = cudaMalloc(&w.p, size);
  }
  if (e != cudaSuccess) {
    if (w.slot) {
      std::lock_guard<std::mutex> lock(g_mutex);
      w.slot->bytes = 0;
    }
    w = HostWorkspace{nullptr, nullptr};
  }
  return e;
}

// keep = false: the call failed, its block is not lent again
void host_workspace_return(HostWorkspace &w, bool keep) {
  if (!w.p) return;
  if (w.slot) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (keep) {
      w.slot->p = w.p;
      w.slot->lent = false;
    } else {
      w.slot->bytes = 0;
    }
  }
  if (!w.slot || !keep) cudaFree(w.p);
  w = HostWorkspace{nullptr, nullptr};
}

int host_workspace_release_idle() {
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    const HostSlot *s = g_slots;
    while (s && !s->bytes) s = s->next;
    if (!s) return 0;  // nothing is held: no context is made for this
  }
  cudaFree(nullptr);  // a thread without a context yet: the runtime's, as for a call
  return (int)release_idle(context_id(), nullptr);
}

}  // namespace cogni
