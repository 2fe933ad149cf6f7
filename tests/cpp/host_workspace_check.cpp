// The memory that the host-buffer call keeps (csrc/host_workspace.cu), on a device that is made up: a
// memory of fixed size whose blocks belong to the context that is current, and contexts that come and go.
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <string.h>

#include <map>
#include <vector>

#include "../../cogni_ml_b200/csrc/host_workspace.cuh"

namespace {

const size_t kMB = (size_t)1 << 20;
size_t capacity = (size_t)1 << 40, used = 0;
unsigned long long current = 0, runtime_context = 1;  // 0: no context is current on this thread
int mallocs = 0, bad_frees = 0;
cudaError_t last_error = cudaSuccess;
struct Block {
  size_t bytes;
  unsigned long long ctx;
};
std::map<void *, Block> blocks;
char *next_address = reinterpret_cast<char *>((size_t)1 << 40);

CUresult get_current(CUcontext *c) {
  *c = reinterpret_cast<CUcontext>(current);
  return CUDA_SUCCESS;
}
CUresult get_id(CUcontext c, unsigned long long *id) {
  *id = 100 + reinterpret_cast<unsigned long long>(c);
  return CUDA_SUCCESS;
}

void destroy_context() {  // with its memory; the next one that the runtime makes is another
  for (auto it = blocks.begin(); it != blocks.end();) {
    if (it->second.ctx == current) {
      used -= it->second.bytes;
      it = blocks.erase(it);
    } else {
      ++it;
    }
  }
  current = 0;
  runtime_context++;
}

int failures = 0;
void expect(bool ok, const char *what) {
  if (!ok) {
    printf("failed: %s\n", what);
    failures++;
  }
}
bool call(size_t bytes) {  // a whole call
  cogni::HostWorkspace w;
  if (cogni::host_workspace_take(bytes, w) != cudaSuccess) return false;
  cogni::host_workspace_return(w, true);
  return true;
}

}  // namespace

extern "C" {
cudaError_t cudaFree(void *p) {
  if (!current) current = runtime_context;
  if (!p) return cudaSuccess;
  auto it = blocks.find(p);
  if (it == blocks.end() || it->second.ctx != current) {
    bad_frees++;
    return cudaErrorInvalidValue;
  }
  used -= it->second.bytes;
  blocks.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t bytes) {
  if (!current) current = runtime_context;
  mallocs++;
  if (used + bytes > capacity) return last_error = cudaErrorMemoryAllocation;
  used += bytes;
  *p = next_address;
  next_address += bytes;
  blocks[*p] = Block{bytes, current};
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *q) {
  *f = !strcmp(name, "cuCtxGetId") ? reinterpret_cast<void *>(get_id) : reinterpret_cast<void *>(get_current);
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}

int main(int argc, char **argv) {
  const char *what = argc > 1 ? argv[1] : "";
  if (!strcmp(what, "memory")) {  // the device has room for the call, but not beside the idle blocks
    capacity = 300 * kMB;
    cogni::HostWorkspace a, b;
    expect(cogni::host_workspace_take(100 * kMB, a) == cudaSuccess, "first block");
    expect(cogni::host_workspace_take(120 * kMB, b) == cudaSuccess, "second block");
    cogni::host_workspace_return(a, true);
    cogni::host_workspace_return(b, true);
    expect(call(250 * kMB), "a call that fits the device without the idle blocks");
    expect(last_error == cudaSuccess, "no error left for the next launch to report");
    expect(!call(400 * kMB), "a call that does not fit the device");
    expect(last_error == cudaSuccess, "no error left after a failed call");
    expect(call(50 * kMB) && call(50 * kMB), "calls after it");
  } else if (!strcmp(what, "contexts")) {  // blocks are kept in a context however many were destroyed before it
    for (int i = 0; i < 40; i++) {
      expect(call(40 * kMB), "first call of a context");
      const int before = mallocs;
      expect(call(40 * kMB) && call(30 * kMB) && mallocs == before, "later calls of the context allocate nothing");
      destroy_context();
    }
    // several blocks at once, no more than eight and 256 MB of them kept
    std::vector<cogni::HostWorkspace> ws(12);
    for (auto &w : ws) expect(cogni::host_workspace_take(20 * kMB, w) == cudaSuccess, "one of twelve blocks");
    for (auto &w : ws) cogni::host_workspace_return(w, true);
    expect(blocks.size() == 8 && used == 160 * kMB, "eight blocks are kept");
    expect(call(240 * kMB) && used <= 256 * kMB, "256 MB are kept");
  } else if (!strcmp(what, "thread")) {  // a thread that has not used CUDA yet gives the idle blocks back
    expect(cogni::host_workspace_release_idle() == 0 && !current, "no context is made where nothing is held");
    expect(call(40 * kMB) && used == 40 * kMB, "a call keeps its block");
    current = 0;
    expect(cogni::host_workspace_release_idle() == 0 && used == 0, "the block is given back");
  } else {
    printf("unknown check %s\n", what);
    return 2;
  }
  expect(bad_frees == 0, "no free of another context's or an unknown block");
  if (!failures) printf("ok\n");
  return failures ? 1 : 0;
}
