// See fake_cudart.hpp. Defines the runtime's entry points that capi.cu uses and the
// kernel launchers that kernels.cu would define.
#include "fake_cudart.hpp"

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include <sys/mman.h>

#ifndef __CUDA_ARCH__  // host code only: the device pass has declarations of its own

using namespace optx;

namespace fake {

int devices = 2;
thread_local int current = 0;
bool frees_fail = false;
int faults = 0, mallocs = 0, instantiations = 0, history_block = 0;
std::function<void()> on_shares;
std::vector<Run> runs;

namespace {

struct Block {
  size_t bytes;
  int device;  // -1: pinned host memory
};
std::mutex mu;
std::map<uintptr_t, Block> blocks;
thread_local cudaError_t last = cudaSuccess;

cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

size_t pages(size_t b) { return (b + 4095u) & ~size_t(4095); }

cudaError_t alloc(void** p, size_t bytes, int device) {
  void* q = mmap(nullptr, pages(bytes ? bytes : 1), PROT_READ | PROT_WRITE,
                 MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (q == MAP_FAILED) return set(cudaErrorMemoryAllocation);
  std::lock_guard<std::mutex> lk(mu);
  blocks[reinterpret_cast<uintptr_t>(q)] = {bytes ? bytes : 1, device};
  *p = q;
  return cudaSuccess;
}

cudaError_t release(void* p) {
  if (p == nullptr) return cudaSuccess;
  if (frees_fail) return set(cudaErrorInvalidValue);
  std::lock_guard<std::mutex> lk(mu);
  const auto it = blocks.find(reinterpret_cast<uintptr_t>(p));
  if (it == blocks.end()) return set(cudaErrorInvalidValue);
  munmap(p, pages(it->second.bytes));
  blocks.erase(it);
  return cudaSuccess;
}

const Block* find(const void* p) {
  const auto a = reinterpret_cast<uintptr_t>(p);
  auto it = blocks.upper_bound(a);
  if (it == blocks.begin()) return nullptr;
  --it;
  return a < it->first + it->second.bytes ? &it->second : nullptr;
}

// True when every pointer that is not null is memory of the current device.
bool mine(std::initializer_list<const void*> ps) {
  std::lock_guard<std::mutex> lk(mu);
  for (const void* p : ps) {
    if (p == nullptr) continue;
    const Block* b = find(p);
    if (b == nullptr || b->device != current) return false;
  }
  return true;
}

struct Stream {
  int device;
};
struct Event {
  int device;
};
Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
Event* of(cudaEvent_t e) { return reinterpret_cast<Event*>(e); }
int device_of(cudaStream_t s) { return s == nullptr ? current : of(s)->device; }

cudaError_t launchable(cudaStream_t s, std::initializer_list<const void*> ps) {
  if (device_of(s) != current) return set(cudaErrorInvalidResourceHandle);
  if (!mine(ps)) {
    ++faults;
    return set(cudaErrorIllegalAddress);
  }
  return cudaSuccess;
}

void write_records(const DevRecords& r, uint64_t first_id, uint64_t lo, uint64_t hi) {
  for (uint64_t i = lo; i < hi; ++i) {
    const uint64_t id = first_id + i;
    r.fate[i] = fate(id);
    r.n_boundary[i] = word(id);
    r.n_scatter[i] = word(id + 1);
    float* f[5] = {r.t + i, r.x + i, r.y + i, r.z + i, r.path + i};
    for (uint32_t k = 0; k < 5; ++k) *f[k] = static_cast<float>((word(id) >> 8) + k);
  }
}

cudaError_t prep(const WaveArgs& a, WaveCtrl* c, cudaStream_t st) {
  const cudaError_t e = launchable(st, {c, a.tally, a.grad});
  if (e != cudaSuccess) return e;
  const unsigned gs = c->gs_error;
  std::memset(c, 0, sizeof(*c));
  c->gs_error = gs;
  c->active = 1;
  return cudaSuccess;
}

cudaError_t wave(const DevParams& P, const WaveArgs& a, WaveCtrl* c, cudaStream_t st) {
  const DevRecords& r = a.rec;
  const cudaError_t e = launchable(st, {c, a.tally, a.grad, a.params, a.offsets, a.qa, a.qb, r.fate, r.n_boundary,
                                        r.n_scatter, r.t, r.x, r.y, r.z, r.path});
  if (e != cudaSuccess) return e;
  runs.push_back({a, P});
  if (r.fate != nullptr) write_records(r, a.first_id, a.item_lo, a.total);
  c->active = 0;
  c->wave = 1;
  return cudaSuccess;
}

// Functions of the kernels as the runtime sees them.
char wave_fn, prep_fn, sorted_fn, sorted_prep;

struct Node {
  const void* func;
  WaveArgs args;
  DevParams p0;
  WaveCtrl* ctrl;
};
Node read(const cudaKernelNodeParams* p) {
  Node n{};
  n.func = p->func;
  if (p->func == &wave_fn) {
    n.p0 = *static_cast<const DevParams*>(p->kernelParams[0]);
    n.args = *static_cast<const WaveArgs*>(p->kernelParams[1]);
    n.ctrl = *static_cast<WaveCtrl**>(p->kernelParams[2]);
  } else {
    n.args = *static_cast<const WaveArgs*>(p->kernelParams[0]);
    n.ctrl = *static_cast<WaveCtrl**>(p->kernelParams[1]);
  }
  return n;
}
struct Graph {
  std::vector<Node*> nodes;  // the body's too
  Graph* body = nullptr;
};
struct Exec {
  std::map<Node*, Node> nodes;
};
Graph* of(cudaGraph_t g) { return reinterpret_cast<Graph*>(g); }
Exec* of(cudaGraphExec_t g) { return reinterpret_cast<Exec*>(g); }

}  // namespace

size_t device_bytes() {
  std::lock_guard<std::mutex> lk(mu);
  size_t n = 0;
  for (const auto& b : blocks)
    if (b.second.device >= 0) n += b.second.bytes;
  return n;
}
bool stale_error() { return last != cudaSuccess; }

}  // namespace fake

using namespace fake;

extern "C" {

cudaError_t cudaGetDeviceCount(int* n) { *n = devices; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorIllegalAddress ? "illegal address" : "refused"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0);
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof(*p)); return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof(*a));
  a->sharedSizeBytes = 600;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t bytes) { ++mallocs; return alloc(p, bytes, current); }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { return alloc(p, bytes, -1); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeHost(void* p) { return release(p); }
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind) { std::memcpy(to, from, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(to, from, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::lock_guard<std::mutex> lk(mu);
  std::memset(a, 0, sizeof(*a));
  const Block* b = find(p);
  a->type = b == nullptr ? cudaMemoryTypeUnregistered : (b->device < 0 ? cudaMemoryTypeHost : cudaMemoryTypeDevice);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) { *p = const_cast<void*>(symbol); return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(new Stream{current});
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete of(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return frees_fail ? set(cudaErrorInvalidResourceHandle) : cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(new Event{current}); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  if (frees_fail) return set(cudaErrorInvalidResourceHandle);
  delete of(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return of(e)->device == device_of(s) ? cudaSuccess : set(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }

cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) { *g = reinterpret_cast<cudaGraph_t>(new Graph()); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  if (frees_fail) return set(cudaErrorInvalidResourceHandle);
  for (Node* n : of(g)->nodes) delete n;
  if (of(g)->body) {
    for (Node* n : of(g)->body->nodes) delete n;
    delete of(g)->body;
  }
  delete of(g);
  return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t g, unsigned, unsigned) {
  *h = reinterpret_cast<cudaGraphConditionalHandle>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t*, size_t,
                                   const cudaKernelNodeParams* p) {
  Node* k = new Node(read(p));
  of(g)->nodes.push_back(k);
  *n = reinterpret_cast<cudaGraphNode_t>(k);
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
  of(g)->body = new Graph();
  static thread_local cudaGraph_t body;
  body = reinterpret_cast<cudaGraph_t>(of(g)->body);
  p->conditional.phGraph_out = &body;
  *n = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  ++instantiations;
  Exec* e = new Exec();
  for (Node* n : of(g)->nodes) e->nodes[n] = *n;
  if (of(g)->body)
    for (Node* n : of(g)->body->nodes) e->nodes[n] = *n;
  *x = reinterpret_cast<cudaGraphExec_t>(e);
  return cudaSuccess;
}
cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t x, cudaGraphNode_t n, const cudaKernelNodeParams* p) {
  const auto it = of(x)->nodes.find(reinterpret_cast<Node*>(n));
  if (it == of(x)->nodes.end()) return set(cudaErrorInvalidValue);
  it->second = read(p);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  if (frees_fail) return set(cudaErrorInvalidResourceHandle);
  delete of(x);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t st) {
  for (const void* f : {static_cast<const void*>(&prep_fn), static_cast<const void*>(&wave_fn)})
    for (const auto& kv : of(x)->nodes) {
      const Node& n = kv.second;
      if (n.func != f) continue;
      const cudaError_t e = f == &prep_fn ? prep(n.args, n.ctrl, st) : wave(n.p0, n.args, n.ctrl, st);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

// What nvcc's host code calls to register and launch the kernels of capi.cu.
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, CUstream_st*) { return 1; }  // not launched
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"

namespace optx {
#define OPTX_FAKE_LAUNCHERS(NS)                                                                                       \
  namespace NS {                                                                                                      \
  int history_tally_blocks_per_sm(int, size_t) { return 1; }                                                          \
  cudaError_t launch_history_tally(const DevParams&, const TallyDev&, uint64_t, uint64_t n, unsigned long long* t,    \
                                   int block, int, cudaStream_t st) {                                                 \
    history_block = block;                                                                                            \
    const cudaError_t e = launchable(st, {t});                                                                        \
    if (e == cudaSuccess) t[0] += n;                                                                                  \
    return e;                                                                                                         \
  }                                                                                                                   \
  cudaError_t launch_wave_prep(const WaveArgs& a, WaveCtrl* c, int, int, cudaStream_t st) { return prep(a, c, st); }  \
  const void* wave_prep_fn() { return &prep_fn; }                                                                     \
  const void* wave_kernel_fn(int, int, int) { return &wave_fn; }                                                      \
  int wave_blocks_per_sm(int, int, int, int, size_t) { return 3; }                                                    \
  cudaError_t wave_set_smem(int, int, int, size_t) { return cudaSuccess; }                                            \
  cudaError_t launch_wave(int, int, int, const DevParams& P, const WaveArgs& a, WaveCtrl* c, int, int, size_t,        \
                          cudaStream_t st) {                                                                          \
    return wave(P, a, c, st);                                                                                         \
  }                                                                                                                   \
  cudaError_t launch_shares(int, const DevParams&, const WaveArgs& a, WaveCtrl* c, int, size_t, int,                  \
                            cudaStream_t st) {                                                                        \
    const DevRecords& r = a.rec;                                                                                      \
    const cudaError_t e = launchable(st, {c, a.tally, r.fate, r.n_boundary, r.n_scatter, r.t, r.x, r.y, r.z, r.path}); \
    if (e != cudaSuccess) return e;                                                                                   \
    if (const auto f = on_shares) f();                                                                                \
    if (r.fate != nullptr) write_records(r, a.first_id, 0, a.total);                                                  \
    if (a.tally != nullptr) a.tally[0] += a.total;                                                                    \
    return cudaSuccess;                                                                                               \
  }                                                                                                                   \
  cudaError_t launch_event_table(const unsigned long long*, uint32_t, uint32_t*, unsigned long long, uint32_t,        \
                                 cudaStream_t) {                                                                      \
    return cudaSuccess;                                                                                               \
  }                                                                                                                   \
  const void* sorted_prep_fn() { return &sorted_prep; }                                                               \
  const void* sorted_kernel_fn(int) { return &sorted_fn; }                                                            \
  int sorted_blocks_per_sm(int, int) { return 3; }                                                                    \
  cudaError_t launch_sorted(int, const DevParams&, const SortArgs&, SortCtrl*, int, int, cudaStream_t) {              \
    return cudaErrorNotSupported;                                                                                     \
  }                                                                                                                   \
  cudaError_t launch_sorted_prep(const SortArgs&, SortCtrl*, cudaStream_t) { return cudaErrorNotSupported; }          \
  }
OPTX_FAKE_LAUNCHERS(fast)
OPTX_FAKE_LAUNCHERS(exact)
OPTX_FAKE_LAUNCHERS(approx)
}  // namespace optx

#endif
