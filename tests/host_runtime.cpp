// A CUDA runtime in host memory, for tests of the library's host code without
// a GPU: the library's objects are linked against it, allocations are host
// memory, copies are checked against them and kernels do nothing.
//
// What it watches (hr_bad counts, hr_last_bad names the last one): a copy or
// memset outside a live allocation, and a launch of the sweep or of the output
// records whose case table, case or arguments hold an address inside a freed
// allocation.  Freed memory is kept, so an address never comes back.
// hr_limit(n): allocations of more than n bytes fail (0: none do); hr_fail_at(k):
// the k-th allocation from now on fails.
// A read of a case's control block says that the march ended after hr_steps
// (three) steps.  hr_block(size): the live allocation of that size.  hr_sms(n): the
// device has n SMs.  hr_blocks_of(kernel): the blocks of the largest launch
// of a kernel whose mangled name has this text.  hr_sweep_bufs(): the tile buffers
// of the last sweep launched.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "types.h"

namespace {
struct Block {
  size_t size;
  bool live;
};
std::map<uintptr_t, Block> blocks;
size_t limit_bytes = 0;
long fail_at = -1;
int march_steps = 3, sms = 148, sweep_bufs = 0, bad = 0;
std::string last_bad;
// (a function's static: the objects register their kernels before this file's are made)
std::map<const void*, std::string>& kernels() {
  static std::map<const void*, std::string> k;
  return k;
}

struct Launch {
  uintptr_t table = 0;            // the case table of a sweep launch
  std::vector<uintptr_t> words;   // its case, or the records' arguments
  const char* what = "";
};
struct Graph {
  std::vector<Launch> launches;
};
Graph* capturing = nullptr;

void report(const std::string& m) {
  ++bad;
  last_bad = m;
}
std::map<uintptr_t, Block>::iterator find(uintptr_t p) {
  auto it = blocks.upper_bound(p);
  if (it == blocks.begin()) return blocks.end();
  --it;
  return p < it->first + it->second.size ? it : blocks.end();
}
// dst / src on the device: inside one live allocation
bool device_range(const void* p, size_t n, const char* what) {
  const auto it = find((uintptr_t)p);
  if (it != blocks.end() && it->second.live && (uintptr_t)p + n <= it->first + it->second.size) return true;
  if (it != blocks.end()) report(std::string(what) + (it->second.live ? " past the end of" : " of freed") + " memory");
  return false;
}
void check_words(const uintptr_t* w, size_t n, const char* what) {
  for (size_t i = 0; i < n; ++i) {
    const auto it = find(w[i]);
    if (it != blocks.end() && !it->second.live) return report(std::string(what) + " holds a freed address");
  }
}
void execute(const Launch& l) {
  if (l.table) {
    const auto it = find(l.table);
    if (it == blocks.end() || !it->second.live) return report("the case table is freed");
    check_words((const uintptr_t*)it->first, it->second.size / 8, "the case table");
  }
  check_words(l.words.data(), l.words.size(), l.what);
}
std::map<std::string, unsigned> grids;
cudaError_t launch(const void* fn, dim3 grid, void** args) {
  const std::string& name = kernels()[fn];
  grids[name] = std::max(grids[name], grid.x * grid.y);
  Launch l;
  if (name.find("k_sweep") != std::string::npos) {
    // (BatchArgs, whose first word is the case table; total units; the case,
    // as large as an entry of the table of one)
    l.table = *(const uintptr_t*)args[0];
    l.what = "the sweep's case";
    const auto it = find(l.table);
    const int* ints = (const int*)args[0] + 10;  // after the table, three offsets and the control block
    const int ncases = ints[0];
    sweep_bufs = ints[2];  // after the widest halo
    if (it != blocks.end() && ncases == 1)
      l.words.assign((const uintptr_t*)args[2], (const uintptr_t*)args[2] + it->second.size / 8);
  } else if (name.find("k_out_") != std::string::npos) {
    l.what = "the output records' arguments";
    l.words.assign((const uintptr_t*)args[0], (const uintptr_t*)args[0] + 23);
    if (l.words[20] == 0 && l.words[22] == 0) report("output records without a ring");  // ring, direct
  } else {
    return cudaSuccess;
  }
  if (capturing)
    capturing->launches.push_back(l);
  else
    execute(l);
  return cudaSuccess;
}
cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  if (n == 0) return cudaSuccess;
  if (!d || !s) return cudaErrorInvalidValue;
  const bool to = k == cudaMemcpyHostToDevice || k == cudaMemcpyDeviceToDevice;
  const bool from = k == cudaMemcpyDeviceToHost || k == cudaMemcpyDeviceToDevice;
  if ((to && !device_range(d, n, "copy to")) || (from && !device_range(s, n, "copy from"))) return cudaErrorInvalidValue;
  if (k == cudaMemcpyDeviceToHost && n == sizeof(dgbgk::Ctrl)) {
    auto* c = (dgbgk::Ctrl*)s;
    c->step = std::min(c->max_steps, march_steps);
    c->done = 1;
  }
  std::memmove(d, s, n);
  return cudaSuccess;
}
}  // namespace

extern "C" {
void hr_limit(size_t n) { limit_bytes = n; }
void hr_fail_at(long k) { fail_at = k; }
void hr_steps(int n) { march_steps = n; }
void hr_sms(int n) { sms = n; }
int hr_sweep_bufs() { return sweep_bufs; }
unsigned hr_blocks_of(const char* kernel) {
  for (const auto& g : grids)
    if (g.first.find(kernel) != std::string::npos) return g.second;
  return 0;
}
int hr_bad() { return bad; }
const char* hr_last_bad() { return last_bad.c_str(); }
void* hr_block(size_t size) {
  for (const auto& b : blocks)
    if (b.second.live && b.second.size == size) return (void*)b.first;
  return nullptr;
}

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  if (limit_bytes && n > limit_bytes) return cudaErrorMemoryAllocation;
  if (fail_at > 0 && --fail_at == 0) return cudaErrorMemoryAllocation;
  *p = calloc(1, n + 64);
  if (!*p) return cudaErrorMemoryAllocation;
  blocks[(uintptr_t)*p] = {n, true};
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  const auto it = blocks.find((uintptr_t)p);
  if (it == blocks.end() || !it->second.live) {
    report("free of memory that is not live");
    return cudaErrorInvalidValue;
  }
  it->second.live = false;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return (*p = calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return copy(d, s, n, k);
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k) {
  // cudaDeviceProp::memPitch, the range stated (a driver may let larger ones through)
  if (dp > 0x7fffffff || sp > 0x7fffffff) return cudaErrorInvalidPitchValue;
  for (size_t i = 0; i < h; ++i)
    if (const cudaError_t e = copy((char*)d + i * dp, (const char*)s + i * sp, w, k)) return e;
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  if (!d || !device_range(d, n, "memset of")) return cudaErrorInvalidValue;
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }

cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3, void** args, size_t, cudaStream_t) { return launch(f, g, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, c->gridDim, args);
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = new Graph;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)capturing;
  capturing = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t) new Graph(*(Graph*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete (Graph*)g, cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return delete (Graph*)e, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (const auto& l : ((Graph*)e)->launches) execute(l);
  return cudaSuccess;
}

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset((void*)p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = sms;
  p->memPitch = 0x7fffffff;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : sms;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  return std::memset((void*)a, 0, sizeof *a), cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  return *n = 1, cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : "host runtime error";
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return cudaMalloc(p, 8 << 20); }
CUresult hr_encode(...) { return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *f = (void*)hr_encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free((void*)s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)malloc(1), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free((void*)e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { return *t = 1.f, cudaSuccess; }

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  kernels()[host] = name;
}
static struct {
  dim3 g, b;
  size_t m;
  void* s;
} pushed;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void* s) {
  pushed = {g, b, m, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = pushed.g;
  *b = pushed.b;
  *m = pushed.m;
  *(void**)s = pushed.s;
  return cudaSuccess;
}
}  // extern "C"
