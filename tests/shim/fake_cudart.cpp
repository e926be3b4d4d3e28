#include "fake_cudart.hpp"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <mutex>

namespace {

struct Copy {
  void* dst;
  const void* src;
  size_t n;
};
std::recursive_mutex m;
std::map<cudaStream_t, std::vector<Copy>> pending;
std::map<void*, std::pair<size_t, int>> device_blocks;
std::map<const void*, size_t> pinned_sizes;
std::set<cudaStream_t> own_streams;
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> n;
  return n;
}

bool pinned(const void* p) {
  for (auto& b : pinned_sizes)
    if ((const char*)p >= (const char*)b.first && (const char*)p < (const char*)b.first + b.second) return true;
  return false;
}

void flush(cudaStream_t st) {
  for (auto& c : pending[st]) memcpy(c.dst, c.src, c.n);
  pending[st].clear();
}

bool captured(cudaStream_t st) { return fake::state().capturing && !own_streams.count(st); }

cudaError_t launch(const void* f, dim3 grid, size_t smem, void** args) {
  std::lock_guard<std::recursive_mutex> l(m);
  fake::State& s = fake::state();
  const std::string& name = names()[f];
  if (smem > 48 * 1024) {
    auto it = s.opted_in.find({s.device, name});
    if (it == s.opted_in.end() || it->second < (int)smem) {
      s.refused.push_back(name);
      return cudaErrorInvalidValue;
    }
  }
  s.launches[name] += 1;
  s.grids[name] = {grid.x, grid.y};
  if (s.on_launch) s.on_launch(name, args);
  return cudaSuccess;
}

}  // namespace

namespace fake {
State& state() {
  static State s;
  return s;
}
int device_of(const void* p) {
  for (auto& b : device_blocks)
    if ((const char*)p >= (const char*)b.first && (const char*)p < (const char*)b.first + b.second.first)
      return b.second.second;
  return -1;
}
size_t kept_on(int device) {
  size_t n = 0;
  for (auto& b : device_blocks)
    if (b.second.second == device) n += b.second.first;
  return n;
}
}  // namespace fake

extern "C" {

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*,
                            int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
static thread_local struct {
  dim3 g, b;
  size_t s;
  cudaStream_t st;
} config;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  config = {g, b, s, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = config.g;
  *b = config.b;
  *s = config.s;
  *(cudaStream_t*)st = config.st;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void** args, size_t smem, cudaStream_t) {
  return launch((const void*)k, grid, smem, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, c->gridDim, c->dynamicSmemBytes, args);
}
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::recursive_mutex> l(m);
  fake::State& s = fake::state();
  if (s.fail_mallocs > 0 || n > s.memory - s.in_use) {
    if (s.fail_mallocs > 0) --s.fail_mallocs;
    return cudaErrorMemoryAllocation;
  }
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  memset(*p, 0xff, (n + 255) / 256 * 256);
  device_blocks[*p] = {n, s.device};
  s.in_use += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::recursive_mutex> l(m);
  fake::state().in_use -= device_blocks[p].first;
  device_blocks.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  std::lock_guard<std::recursive_mutex> l(m);
  *p = calloc(1, n);
  pinned_sizes[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::recursive_mutex> l(m);
  pinned_sizes.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> l(m);
  if (k == cudaMemcpyHostToDevice && fake::state().defer_copies && !pinned(s)) {
    pending[st].push_back({d, s, n});
    return cudaSuccess;
  }
  flush(st);
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> l(m);
  if (captured(st)) fake::state().recorded += 1;
  else memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> l(m);
  if (captured(st)) return cudaErrorStreamCaptureUnsupported;
  fake::state().waits += 1;
  flush(st);
  if (fake::state().on_wait) fake::state().on_wait();
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus* s) {
  *s = captured(st) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::recursive_mutex> l(m);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    int& have = fake::state().opted_in[{fake::state().device, names()[f]}];
    have = v;
  }
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof(*a));
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = fake::state().device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  fake::state().device = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? fake::state().sms : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *t = fake::state().memory;
  *f = fake::state().memory - fake::state().in_use;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaStreamGetId(cudaStream_t st, unsigned long long* id) {
  *id = (unsigned long long)(size_t)st;
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) {
  std::lock_guard<std::recursive_mutex> l(m);
  *st = (cudaStream_t)malloc(1);
  own_streams.insert(*st);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> l(m);
  own_streams.erase(st);
  free(st);
  return cudaSuccess;
}
static int encode_stub(...) { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *f = (void*)encode_stub;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

}  // extern "C"
