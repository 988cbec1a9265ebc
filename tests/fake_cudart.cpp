// A stand-in for the CUDA runtime: the library's host code runs on a machine without a
// GPU.  Device memory is host memory, copies are copies, kernels do nothing.  It keeps
// what a test asks about (the live allocations, the launches) and refuses what the
// runtime refuses: copies outside an allocation or to a null pointer, and launches with
// more than 48 KB of dynamic shared memory for which the kernel has not opted in on the
// current device.  fake_* are the tests' controls.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

namespace {
struct Block {
  size_t bytes;
  int device;  // -1: pinned host memory
};
std::recursive_mutex mu;
std::map<uintptr_t, Block> blocks;  // by start address
std::map<const void*, std::string> kernels;
std::map<std::pair<const void*, int>, size_t> optIn;
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
long launches = 0, failAt = -1;
std::string lastKernel;
std::map<uintptr_t, size_t> copiedTo;  // destinations of copies
struct Config {
  dim3 grid, block;
  size_t smem = 0;
  cudaStream_t stream = nullptr;
};
thread_local Config pushed;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
// the block that holds p, or end()
std::map<uintptr_t, Block>::iterator find(const void* p) {
  auto it = blocks.upper_bound((uintptr_t)p);
  if (it == blocks.begin()) return blocks.end();
  --it;
  return (uintptr_t)p < it->first + it->second.bytes ? it : blocks.end();
}
bool inside(const void* p, size_t bytes) {
  auto it = find(p);
  return it == blocks.end() ? p != nullptr : (uintptr_t)p + bytes <= it->first + it->second.bytes;
}
cudaError_t allocate(void** p, size_t bytes, int device) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *p = nullptr;
  if (posix_memalign(p, 512, bytes ? bytes : 1)) return done(cudaErrorMemoryAllocation);
  memset(*p, 0, bytes);
  blocks[(uintptr_t)*p] = {bytes, device};
  return cudaSuccess;
}
cudaError_t release(void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!p) return cudaSuccess;
  if (!blocks.erase((uintptr_t)p)) return done(cudaErrorInvalidValue);
  free(p);
  return cudaSuccess;
}
cudaError_t launch(const void* f, size_t smem) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  lastKernel = kernels[f];
  if (launches++ == failAt) return done(cudaErrorLaunchOutOfResources);
  if (smem > 48 * 1024) {
    auto it = optIn.find({f, current});
    if (it == optIn.end() || it->second < smem) return done(cudaErrorInvalidValue);
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- controls
size_t fake_device_bytes() {
  std::lock_guard<std::recursive_mutex> lk(mu);
  size_t n = 0;
  for (auto& b : blocks)
    if (b.second.device >= 0) n += b.second.bytes;
  return n;
}
long fake_launches() { return launches; }
void fake_fail_at(long n) { failAt = n; }  // the n-th launch from the start fails; -1: none
const char* fake_last_kernel() { return lastKernel.c_str(); }
void fake_set_device(int d) { current = d; }
void fake_count_up() {  // the doubles of every device block become 0, 1, 2, ...
  std::lock_guard<std::recursive_mutex> lk(mu);
  for (auto& b : blocks)
    for (size_t i = 0; b.second.device >= 0 && i < b.second.bytes / 8; ++i) ((double*)b.first)[i] = (double)i;
}
size_t fake_copied_to(const void* p) {  // bytes of the last copy to p (0: none)
  std::lock_guard<std::recursive_mutex> lk(mu);
  auto it = copiedTo.find((uintptr_t)p);
  return it == copiedTo.end() ? 0 : it->second;
}

// ---- kernels
void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
  pushed = {grid, block, smem, (cudaStream_t)stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *(cudaStream_t*)stream = pushed.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->dynamicSmemBytes); }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) optIn[{f, current}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof(*a));
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 16;
  return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t bytes) { return allocate(p, bytes, current); }
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) { return allocate(p, bytes, current); }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { return allocate(p, bytes, -1); }
cudaError_t cudaMallocHost(void** p, size_t bytes) { return allocate(p, bytes, -1); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return release(p); }
cudaError_t cudaFreeHost(void* p) { return release(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = *t = (size_t)180 << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (!inside(d, bytes) || !inside(s, bytes)) return done(cudaErrorInvalidValue);
    copiedTo[(uintptr_t)d] = bytes;
  }
  memmove(d, s, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  for (size_t r = 0; r < h; ++r) memmove((char*)d + r * dp, (const char*)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t bytes, cudaStream_t) {
  if (!inside(d, bytes)) return done(cudaErrorInvalidValue);
  memset(d, v, bytes);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  memset(a, 0, sizeof(*a));
  auto it = find(p);
  a->type = it == blocks.end() ? cudaMemoryTypeUnregistered : it->second.device < 0 ? cudaMemoryTypeHost : cudaMemoryTypeDevice;
  a->device = it == blocks.end() ? -1 : it->second.device;
  return cudaSuccess;
}
static CUresult address_range(CUdeviceptr* base, size_t* size, CUdeviceptr p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  auto it = find((const void*)(uintptr_t)p);
  if (it == blocks.end()) return CUDA_ERROR_NOT_FOUND;
  *base = (CUdeviceptr)it->first;
  *size = it->second.bytes;
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* found) {
  const bool known = !strcmp(name, "cuMemGetAddressRange");
  *f = known ? (void*)address_range : nullptr;
  if (found) *found = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
  *p = const_cast<void*>(symbol);
  return cudaSuccess;
}

// ---- the rest
cudaError_t cudaGetDevice(int* d) {
  *d = current;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  current = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaStreamCreate(cudaStream_t* s) {
  *s = (cudaStream_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return "refused by the stand-in runtime"; }
}
