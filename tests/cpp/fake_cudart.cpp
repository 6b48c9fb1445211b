// A CUDA runtime on host memory, for tests of the library's host code without a
// GPU: every call the library makes is served from here.  Kernels do nothing;
// copies happen at once; calls that carry an order (copies, launches, frees and
// waits) go to a log.  Memory pools keep freed blocks as CUDA's do: what a pool
// holds beyond its release threshold goes back at the next wait, or by a trim.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {

struct Pool {
  size_t used = 0, reserved = 0, threshold = 0;
};
struct Block {
  size_t bytes = 0;
  Pool* pool = nullptr;  // null: cudaMalloc
};

std::recursive_mutex mu;
std::vector<std::string> lines;
std::map<void*, Block> live;
std::map<const void*, std::string> kernels;
std::vector<Pool*> pools;
Pool default_pool;
size_t plain = 0;                       // bytes of cudaMalloc
const size_t kTotal = size_t(1) << 38;  // the device's memory
size_t limit = kTotal;                  // .. of which allocations get this much
int fail_copy = 0;                      // 1: the next copy fails, 2: the one after, ..
cudaError_t last = cudaSuccess;

template <typename... A>
void note(const char* f, A... a) {
  char s[256];
  snprintf(s, sizeof s, f, a...);
  lines.push_back(s);
}
cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
size_t taken() {
  size_t n = plain + default_pool.reserved;
  for (Pool* p : pools) n += p->reserved;
  return n;
}
void wait_for(const char* what, cudaStream_t s) {
  note("%s %p", what, (void*)s);
  pools.push_back(&default_pool);
  for (Pool* p : pools)
    if (p->reserved > p->threshold) p->reserved = p->used > p->threshold ? p->used : p->threshold;
  pools.pop_back();
}
cudaError_t take(void** p, size_t n, Pool* pool) {
  *p = nullptr;
  const size_t more = pool ? (pool->used + n > pool->reserved ? pool->used + n - pool->reserved : 0) : n;
  if (taken() + more > limit) return ret(cudaErrorMemoryAllocation);
  *p = calloc(1, n ? n : 1);
  live[*p] = {n, pool};
  if (pool) {
    pool->used += n;
    pool->reserved += more;
  } else {
    plain += n;
  }
  return cudaSuccess;
}
cudaError_t give(void* p) {
  if (!p) return cudaSuccess;
  const auto it = live.find(p);
  if (it == live.end()) return ret(cudaErrorInvalidValue);
  if (it->second.pool) it->second.pool->used -= it->second.bytes;
  else plain -= it->second.bytes;
  live.erase(it);
  free(p);
  return cudaSuccess;
}
const char* kind_name(cudaMemcpyKind k) { return k == cudaMemcpyHostToDevice ? "h2d" : (k == cudaMemcpyDeviceToHost ? "d2h" : "d2d"); }
cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st, bool async) {
  note("%s %s %p %p %zu", async ? "copy" : "copy_and_return", kind_name(k), (void*)st, d, n);
  if (fail_copy && --fail_copy == 0) return ret(cudaErrorUnknown);
  memcpy(d, s, n);
  return cudaSuccess;
}
template <typename T>
T* token() {
  return reinterpret_cast<T*>(new char[1]);
}
struct Config {
  dim3 grid, block;
  size_t shared;
  cudaStream_t st;
};
thread_local std::vector<Config> configs;

}  // namespace

#define GUARD std::lock_guard<std::recursive_mutex> lk(mu)

extern "C" {

// ---- what the tests read and set
size_t fake_log(char* out, size_t n) {
  GUARD;
  std::string all;
  for (const auto& l : lines) all += l + "\n";
  if (out && n) snprintf(out, n, "%s", all.c_str());
  return all.size() + 1;
}
void fake_clear_log() {
  GUARD;
  lines.clear();
}
size_t fake_taken() {
  GUARD;
  return taken();
}
size_t fake_live_bytes() {
  GUARD;
  size_t n = 0;
  for (const auto& b : live) n += b.second.bytes;
  return n;
}
void fake_limit(size_t n) {
  GUARD;
  limit = n ? n : kTotal;
}
void fake_fail_copy(int n) {
  GUARD;
  fail_copy = n;
}

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(token<void>()); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  GUARD;
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, CUstream_st* st) {
  configs.push_back({grid, block, shared, st});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* st) {
  const Config c = configs.back();
  configs.pop_back();
  *grid = c.grid;
  *block = c.block;
  *shared = c.shared;
  *static_cast<cudaStream_t*>(st) = c.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(host));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t, cudaStream_t st) {
  GUARD;
  note("launch %p %s %u %u", (void*)st, kernels[reinterpret_cast<const void*>(k)].c_str(), grid.x, block.x);
  return cudaSuccess;
}

// ---- device
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof *p);
  p->major = 10;
  p->minor = 3;
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  GUARD;
  wait_for("wait_device", nullptr);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  GUARD;
  *t = kTotal;
  *f = kTotal - taken();
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  GUARD;
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the test's CUDA runtime"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, cudaErrorInvalidSymbol; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) {
  return cudaErrorInvalidValue;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
  GUARD;
  return take(p, n, nullptr);
}
cudaError_t cudaFree(void* p) {
  GUARD;
  return give(p);
}
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
  GUARD;
  return take(p, n, &default_pool);
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  GUARD;
  return take(p, n, reinterpret_cast<Pool*>(pool));
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t st) {
  GUARD;
  if (p) note("free %p %p", (void*)st, p);
  return give(p);
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) {
  return *p = reinterpret_cast<cudaMemPool_t>(&default_pool), cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  GUARD;
  pools.push_back(new Pool());
  return *p = reinterpret_cast<cudaMemPool_t>(pools.back()), cudaSuccess;
}
// (blocks that still live keep the pool's memory; the fake keeps all that it holds)
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  GUARD;
  Pool* q = reinterpret_cast<Pool*>(p);
  if (!q->used) q->reserved = 0;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  GUARD;
  if (a != cudaMemPoolAttrReleaseThreshold) return ret(cudaErrorInvalidValue);
  reinterpret_cast<Pool*>(p)->threshold = *static_cast<unsigned long long*>(v);
  return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  GUARD;
  const Pool* q = reinterpret_cast<Pool*>(p);
  if (a == cudaMemPoolAttrReleaseThreshold) *static_cast<unsigned long long*>(v) = q->threshold;
  else if (a == cudaMemPoolAttrReservedMemCurrent) *static_cast<unsigned long long*>(v) = q->reserved;
  else if (a == cudaMemPoolAttrUsedMemCurrent) *static_cast<unsigned long long*>(v) = q->used;
  else return ret(cudaErrorInvalidValue);
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  GUARD;
  Pool* q = reinterpret_cast<Pool*>(p);
  if (q->reserved > keep) q->reserved = q->used > keep ? q->used : keep;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  GUARD;
  return copy(d, s, n, k, cudaStreamLegacy, false);
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  GUARD;
  return copy(d, s, n, k, st, true);
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = token<CUstream_st>(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  GUARD;
  wait_for("wait", s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = token<CUevent_st>(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"
