// fake_cudart.cpp -- the CUDA runtime calls of the engine library on the host,
// for tests of what its host code does when a call fails.  Device memory is
// host memory, copies and fills are done, streams run at once, kernels only
// leave their names behind.  Tests set limits and failures by name
// (fake_set) and read what was launched (fake_launched).
#include <cuda.h>
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>

namespace {

std::recursive_mutex mu;
std::map<std::string, long long>& knobs() {
  static std::map<std::string, long long> k = {
      {"sms", 148}, {"capacity", 180ll << 30},
      {"fail_host", 0},         // cudaMallocHost calls to refuse (-1: all)
      {"pass_host", 0},         // ... after letting this many through
      {"fail_pool_from", -1},   // refuse pool allocations of at least this many bytes
      {"fail_instantiate", 0},  // graph instantiations to refuse
      {"fail_graph_launch", 0}, // graph launches to refuse
      {"fail_kernel", 0},       // kernel launches to refuse ...
      {"pass_kernel", 0},       // ... after letting this many through
      {"pass_ns", 10000},       // time of a fused pass' launch between two events
      {"update_ns", 10000},     // ... of an update kernel's
      {"real_time", 0},         // 1: that time passes on the host
  };
  return k;
}
std::map<std::string, long long>& launched() {
  static std::map<std::string, long long> m;
  return m;
}
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
struct Block {
  size_t bytes;
  bool pool;
};
std::map<void*, Block>& blocks() {
  static std::map<void*, Block> m;
  return m;
}
long long direct = 0, pooled = 0, reserved = 0, streams = 0, pinned = 0, pins = 0, copies = 0, instantiated = 0, captured = 0, largest = 0;
long long clock_ns = 0;  // of the launches so far
thread_local cudaError_t last = cudaSuccess;
thread_local int capturing = 0;
thread_local long long captured_ns = 0;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
// One use of a failure armed `key` times (after `pass` more uses): true to refuse.
bool refuse(const char* key, const char* pass = nullptr) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (pass && knobs()[pass] > 0) {
    knobs()[pass]--;
    return false;
  }
  long long& n = knobs()[key];
  if (n == 0) return false;
  if (n > 0) --n;
  return true;
}
void* take(size_t bytes) {
  void* p = mmap(nullptr, std::max<size_t>(bytes, 1), PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE,
                 -1, 0);
  return p == MAP_FAILED ? nullptr : p;
}
cudaError_t alloc(void** p, size_t bytes, bool pool) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const long long n = (long long)bytes, cap = knobs()["capacity"], from = knobs()["fail_pool_from"];
  if (pool && from >= 0 && n >= from) return ret(cudaErrorMemoryAllocation);
  const long long grow = pool ? std::max(0ll, pooled + n - reserved) : n;
  if (direct + reserved + grow > cap) return ret(cudaErrorMemoryAllocation);
  if (!(*p = take(bytes))) return ret(cudaErrorMemoryAllocation);
  if (pool) {
    pooled += n;
    reserved += grow;
  } else {
    direct += n;
  }
  blocks()[*p] = {bytes, pool};
  return cudaSuccess;
}
cudaError_t give(void* p) {
  if (!p) return cudaSuccess;
  std::lock_guard<std::recursive_mutex> lk(mu);
  auto it = blocks().find(p);
  if (it == blocks().end()) return ret(cudaErrorInvalidValue);
  (it->second.pool ? pooled : direct) -= (long long)it->second.bytes;
  munmap(p, std::max<size_t>(it->second.bytes, 1));
  blocks().erase(it);
  return cudaSuccess;
}
cudaError_t launch(const void* f) {
  if (refuse("fail_kernel", "pass_kernel")) return ret(cudaErrorLaunchOutOfResources);
  std::lock_guard<std::recursive_mutex> lk(mu);
  const std::string name = names().count(f) ? names()[f] : "?";
  launched()[name]++;
  const long long ns = name.find("k_fused") != std::string::npos    ? knobs()["pass_ns"]
                       : name.find("k_update") != std::string::npos ? knobs()["update_ns"]
                                                                    : 0;
  (capturing ? captured_ns : clock_ns) += ns;
  if (!capturing && knobs()["real_time"]) std::this_thread::sleep_for(std::chrono::nanoseconds(ns));
  if (capturing) largest = std::max(largest, ++captured);
  return cudaSuccess;
}
CUresult encode(...) { return CUDA_SUCCESS; }

}  // namespace

extern "C" {

void fake_set(const char* key, long long v) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  knobs()[key] = v;
}
// Launches (captured ones count once) of kernels whose mangled name contains `part`; all are forgotten if `reset`.
long long fake_launched(const char* part, int reset) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  long long n = 0;
  for (auto& kv : launched())
    if (kv.first.find(part) != std::string::npos) n += kv.second;
  if (reset) launched().clear();
  return n;
}
long long fake_pool_used() { return pooled; }
long long fake_pinned() { return pinned; }  // bytes now
long long fake_pins() { return pins; }      // calls so far
long long fake_copies() { return copies; }  // linear ones, asked for so far
long long fake_instantiated() { return instantiated; }
long long fake_largest_graph() { return largest; }  // kernels in it

cudaError_t cudaMalloc(void** p, size_t n) { return alloc(p, n, false); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return alloc(p, n, true); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (refuse("fail_host", "pass_host")) return ret(cudaErrorMemoryAllocation);
  std::lock_guard<std::recursive_mutex> lk(mu);
  char* q = static_cast<char*>(std::malloc(n + 64));
  if (!q) return ret(cudaErrorMemoryAllocation);
  std::memcpy(q, &n, sizeof(n));
  pinned += (long long)n;
  ++pins;
  *p = q + 64;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  size_t n = 0;
  char* q = static_cast<char*>(p) - 64;
  std::memcpy(&n, q, sizeof(n));
  pinned -= (long long)n;
  std::free(q);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *t = (size_t)knobs()["capacity"];
  *f = (size_t)(knobs()["capacity"] - direct - reserved);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  *p = reinterpret_cast<cudaMemPool_t>(8);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr a, void* v) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *static_cast<uint64_t*>(v) = (uint64_t)(a == cudaMemPoolAttrUsedMemCurrent ? pooled : reserved);
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  reserved = pooled;
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  if (v == 0 && n > (1u << 20)) {  // whole pages back to zero pages
    const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 4095) / 4096 * 4096;
    const uintptr_t b = (reinterpret_cast<uintptr_t>(p) + n) / 4096 * 4096;
    std::memset(p, 0, a - reinterpret_cast<uintptr_t>(p));
    std::memset(reinterpret_cast<void*>(b), 0, reinterpret_cast<uintptr_t>(p) + n - b);
    madvise(reinterpret_cast<void*>(a), b - a, MADV_DONTNEED);
  } else {
    std::memset(p, v, n);
  }
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  ++copies;
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t r = 0; r < h; ++r) std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
  return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount                ? (int)knobs()["sms"]
       : a == cudaDevAttrMaxSharedMemoryPerBlockOptin     ? 232448
       : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472
       : a == cudaDevAttrComputeCapabilityMajor           ? 10
                                                          : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *f = reinterpret_cast<void*>(&encode);
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *s = reinterpret_cast<cudaStream_t>((uintptr_t)(16 * ++streams));
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new long long(0));
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<long long*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  *reinterpret_cast<long long*>(e) = clock_ns;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(*reinterpret_cast<long long*>(b) - *reinterpret_cast<long long*>(a)) * 1e-6f;
  return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  ++capturing;
  captured = captured_ns = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  --capturing;
  *g = reinterpret_cast<cudaGraph_t>(captured_ns + 1);  // (a graph's handle is its time)
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  if (refuse("fail_instantiate")) return ret(cudaErrorMemoryAllocation);
  std::lock_guard<std::recursive_mutex> lk(mu);
  ++instantiated;
  *e = reinterpret_cast<cudaGraphExec_t>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  if (refuse("fail_graph_launch")) return ret(cudaErrorMemoryAllocation);
  std::lock_guard<std::recursive_mutex> lk(mu);
  const long long ns = (long long)reinterpret_cast<uintptr_t>(e) - 1;
  clock_ns += ns;
  if (knobs()["real_time"]) std::this_thread::sleep_for(std::chrono::nanoseconds(ns));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) { return launch(f); }

// what nvcc's host code calls around a launch and at load time
static thread_local struct {
  dim3 g, b;
  size_t smem;
  cudaStream_t s;
} config;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
  config = {g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = config.g;
  *b = config.b;
  *smem = config.smem;
  *static_cast<cudaStream_t*>(s) = config.s;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"
