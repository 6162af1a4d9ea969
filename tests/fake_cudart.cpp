// A CUDA runtime without a GPU, for tests of the library's host side (test_host_runtime.py preloads
// it): device memory is host memory, kernels do nothing, and every call that orders work or takes
// memory leaves a line in a log.  Handles are small numbers.  Two devices that can reach each other,
// each with `limit` bytes; a pool holds on to what it was given back until it is trimmed.
#include <cuda_runtime_api.h>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <unistd.h>

namespace {

struct Block { size_t bytes; int pool; };  // pool -1: of cudaMalloc
struct Call { dim3 grid, block; size_t smem; cudaStream_t st; };

// (never destroyed: the library may call while the process exits)
std::recursive_mutex mu;
std::string& text = *new std::string;
struct Failure { int status, calls; };
std::map<std::string, Failure>& fail = *new std::map<std::string, Failure>;   // function -> status of its `calls`th call from now
std::map<std::string, long>& knob =
    *new std::map<std::string, long>{{"limit", 1L << 50}, {"capturing", 0}, {"free_us", 0}, {"entries", 0}};
std::map<void*, Block>& live = *new std::map<void*, Block>;
std::map<const void*, std::string>& names = *new std::map<const void*, std::string>;  // kernels
size_t in_use = 0, idle[64] = {};
long next_handle = 16, pools = 0;
thread_local int device = 0;
thread_local Call pushed;
thread_local cudaError_t last = cudaSuccess;

cudaError_t log(const char* f, const char* fmt = "", ...) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  char b[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(b, sizeof b, fmt, ap);
  va_end(ap);
  text += std::string(f) + " " + b + "\n";
  auto it = fail.find(f);
  if (it == fail.end() || it->second.calls-- != 1) return cudaSuccess;
  last = (cudaError_t)it->second.status;
  return last;
}

template <typename T>
T handle() {
  std::lock_guard<std::recursive_mutex> lk(mu);
  return (T)(next_handle++);
}

cudaError_t take(void** p, size_t bytes, int pool) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const size_t reuse = pool >= 0 && bytes <= idle[pool] ? bytes : 0;  // (idle memory is one piece)
  size_t held = in_use;
  for (size_t i : idle) held += i;
  if (held + bytes - reuse > (size_t)knob["limit"]) return last = cudaErrorMemoryAllocation;
  if (pool >= 0) idle[pool] -= reuse;
  in_use += bytes;
  *p = calloc(1, bytes + 256);
  live[*p] = {bytes, pool};
  return cudaSuccess;
}

cudaError_t give(void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!p) return cudaSuccess;
  auto it = live.find(p);
  if (it == live.end()) return cudaErrorInvalidValue;
  in_use -= it->second.bytes;
  if (it->second.pool >= 0) idle[it->second.pool] += it->second.bytes;
  live.erase(it);
  free(p);
  return cudaSuccess;
}

#define LOGGED(...)                              \
  do {                                           \
    const cudaError_t e_ = log(__VA_ARGS__);     \
    if (e_ != cudaSuccess) return e_;            \
  } while (0)

int encode_nothing(...) { return 0; }

// An exit handler from before the library was loaded, which therefore runs after its destructors.
int (*at_exit)(void*) = nullptr;
void* at_exit_arg = nullptr;
__attribute__((constructor)) void early() {
  atexit([] { if (at_exit && at_exit(at_exit_arg) != 0) _exit(3); });
}

}  // namespace

extern "C" {

// ---- the test's side
const char* fake_log() { return text.c_str(); }
void fake_clear() { text.clear(); }
void fake_fail(const char* f, int status, int calls) { fail[f] = {status, calls}; }
void fake_set(const char* k, long v) { knob[k] = v; }
void fake_at_exit(int (*f)(void*), void* arg) { at_exit = f; at_exit_arg = arg; }
long fake_live() { return (long)live.size(); }

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* st) {
  pushed = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = pushed.grid; *b = pushed.block; *smem = pushed.smem; *(cudaStream_t*)st = pushed.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3, void** args, size_t, cudaStream_t st) {
  if (names[f].find("k_fl_count") != std::string::npos) **(double**)args[4] = knob["entries"];
  LOGGED("launch", "%ld %u %s", (long)st, g.z, names[f].c_str());
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  LOGGED("launch", "%ld %u %s", (long)c->stream, c->gridDim.z, names[f].c_str());
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode_nothing;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)s; return cudaSuccess; }

// ---- devices
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceCanAccessPeer(int* can, int a, int b) { *can = a != b; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  LOGGED("cudaDeviceSynchronize");
  return knob["capturing"] ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { LOGGED("cudaMalloc", "%zu", n); return take(p, n, -1); }
cudaError_t cudaFree(void* p) {
  LOGGED("cudaFree", "%p", p);
  if (p) usleep(knob["free_us"]);  // (as if work on the device had to end first)
  return give(p);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)(++pools); return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  LOGGED("cudaMemPoolSetAttribute", "%ld %d %d", (long)p, (int)a, *(int*)v);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAccess(cudaMemPool_t p, const cudaMemAccessDesc* d, size_t n) {
  for (size_t i = 0; i < n; i++) LOGGED("cudaMemPoolSetAccess", "%ld %d %d", (long)p, d[i].location.id, (int)d[i].flags);
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  LOGGED("cudaMemPoolTrimTo", "%ld %zu", (long)p, keep);
  idle[(long)p] = 0;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t st) {
  LOGGED("cudaMallocFromPoolAsync", "%ld %zu", (long)st, n);
  return take(p, n, (int)(long)pool);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t st) {
  if (!p) return last = cudaErrorInvalidValue;  // (unlike cudaFree)
  LOGGED("cudaFreeAsync", "%ld %p", (long)st, p); return give(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  LOGGED("cudaMemcpy", "%d", (int)k);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  LOGGED("cudaMemcpyAsync", "%ld %d", (long)st, (int)k);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyPeerAsync(void* d, int, const void* s, int, size_t n, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  for (size_t r = 0; r < h; r++) memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { LOGGED("cudaMemset"); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = handle<cudaStream_t>(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { LOGGED("cudaStreamDestroy", "%ld", (long)s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { LOGGED("cudaStreamSynchronize", "%ld", (long)s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { LOGGED("wait", "%ld %ld", (long)s, (long)e); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = handle<cudaGraph_t>(); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = handle<cudaGraphExec_t>(); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = handle<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = handle<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { LOGGED("record", "%ld %ld", (long)e, (long)s); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }

}  // extern "C"
