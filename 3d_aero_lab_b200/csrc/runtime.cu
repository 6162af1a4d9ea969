// runtime.cu - library-wide plumbing: error strings, device selection, grid/geometry buffers.
#include <algorithm>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <set>
#include <string>
#include <vector>
#include "geom.cuh"

namespace a3d {

namespace {
thread_local std::string g_last_error;
}

void set_error(const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_last_error = buf;
}

void clear_error() { g_last_error.clear(); }

int use_device(int device) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) {
    set_error("no CUDA device visible (%s)", e == cudaSuccess ? "0 devices" : cudaGetErrorString(e));
    return A3D_ERR_NODEVICE;
  }
  if (device >= 0) {
    if (device >= n) { set_error("device %d out of range (%d visible)", device, n); return A3D_ERR_ARG; }
    A3D_CUDA(cudaSetDevice(device));
  }
  return A3D_OK;
}

// ---- memory ------------------------------------------------------------------------------
// cudaMalloc, cudaFree and the default pool (which gives its memory back at every
// synchronisation) map and unmap device memory: 0.2 to 6 ms a call, more than the work of a
// case's setup (1M cells: 12 ms with a dozen of them, 0.3 ms of kernels) or of sampling 20,000
// points.  The library therefore has a pool of its own on each device: 2 us a call.  Memory that
// nothing uses stays while the pool's whole, used and unused, is below kPoolKeep bytes, and not at
// all once the last block is freed (the next case then pays as without the pool).
// Blocks beyond kPoolBlock, of which a pool could keep none, come from cudaMalloc as before (growing
// the pool by gigabytes takes longer: 120M cells' setup 0.12 s instead of 0.10).
namespace {

constexpr unsigned long long kPoolKeep = 1ull << 30;
constexpr size_t kPoolBlock = 256u << 20;

struct Pool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;  // orders the blocks of dev_alloc / dev_free
  long blocks = 0;            // of dev_alloc, in use
  std::set<void*> large;      // those from cudaMalloc
  std::vector<cudaStream_t> streams;  // free ones
  long streams_out = 0;       // streams in use
  void* byte = nullptr;       // of device_wait
  std::set<int> peers;        // devices that may address the pool's blocks
  bool shared = false;        // all that can
};

std::mutex g_pool_mu;
// by device; never destroyed: solvers may be, and threads may run, while the process exits
std::vector<Pool>& g_pools = *new std::vector<Pool>;

// The current device's pool, made at its first use.  Caller holds g_pool_mu.
cudaError_t current_pool(Pool** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((int)g_pools.size() <= dev) g_pools.resize(dev + 1);
  Pool& p = g_pools[dev];
  if (!p.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    e = cudaMemPoolCreate(&pool, &props);
    unsigned long long keep = kPoolKeep;
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    // a block never waits for what another stream has yet to give back (it would for all that is
    // queued there, another solver's steps)
    int wait = 0;
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &wait);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p.st, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      if (pool) cudaMemPoolDestroy(pool);
      return e;
    }
    p.pool = pool;
  }
  *out = &p;
  return cudaSuccess;
}

}  // namespace

// Blocks are taken and given back without the lock: cudaMalloc and cudaFree may take milliseconds, or
// wait for the device.  A block counts as in use from before it is taken, so that no other thread's
// last dev_free trims the pool under it.
cudaError_t dev_alloc_raw(void** p, size_t bytes) {
  const bool large = bytes > kPoolBlock;
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pool* q = nullptr;
    const cudaError_t e = current_pool(&q);
    if (e != cudaSuccess) return e;
    pool = q->pool;
    st = q->st;
    if (!large) q->blocks++;
  }
  cudaError_t e;
  if (large) {
    e = cudaMalloc(p, bytes);
  } else {
    e = cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), pool, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) return e;
  }
  std::lock_guard<std::mutex> lk(g_pool_mu);
  Pool* q = nullptr;
  if (current_pool(&q) != cudaSuccess) return e;
  if (e == cudaSuccess && large) q->large.insert(*p);
  if (e != cudaSuccess && !large) q->blocks--;
  if (e != cudaSuccess) cudaGetLastError();  // (reported by the caller; not by its next launch's check)
  return e;
}

void dev_free(void* p) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pool* pool = nullptr;
    if (current_pool(&pool) != cudaSuccess) return;
    if (!pool->large.erase(p)) {
      cudaFreeAsync(p, pool->st);
      if (--pool->blocks == 0) {
        cudaStreamSynchronize(pool->st);
        cudaMemPoolTrimTo(pool->pool, 0);
      }
      return;
    }
  }
  cudaFree(p);
}

// cudaDeviceSynchronize is refused while any stream of the device is being captured, by another
// thread too (a batch's graph), and spoils that capture.  Freeing a block of cudaMalloc waits as
// well, and other threads' captures allow it.  A byte that is never freed keeps the 2 MB mapped that
// such small blocks are cut from: 5 us for the two calls on an idle device, 640 us without it.
// Where not even a byte is left, it is cudaDeviceSynchronize after all, so that memory can be freed.
cudaError_t device_wait() {
  cudaError_t e = cudaSuccess;
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pool* pool = nullptr;
    e = current_pool(&pool);
    if (e == cudaSuccess && !pool->byte) e = cudaMalloc(&pool->byte, 1);
  }
  void* p = nullptr;
  if (e == cudaSuccess) e = cudaMalloc(&p, 1);
  if (e == cudaSuccess) return cudaFree(p);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  return cudaDeviceSynchronize();
}

// Streams of the current device; making and destroying one takes 50 us each, a case has up to
// five.  At most kStreamsKeep idle ones are kept, none once the last one in use comes back.
cudaError_t stream_get(cudaStream_t* st) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  Pool* pool = nullptr;
  cudaError_t e = current_pool(&pool);
  if (e != cudaSuccess) return e;
  if (!pool->streams.empty()) {
    *st = pool->streams.back();
    pool->streams.pop_back();
  } else {
    e = cudaStreamCreateWithFlags(st, cudaStreamNonBlocking);
  }
  if (e == cudaSuccess) pool->streams_out++;
  return e;
}

void stream_put(cudaStream_t st) {
  if (!st) return;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  Pool* pool = nullptr;
  if (current_pool(&pool) != cudaSuccess) return;
  constexpr size_t kStreamsKeep = 32;
  if (pool->streams.size() < kStreamsKeep) pool->streams.push_back(st);
  else cudaStreamDestroy(st);
  if (--pool->streams_out == 0) {
    for (cudaStream_t s : pool->streams) cudaStreamDestroy(s);
    pool->streams.clear();
  }
}

cudaError_t temp_alloc_raw(void** p, size_t bytes, cudaStream_t st) {
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pool* q = nullptr;
    const cudaError_t e = current_pool(&q);
    if (e != cudaSuccess) return e;
    pool = q->pool;
  }
  const cudaError_t e = cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), pool, st);
  if (e != cudaSuccess) cudaGetLastError();  // (as in dev_alloc)
  return e;
}

// (asked once for each pair: cudaMemPoolSetAccess is no call for every halo exchange)
cudaError_t pool_peer_access(int device, int peer) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (device >= (int)g_pools.size() || !g_pools[device].pool || g_pools[device].peers.count(peer)) return cudaSuccess;
  cudaMemAccessDesc d = {};
  d.location.type = cudaMemLocationTypeDevice;
  d.location.id = peer;
  d.flags = cudaMemAccessFlagsProtReadWrite;
  const cudaError_t e = cudaMemPoolSetAccess(g_pools[device].pool, &d, 1);
  if (e == cudaSuccess) g_pools[device].peers.insert(peer);
  return e;
}

void pool_share(int device) {
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (device >= (int)g_pools.size() || g_pools[device].shared) return;
    g_pools[device].shared = true;
  }
  int n = 0, can = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) n = 0;
  for (int d = 0; d < n; d++)
    if (d != device && cudaDeviceCanAccessPeer(&can, d, device) == cudaSuccess && can) pool_peer_access(device, d);
  cudaGetLastError();
}

// Small page-locked blocks (a solver's reduction results), cut from pages that are given back
// once none of their blocks is in use: page-locking costs 2 ms.
namespace {

constexpr int kPinnedBlocks = 64;
struct PinnedPage {
  char* base = nullptr;
  int used = 0;
  bool taken[kPinnedBlocks] = {};
};
std::mutex g_pinned_mu;
std::vector<PinnedPage>& g_pinned = *new std::vector<PinnedPage>;  // (as g_pools)

}  // namespace

cudaError_t pinned_alloc(double** p) {
  std::lock_guard<std::mutex> lk(g_pinned_mu);
  PinnedPage* page = nullptr;
  for (PinnedPage& g : g_pinned)
    if (g.used < kPinnedBlocks) { page = &g; break; }
  if (!page) {
    PinnedPage g;
    const cudaError_t e = cudaHostAlloc((void**)&g.base, kPinnedBlocks * kPinnedBytes, cudaHostAllocPortable);
    if (e != cudaSuccess) return e;
    g_pinned.push_back(g);
    page = &g_pinned.back();
  }
  for (int b = 0; b < kPinnedBlocks; b++)
    if (!page->taken[b]) {
      page->taken[b] = true;
      page->used++;
      *p = (double*)(page->base + b * kPinnedBytes);
      break;
    }
  return cudaSuccess;
}

void pinned_free(double* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_pinned_mu);
  for (size_t g = 0; g < g_pinned.size(); g++) {
    PinnedPage& page = g_pinned[g];
    const long off = (char*)p - page.base;
    if (off < 0 || off >= (long)(kPinnedBlocks * kPinnedBytes)) continue;
    page.taken[off / kPinnedBytes] = false;
    if (--page.used == 0) {
      cudaFreeHost(page.base);
      g_pinned.erase(g_pinned.begin() + g);
    }
    return;
  }
}

int grid_upload(const int32_t dims[3], const double* xf, const double* yf, const double* zf, cudaStream_t st,
                GridDev& gd) {
  gd.NX = dims[0]; gd.NY = dims[1]; gd.NZ = dims[2];
  const int n[3] = {gd.NX, gd.NY, gd.NZ};
  const double* f[3] = {xf, yf, zf};
  std::vector<double>* hf[3] = {&gd.hXf, &gd.hYf, &gd.hZf};
  std::vector<float>* hd[3] = {&gd.hXd, &gd.hYd, &gd.hZd};
  std::vector<float>* hc[3] = {&gd.hXc, &gd.hYc, &gd.hZc};
  for (int a = 0; a < 3; a++) {
    hf[a]->assign(f[a], f[a] + n[a] + 1);
    hd[a]->resize(n[a]);
    hc[a]->resize(n[a]);
    for (int i = 0; i < n[a]; i++) {  // centres and sizes stored in float32 (src/air_cfd.js:36)
      (*hc[a])[i] = (float)(0.5 * (f[a][i] + f[a][i + 1]));
      (*hd[a])[i] = (float)(f[a][i + 1] - f[a][i]);
    }
  }
  gd.hYd0 = gd.hYd[0];
  gd.hZd0 = gd.hZd[0];
  // one block: 3 face arrays (f64) then 9 float arrays, each padded to 256 bytes
  size_t off = 0, offs[12];
  for (int a = 0; a < 3; a++) { offs[a] = off; off += round_up((n[a] + 1) * 8, 256); }
  for (int k = 0; k < 9; k++) { offs[3 + k] = off; off += round_up(n[k % 3] * 4 + 4, 256); }
  char* base = nullptr;
  A3D_CUDA(dev_alloc(&base, off));
  gd.block = base;
  double** df[3] = {&gd.Xf, &gd.Yf, &gd.Zf};
  float** dd[3] = {&gd.Xd, &gd.Yd, &gd.Zd};
  float** dc[3] = {&gd.Xc, &gd.Yc, &gd.Zc};
  float** dr[3] = {&gd.rXd, &gd.rYd, &gd.rZd};
  for (int a = 0; a < 3; a++) {
    *df[a] = (double*)(base + offs[a]);
    *dd[a] = (float*)(base + offs[3 + a]);
    *dc[a] = (float*)(base + offs[6 + a]);
    *dr[a] = (float*)(base + offs[9 + a]);
  }
  std::vector<char> h(off, 0);  // the block's image: one copy
  for (int a = 0; a < 3; a++) {
    memcpy(&h[offs[a]], hf[a]->data(), (n[a] + 1) * 8);
    memcpy(&h[offs[3 + a]], hd[a]->data(), n[a] * 4);
    memcpy(&h[offs[6 + a]], hc[a]->data(), n[a] * 4);
    float* rec = (float*)&h[offs[9 + a]];
    for (int i = 0; i < n[a]; i++) rec[i] = 1.0f / (*hd[a])[i];
  }
  // on the stream of the kernels that read it: a copy from pageable memory returns once the source
  // is staged, which may be before it has reached the device
  A3D_CUDA(cudaMemcpyAsync(base, h.data(), off, cudaMemcpyHostToDevice, st));
  return A3D_OK;
}

void grid_free(GridDev& gd) {
  dev_free(gd.block);
  gd.block = nullptr;
}

int geom_alloc(long N, GeomDev& g) {
  const size_t fb = round_up(N * 4, 256), tb = round_up(N, 256);
  char* base = nullptr;
  A3D_CUDA(dev_alloc(&base, tb + 5 * fb));
  g.block = base;
  g.t = (uint8_t*)base;
  g.phi = (float*)(base + tb);
  g.ap0 = (float*)(base + tb + fb);
  g.ap1 = (float*)(base + tb + 2 * fb);
  g.ap2 = (float*)(base + tb + 3 * fb);
  g.ap3 = (float*)(base + tb + 4 * fb);
  return A3D_OK;
}

void geom_free(GeomDev& g) {
  dev_free(g.block);
  g.block = nullptr;
}

}  // namespace a3d

extern "C" const char* a3d_last_error(void) { return a3d::g_last_error.c_str(); }
extern "C" int a3d_abi_version(void) { return 1; }
