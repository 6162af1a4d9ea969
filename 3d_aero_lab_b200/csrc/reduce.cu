// reduce.cu - force list and the FP64 post-processing reductions of a solver case:
//   cfdForceList (src/air_cfd.js:143-152)    deterministic stream compaction in cell order
//   cfdForces    (src/air_cfd.js:443-452)    C_L, C_D, C_m over the force list
//   Trefftz CD_i (src/air_cfd.js:560-570)    transverse kinetic energy on a cross plane
//   residual     (src/air_cfd.js:552-555)    RMS density change, with a non-finite flag
//   Mach max     (src/air_cfd.js:571-572)
// Every reduction is one launch: its CTAs (a number that the problem's size alone gives) write
// partials, and the last one to finish sums them in a fixed order, so that results do not depend
// on scheduling, and writes them to page-locked host memory.  What bounds these calls is latency:
// a launch and a wait.  With a second launch to sum, a copy back and 256 CTAs for any size the
// residual (with its snapshot a copy of its own), forces, Trefftz plane and Mach maximum of an
// 825k-cell case took 46, 29, 26 and 34 us; now 23, 22, 20 and 24.
#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>
#include <algorithm>
#include <cmath>
#include <vector>
#include "solver.cuh"

namespace a3d {

namespace {

constexpr int kRedThreads = 256, kRedBlocksMax = 1184;  // 8 CTAs on each of 148 SMs
constexpr int kFlThreads = 256, kFlPerThread = 4, kFlPerBlock = kFlThreads * kFlPerThread;
constexpr double kCG = 1.4;

struct FlArgs {
  int NX, NY, NZ;
  int k0, k1;  // owned planes
  const uint8_t* t;
  const float *ap0, *ap2, *Xd, *Yd, *Zd, *Xc, *Zc;
};

// Fluid cell whose x or z aperture jumps: projected areas cx, cz (src/air_cfd.js:146-149).
__device__ __forceinline__ bool force_entry(const FlArgs& f, long q, double& cx, double& cz) {
  if (f.t[q] != T_FLUID) return false;
  const long NX = f.NX, NXY = NX * f.NY;
  const int i = (int)(q % NX), j = (int)((q / NX) % f.NY), k = (int)(q / NXY);
  if (k < f.k0 || k >= f.k1) return false;
  const double axm = i > 0 ? (double)f.ap0[q - 1] : 1.0, azm = k > 0 ? (double)f.ap2[q - NXY] : 1.0;
  cx = ((double)f.ap0[q] - axm) * (double)f.Yd[j] * (double)f.Zd[k];
  cz = ((double)f.ap2[q] - azm) * (double)f.Xd[i] * (double)f.Yd[j];
  return cx != 0 || cz != 0;
}

// Entries of each block of kFlPerBlock cells; the last block to finish turns them into the blocks'
// places in the list and writes the list's length to *total (page-locked host memory).
__global__ void __launch_bounds__(kFlThreads) k_fl_count(FlArgs f, long N, long* offsets, unsigned* finished,
                                                         double* total) {
  typedef cub::BlockReduce<int, kFlThreads> BR;
  typedef cub::BlockScan<long, kFlThreads> BS;
  __shared__ union { typename BR::TempStorage r; typename BS::TempStorage s; } tmp;
  __shared__ bool last;
  int n = 0;
  for (int e = 0; e < kFlPerThread; e++) {
    const long q = (long)blockIdx.x * kFlPerBlock + e * kFlThreads + threadIdx.x;
    double cx, cz;
    if (q < N && force_entry(f, q, cx, cz)) n++;
  }
  const int tot = BR(tmp.r).Sum(n);
  if (threadIdx.x == 0) {
    offsets[blockIdx.x] = tot;
    __threadfence();
    last = atomicAdd(finished, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  long before = 0;
  for (unsigned b0 = 0; b0 < gridDim.x; b0 += kFlThreads) {
    const unsigned b = b0 + threadIdx.x;
    const long v = b < gridDim.x ? __ldcg(offsets + b) : 0;
    long pre, all;
    BS(tmp.s).ExclusiveSum(v, pre, all);
    if (b < gridDim.x) offsets[b] = before + pre;
    before += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *finished = 0;
    *total = (double)before;
  }
}

// The entries in cell order: warp w of a block takes cells [128 w, 128 w + 128), 32 at a time.
__global__ void __launch_bounds__(kFlThreads) k_fl_write(FlArgs f, long N, const long* offsets, int64_t* oq,
                                                         double* ocx, double* ocz, double* ox, double* oz) {
  constexpr int kWarps = kFlThreads / 32;
  __shared__ int in_warp[kWarps];
  const int w = threadIdx.x / 32, lane = threadIdx.x & 31;
  const long base = (long)blockIdx.x * kFlPerBlock + w * (32 * kFlPerThread) + lane;
  unsigned hits[kFlPerThread];
  double cx[kFlPerThread], cz[kFlPerThread];
  int n = 0;
  for (int e = 0; e < kFlPerThread; e++) {
    const long q = base + 32 * e;
    hits[e] = __ballot_sync(0xffffffffu, q < N && force_entry(f, q, cx[e], cz[e]));
    n += __popc(hits[e]);
  }
  if (lane == 0) in_warp[w] = n;
  __syncthreads();
  long o = offsets[blockIdx.x];
  for (int v = 0; v < w; v++) o += in_warp[v];
  const long NX = f.NX, NXY = NX * f.NY;
  for (int e = 0; e < kFlPerThread; e++) {
    if (hits[e] >> lane & 1) {
      const long q = base + 32 * e, p = o + __popc(hits[e] & ((1u << lane) - 1));
      oq[p] = q; ocx[p] = cx[e]; ocz[p] = cz[e];
      ox[p] = f.Xc[q % NX]; oz[p] = f.Zc[q / NXY];
    }
    o += __popc(hits[e]);
  }
}

// ---- deterministic reduction of K doubles over the grid ----
struct Sum {
  static constexpr double zero = 0;
  __device__ static double join(double a, double b) { return a + b; }
};
struct Max {
  static constexpr double zero = 0;  // (of squares)
  __device__ static double join(double a, double b) { return fmax(a, b); }
};

// The CTA's joined values in thread 0.
template <class Op, int K>
__device__ __forceinline__ void block_join(double v[K]) {
  __shared__ double sh[K][kRedThreads / 32];
  for (int c = 0; c < K; c++)
    for (int o = 16; o; o >>= 1) v[c] = Op::join(v[c], __shfl_down_sync(0xffffffffu, v[c], o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();  // (sh may be in use from an earlier call)
  if (l == 0)
    for (int c = 0; c < K; c++) sh[c][w] = v[c];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int c = 0; c < K; c++) {
      double s = Op::zero;
      for (int x = 0; x < kRedThreads / 32; x++) s = Op::join(s, sh[c][x]);
      v[c] = s;
    }
}

struct RedArgs {
  double* partials;    // kRedBlocksMax x K
  unsigned* finished;  // CTAs done; 0 between launches
  double* out;         // page-locked host memory
};

// Joins v over the grid; thread 0 of the last CTA to finish has the result and true.
template <class Op, int K>
__device__ __forceinline__ bool grid_join(const RedArgs& r, double v[K]) {
  __shared__ bool last;
  block_join<Op, K>(v);
  if (threadIdx.x == 0) {
    for (int c = 0; c < K; c++) r.partials[blockIdx.x * K + c] = v[c];
    __threadfence();
    last = atomicAdd(r.finished, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int c = 0; c < K; c++) v[c] = Op::zero;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += kRedThreads)
    for (int c = 0; c < K; c++) v[c] = Op::join(v[c], __ldcg(r.partials + b * K + c));
  block_join<Op, K>(v);
  if (threadIdx.x != 0) return false;
  for (int c = 0; c < K; c++) r.out[c] = v[c];
  *r.finished = 0;
  return true;
}

struct PostArgs {
  const float* Q;  // current state, component stride Np, row pitch NXp
  long Np, N;
  long q0, q1;     // owned cells in the reference layout: [q0, q1)
  int NX, NXp;
  const uint8_t* t;  // cell types in the reference layout
  // (a grid has fewer than 2^31 cells)
  __device__ __forceinline__ long pad(long q) const {
    const uint32_t row = (uint32_t)q / (uint32_t)NX;
    return (long)row * NXp + ((uint32_t)q - row * (uint32_t)NX);
  }
};

__global__ void k_forces(PostArgs p, long n, const int64_t* fq, const double* fcx, const double* fcz,
                         const double* fx, const double* fz, double xcg, double zcg, RedArgs red) {
  double v[3] = {0, 0, 0};
  const double pinf = 1 / kCG;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const long q = p.pad(fq[e]);
    const double r = p.Q[q], u = (double)p.Q[p.Np + q] / r, vv = (double)p.Q[2 * p.Np + q] / r,
                 w = (double)p.Q[3 * p.Np + q] / r;
    const double dp = (kCG - 1) * ((double)p.Q[4 * p.Np + q] - 0.5 * r * (u * u + vv * vv + w * w)) - pinf;
    const double Fx = -dp * fcx[e], Fz = -dp * fcz[e];
    v[0] += Fx; v[1] += Fz; v[2] += (fz[e] - zcg) * Fx - (fx[e] - xcg) * Fz;
  }
  grid_join<Sum, 3>(red, v);
}

__global__ void k_trefftz(PostArgs p, int NX, int NY, int k0, int k1, int i0, double tx, double ca, double sa,
                          const float* Yd, const float* Zd, RedArgs red) {
  double v[1] = {0};
  const long M = (long)NY * (k1 - k0);
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < M; e += (long)gridDim.x * blockDim.x) {
    const int j = (int)(e % NY), k = k0 + (int)(e / NY);
    double u = 0, vv = 0, w = 0, ws = 0;
    for (int di = 0; di < 2; di++) {
      const long qr = ((long)k * NY + j) * NX + i0 + di, q = ((long)k * NY + j) * p.NXp + i0 + di;
      if (p.t[qr] != T_FLUID) continue;
      const double ww = di ? tx : 1 - tx, r = p.Q[q];
      u += ww * (double)p.Q[p.Np + q] / r;
      vv += ww * (double)p.Q[2 * p.Np + q] / r;
      w += ww * (double)p.Q[3 * p.Np + q] / r;
      ws += ww;
    }
    if (ws < 1e-6) continue;
    u /= ws; vv /= ws; w /= ws;
    const double vn = w * ca - u * sa;
    v[0] += (vv * vv + vn * vn) * (double)Yd[j] * (double)Zd[k];
  }
  grid_join<Sum, 1>(red, v);
}

// Squared density changes and their number over the sampled cells (not with `compare` 0), and the
// snapshot for the next call: one pass over the density, four cells of a padded row a thread and
// turn (rows start on 64 bytes).  out[2]: non-zero if a sampled density is not finite.
__global__ void k_residual(PostArgs p, float* prevR, int stride, int compare, RedArgs red, int* flag) {
  double v[2] = {0, 0};
  bool bad = false;
  const uint32_t quads = (uint32_t)(p.Np / 4), row_quads = (uint32_t)p.NXp / 4;
#pragma unroll 2
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < quads; e += gridDim.x * blockDim.x) {
    const float4 now = ((const float4*)p.Q)[e];
    if (compare) {
      const float4 was = ((const float4*)prevR)[e];
      const uint32_t row = e / row_quads, i = 4 * (e - row * row_quads), q = row * (uint32_t)p.NX + i;
      const float a[4] = {now.x, now.y, now.z, now.w}, b[4] = {was.x, was.y, was.z, was.w};
#pragma unroll
      for (uint32_t c = 0; c < 4; c++) {
        if (i + c >= (uint32_t)p.NX || (q + c) % (uint32_t)stride != 0) continue;
        if (q + c < p.q0 || q + c >= p.q1 || p.t[q + c] != T_FLUID) continue;
        if (!isfinite(a[c])) bad = true;
        const double d = (double)a[c] - (double)b[c];
        v[0] += d * d;
        v[1] += 1;
      }
    }
    ((float4*)prevR)[e] = now;
  }
  if (!compare) return;
  if (bad) atomicOr(flag, 1);
  __threadfence();
  if (grid_join<Sum, 2>(red, v)) red.out[2] = atomicExch(flag, 0);
}

__global__ void k_mach(PostArgs p, int stride, RedArgs red) {
  double m2max[1] = {0};
  const long M = (p.N + stride - 1) / stride;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < M; e += (long)gridDim.x * blockDim.x) {
    const long qr = e * stride, q = p.pad(qr);
    if (qr < p.q0 || qr >= p.q1 || p.t[qr] != T_FLUID) continue;
    const double r = p.Q[q], u = (double)p.Q[p.Np + q] / r, v = (double)p.Q[2 * p.Np + q] / r,
                 w = (double)p.Q[3 * p.Np + q] / r;
    const double pr = (kCG - 1) * ((double)p.Q[4 * p.Np + q] - 0.5 * r * (u * u + v * v + w * w));
    const double m2 = (u * u + v * v + w * w) / (kCG * pr / r);
    if (m2 > m2max[0]) m2max[0] = m2;
  }
  grid_join<Max, 1>(red, m2max);
}

// CTAs for `work` items: one item a thread until the chip is full.
int red_blocks(long work) {
  return (int)std::max(1L, std::min<long>((work + kRedThreads - 1) / kRedThreads, kRedBlocksMax));
}

RedArgs red_args(a3d_solver* s) {
  return {s->d_red, (unsigned*)(s->d_red + 4 * kRedBlocksMax), s->h_red};
}

PostArgs post_args(a3d_solver* s) {
  PostArgs p;
  p.Q = s->buf[s->iQ];
  p.Np = s->Np;
  p.N = s->N;
  p.NX = s->grid.NX;
  p.NXp = s->NXp;
  p.t = s->geo.t;
  const long NXY = (long)s->grid.NX * s->grid.NY;
  p.q0 = s->own_k0 * NXY;
  p.q1 = s->own_k1 * NXY;
  return p;
}

FlArgs fl_args(a3d_solver* s) {
  FlArgs f;
  f.NX = s->grid.NX; f.NY = s->grid.NY; f.NZ = s->grid.NZ;
  f.k0 = s->own_k0; f.k1 = s->own_k1;
  f.t = s->geo.t; f.ap0 = s->geo.ap0; f.ap2 = s->geo.ap2;
  f.Xd = s->grid.Xd; f.Yd = s->grid.Yd; f.Zd = s->grid.Zd; f.Xc = s->grid.Xc; f.Zc = s->grid.Zc;
  return f;
}

// cfdLocate (src/air_cfd.js:453): bracketing index and weight on the float32 centres.
void locate(const std::vector<float>& c, double v, int& i, double& tx) {
  const int n = (int)c.size();
  if (v <= c[0]) { i = 0; tx = 0; return; }
  if (v >= c[n - 1]) { i = n - 2; tx = 1; return; }
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) { const int m = (lo + hi) >> 1; if (c[m] <= v) lo = m; else hi = m; }
  i = lo;
  tx = (v - (double)c[lo]) / ((double)c[hi] - (double)c[lo]);
}

}  // namespace

// Queued on the solver's stream; the list's length is known on return.
int build_force_list(a3d_solver* s) {
  const long N = s->N;
  const long nb = (N + kFlPerBlock - 1) / kFlPerBlock;
  FlArgs f = fl_args(s);
  const RedArgs red = red_args(s);
  long* d_off = nullptr;
  A3D_CUDA(temp_alloc(&d_off, nb * sizeof(long), s->st));
  k_fl_count<<<(unsigned)nb, kFlThreads, 0, s->st>>>(f, N, d_off, red.finished, red.out);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->st);
  if (e != cudaSuccess) { cudaFreeAsync(d_off, s->st); set_error("force list count: %s", cudaGetErrorString(e)); return A3D_ERR_CUDA; }
  const long tot = (long)s->h_red[0];
  const size_t n1 = (size_t)std::max(tot, 1L);
  char* blk = nullptr;
  e = dev_alloc(&blk, n1 * (8 + 4 * 8) + 256);
  if (e != cudaSuccess) { cudaFreeAsync(d_off, s->st); set_error("force list alloc: %s", cudaGetErrorString(e)); return A3D_ERR_NOMEM; }
  s->fl.n = tot;
  s->fl.block = blk;
  s->fl.q = (int64_t*)blk;
  s->fl.cx = (double*)(blk + n1 * 8);
  s->fl.cz = s->fl.cx + n1;
  s->fl.x = s->fl.cz + n1;
  s->fl.z = s->fl.x + n1;
  k_fl_write<<<(unsigned)nb, kFlThreads, 0, s->st>>>(f, N, d_off, s->fl.q, s->fl.cx, s->fl.cz, s->fl.x, s->fl.z);
  e = cudaGetLastError();
  cudaFreeAsync(d_off, s->st);
  if (e != cudaSuccess) { set_error("force list write: %s", cudaGetErrorString(e)); return A3D_ERR_CUDA; }
  return A3D_OK;
}

}  // namespace a3d

using namespace a3d;

extern "C" int a3d_solver_force_list(a3d_solver* s, int64_t* n_out, int64_t cap, int64_t* q, double* cx, double* cz,
                                     double* x, double* z) {
  clear_error();
  A3D_ARG(s && n_out, "null pointer");
  A3D_CUDA(cudaSetDevice(s->device));
  *n_out = s->fl.n;
  const long n = std::min<long>(cap, s->fl.n);
  if (n > 0) {
    if (q) A3D_CUDA(cudaMemcpy(q, s->fl.q, n * 8, cudaMemcpyDeviceToHost));
    if (cx) A3D_CUDA(cudaMemcpy(cx, s->fl.cx, n * 8, cudaMemcpyDeviceToHost));
    if (cz) A3D_CUDA(cudaMemcpy(cz, s->fl.cz, n * 8, cudaMemcpyDeviceToHost));
    if (x) A3D_CUDA(cudaMemcpy(x, s->fl.x, n * 8, cudaMemcpyDeviceToHost));
    if (z) A3D_CUDA(cudaMemcpy(z, s->fl.z, n * 8, cudaMemcpyDeviceToHost));
  }
  return A3D_OK;
}

extern "C" int a3d_solver_forces(a3d_solver* s, double alpha_deg, double M, double S, double xcg, double zcg,
                                 double cref, double out[3]) {
  clear_error();
  A3D_ARG(s && out, "null pointer");
  A3D_CUDA(cudaSetDevice(s->device));
  k_forces<<<red_blocks(s->fl.n), kRedThreads, 0, s->st>>>(post_args(s), s->fl.n, s->fl.q, s->fl.cx, s->fl.cz,
                                                           s->fl.x, s->fl.z, xcg, zcg, red_args(s));
  A3D_CUDA(cudaGetLastError());
  A3D_CUDA(cudaStreamSynchronize(s->st));
  const double Fx = s->h_red[0], Fz = s->h_red[1], My = s->h_red[2];
  const double a = alpha_deg * kDeg, qd = 0.5 * M * M, k = 2 / (qd * S);  // src/air_cfd.js:450-451
  out[0] = k * (Fz * std::cos(a) - Fx * std::sin(a));
  out[1] = k * (Fx * std::cos(a) + Fz * std::sin(a));
  out[2] = k * My / cref;
  return A3D_OK;
}

extern "C" int a3d_solver_trefftz(a3d_solver* s, double xT, double alpha_deg, double M, double S, double* cdi) {
  clear_error();
  A3D_ARG(s && cdi, "null pointer");
  A3D_ARG(s->grid.NX >= 2, "Trefftz plane needs NX >= 2");
  A3D_CUDA(cudaSetDevice(s->device));
  int i0;
  double tx;
  locate(s->grid.hXc, xT, i0, tx);
  const double a = alpha_deg * kDeg, Mn = std::max(M, 0.05);
  const long cells = (long)s->grid.NY * (s->own_k1 - s->own_k0);
  k_trefftz<<<red_blocks(cells), kRedThreads, 0, s->st>>>(post_args(s), s->grid.NX, s->grid.NY, s->own_k0, s->own_k1,
                                                          i0, tx, std::cos(a), std::sin(a), s->grid.Yd, s->grid.Zd,
                                                          red_args(s));
  A3D_CUDA(cudaGetLastError());
  A3D_CUDA(cudaStreamSynchronize(s->st));
  *cdi = 2 * s->h_red[0] / (Mn * Mn * S);
  return A3D_OK;
}

extern "C" int a3d_solver_residual(a3d_solver* s, int32_t stride, double* res_out) {
  clear_error();
  A3D_ARG(s && res_out, "null pointer");
  A3D_ARG(stride >= 1, "stride");
  A3D_CUDA(cudaSetDevice(s->device));
  const long nIt = s->it - s->prevIt;
  double res = -1;
  int rc = A3D_OK;
  const bool compare = s->havePrev && nIt > 0;
  k_residual<<<red_blocks(s->Np / 4), kRedThreads, 0, s->st>>>(post_args(s), s->prevR, stride, compare, red_args(s), s->d_flag);
  A3D_CUDA(cudaGetLastError());
  A3D_CUDA(cudaStreamSynchronize(s->st));
  if (compare) {
    res = std::sqrt(s->h_red[0] / std::max(1.0, s->h_red[1])) / (double)nIt;
    s->res_parts[0] = s->h_red[0];
    s->res_parts[1] = s->h_red[1];
    if (s->h_red[2] != 0) { set_error("non-finite density in the state"); rc = A3D_ERR_NONFINITE; }
  }
  s->prevIt = s->it;
  s->havePrev = true;
  *res_out = res;
  return rc;
}

extern "C" int a3d_solver_mach_max(a3d_solver* s, int32_t stride, double* mmax) {
  clear_error();
  A3D_ARG(s && mmax, "null pointer");
  A3D_ARG(stride >= 1, "stride");
  A3D_CUDA(cudaSetDevice(s->device));
  k_mach<<<red_blocks((s->N + stride - 1) / stride), kRedThreads, 0, s->st>>>(post_args(s), stride, red_args(s));
  A3D_CUDA(cudaGetLastError());
  A3D_CUDA(cudaStreamSynchronize(s->st));
  *mmax = std::sqrt(s->h_red[0]);
  return A3D_OK;
}

// Planes [k0, k1) that the force list, the Trefftz plane, the residual and the Mach maximum
// cover: a z slab's own planes, without the halo planes it shares with its neighbours.
extern "C" int a3d_solver_set_owned(a3d_solver* s, int32_t k0, int32_t k1) {
  clear_error();
  A3D_ARG(s, "null solver");
  A3D_ARG(0 <= k0 && k0 < k1 && k1 <= s->grid.NZ, "owned planes must satisfy 0 <= k0 < k1 <= NZ");
  A3D_CUDA(cudaSetDevice(s->device));
  A3D_CUDA(cudaStreamSynchronize(s->st));  // (only the solver's own stream reads the list)
  s->own_k0 = k0;
  s->own_k1 = k1;
  dev_free(s->fl.block);
  s->fl = ForceList();
  A3D_TRY(build_force_list(s));
  A3D_CUDA(cudaStreamSynchronize(s->st));
  return A3D_OK;
}

extern "C" int a3d_solver_residual_parts(a3d_solver* s, double out[2]) {
  clear_error();
  A3D_ARG(s && out, "null pointer");
  out[0] = s->res_parts[0];
  out[1] = s->res_parts[1];
  return A3D_OK;
}
