// geom.cu - cut-cell geometry on the GPU (cfdGeom, src/air_cfd.js:50-141).
//
// Every node of the grid and every sub-sample point of a cut cell runs the inside
// tests of the aircraft (fuselage, volume wing/tail when they are thicker than 1.5
// cells, fin, podded-nacelle envelope; src/air_cfd.js:60-67 and src/air_field.js:115-134)
// in FP64 on the device.  The kernels follow the reference's sequence:
//   node inside flags -> phi (27 samples) and +face apertures (9 samples) -> thin-wing
//   baffles (wing, then the deflected tail) -> solid test phi < 0.2 -> fixed-state jet
//   and intake layers -> face clean-up next to solids -> forced-open fixed-cell faces.
// Results are bit-identical to the reference's arithmetic wherever the device's double
// transcendentals round like the host's; the tests compare every cell.
//
// What bounds a build is latency, not its 21 bytes a cell: the inside tests' FP64 chains in the
// few cells that the surface cuts, launches and waits.  So the cut cells' samples are spread over
// their block, the engine layers are marked without the host, and everything that one cell's
// finished faces need is one pass.  (A 1M-cell airliner case from grid to free stream, with the
// force list and the codes: 700 us before, 372 us now.)
#include <algorithm>
#include <cmath>
#include <vector>
#include "geom.cuh"

namespace a3d {

namespace {

__device__ __forceinline__ double naca_t(double t, double x) {  // src/aircraft.js:58
  x = fmax(0.0, fmin(1.0, x));
  return 5 * t * (0.2969 * sqrt(x) - 0.126 * x - 0.3516 * x * x + 0.2843 * pow(x, 3.0) - 0.1036 * pow(x, 4.0));
}
__device__ __forceinline__ double naca_c(double m, double x) {  // src/aircraft.js:59, p = 0.4
  const double p = 0.4;
  if (m == 0) return 0;
  return x < p ? m / (p * p) * (2 * p * x - x * x) : m / pow(1 - p, 2.0) * ((1 - 2 * p) + 2 * p * x - x * x);
}
__device__ __forceinline__ double s_chord(const a3d_surface& S, double s) { return S.cr + (S.ct - S.cr) * s / S.semi; }
__device__ __forceinline__ double s_xle(const a3d_surface& S, double s) { return S.x0 + s * S.tanL; }
__device__ __forceinline__ double s_tc(const a3d_surface& S, double s) { return S.tcR + (S.tcT - S.tcR) * s / S.semi; }

__device__ double fus_radius(const a3d_shape& a, double x) {  // src/aircraft.js:66-72
  if (x <= 0) return 0;
  if (x < a.fus_Ln) { const double s = 1 - x / a.fus_Ln; return a.fus_R0 * pow(fmax(0.0, 1 - s * s), a.fus_noseP); }
  if (x <= a.fus_xt0) return a.fus_R0;
  if (x >= a.fus_L) return a.fus_Re;
  const double t = (x - a.fus_xt0) / a.fus_Lt;
  return a.fus_Re + (a.fus_R0 - a.fus_Re) * 0.5 * (1 + cos(kPi * t));
}
__device__ __forceinline__ double fus_center(const a3d_shape& a, double x) {  // src/aircraft.js:73
  return x <= a.fus_xt0 ? 0 : a.fus_tailUp * a.fus_R0 * pow((x - a.fus_xt0) / a.fus_Lt, 2.0);
}

// Point inside the thickness envelope of a lifting surface (AirGeom.inLift).
__device__ bool in_lift(const a3d_surface& S, double x, double ay, double z) {
  if (x < S.bb[0] || x > S.bb[1] || z < S.bb[2] || z > S.bb[3] || ay > S.semi) return false;
  const double c = s_chord(S, ay), xc = (x - s_xle(S, ay)) / c;
  if (xc < 0 || xc > 1) return false;
  const double th = naca_t(s_tc(S, ay), xc) * c * (ay >= S.semi - 1e-6 ? 0 : 1);
  const double zm = S.z0 + (ay - S.sA) * S.tanD_deg + naca_c(S.camber, xc) * c + (-(xc - 0.25) * c * S.tanI_deg);
  return z >= zm - th && z <= zm + th;
}
// Point inside the fin on the symmetry plane (AirGeom.inVt).
__device__ bool in_fin(const a3d_surface& V, double x, double ay, double z) {
  const double s = z - V.z0;
  if (s < -0.5 || s > V.semi) return false;
  const double ss = fmax(0.0, s), c = s_chord(V, ss), xc = (x - s_xle(V, ss)) / c;
  if (xc < 0 || xc > 1) return false;
  return ay <= naca_t(s_tc(V, ss), xc) * c;
}

}  // namespace

__device__ bool solid_at(const GeoDev& g, double x, double y, double z) {
  const a3d_shape& a = *g.a;
  const double ay = fabs(y);
  for (int e = 0; e < a.n_engines; e++) {  // podded nacelle envelope (float32 radius table)
    const a3d_engine& v = a.engines[e];
    if (v.internal || v.env_n == 0) continue;
    const double xe = x - v.x0;
    if (xe < 0 || xe > v.env_xmax) continue;
    const double f = xe / v.env_xmax * v.env_n;
    const int k = min(v.env_n - 1, (int)floor(f));
    const double r = (double)v.env_R[k] + ((double)v.env_R[k + 1] - (double)v.env_R[k]) * (f - k);
    if (hypot(ay - v.y, z - v.z) < r) return true;
  }
  // fuselage (AirGeom.inFus); no radius exceeds the larger of R0 and Re while noseP >= 0 (radii count
  // by their squares)
  if (x >= 0 && x <= a.fus_L && (ay <= 1.0001 * fmax(fabs(a.fus_R0), fabs(a.fus_Re)) || a.fus_noseP < 0)) {
    const double R = fus_radius(a, x), dz = z - fus_center(a, x);
    if (ay * ay + dz * dz <= R * R) return true;
  }
  if (g.volW && ay >= a.wing.sA * 0.9 && in_lift(a.wing, x, ay, z)) return true;
  if (g.volH && ay >= a.htail.sA * 0.9) {  // tail deflected by delta about its quarter root chord
    const double dx = x - g.hp0, dz = z - g.hp1;
    if (in_lift(a.htail, g.hp0 + dx * g.cR - dz * g.sR, ay, g.hp1 + dx * g.sR + dz * g.cR)) return true;
  }
  return g.volV && in_fin(a.vtail, x, ay, z);
}

namespace {

__constant__ double kSub[3] = {1.0 / 6, 0.5, 5.0 / 6};  // sub-sample offsets (src/air_cfd.js:72)

__global__ void k_nodes(GeoDev g, uint8_t* cin) {
  const long NX1 = g.NX + 1, NY1 = g.NY + 1, total = NX1 * NY1 * (g.NZ + 1);
  for (long n = blockIdx.x * (long)blockDim.x + threadIdx.x; n < total; n += (long)gridDim.x * blockDim.x) {
    const int i = (int)(n % NX1), j = (int)((n / NX1) % NY1), k = (int)(n / (NX1 * NY1));
    cin[n] = solid_at(g, g.Xf[i], g.Yf[j], g.Zf[k]) ? 1 : 0;
  }
}

// phi by 27 sub-samples, the three +face apertures by 9 sub-samples (src/air_cfd.js:73-90) and the
// solid test (src/air_cfd.js:114).  A block's 8 warps take 32 consecutive cells each, from 8 parts
// of the grid, so that the cut cells (a few per cent, side by side along the surface) are shared
// out; the block then takes the samples of its cut cells and faces one a thread.  One thread for
// all samples of its cell took 100-160 us for 1M cells of an airliner, this takes 31.
__global__ void __launch_bounds__(256) k_cells(GeoDev g, const uint8_t* __restrict__ cin, float* phi, float* ap0,
                                               float* ap1, float* ap2, float* ap3, uint8_t* t) {
  __shared__ uint16_t cut[256], face[3 * 256];  // thread; thread * 3 + direction
  __shared__ int n_cut, n_face, open[256][4];   // samples outside: of phi, of the +x, +y, +z face
  __shared__ int ijk[256][3];
  const long NX = g.NX, NY = g.NY, N = NX * NY * g.NZ;
  const long NX1 = NX + 1, NXY1 = NX1 * (NY + 1);
  const long tiles = (N + 255) / 256;
  const int tid = threadIdx.x;
  for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long q = ((tid >> 5) * tiles + tile) * 32 + (tid & 31);
    if (tid == 0) n_cut = n_face = 0;
    for (int w = 0; w < 4; w++) open[tid][w] = 0;
    __syncthreads();
    int s = 0, m[3] = {0, 0, 0};
    if (q < N) {
      const long row = q / NX;
      const int i = (int)(q - row * NX), k = (int)(row / NY), j = (int)(row - k * NY);
      ijk[tid][0] = i; ijk[tid][1] = j; ijk[tid][2] = k;
      const uint8_t* c = cin + k * NXY1 + j * NX1 + i;
      const int c000 = c[0], c100 = c[1], c010 = c[NX1], c110 = c[NX1 + 1];
      const int c001 = c[NXY1], c101 = c[NXY1 + 1], c011 = c[NXY1 + NX1], c111 = c[NXY1 + NX1 + 1];
      s = c000 + c100 + c010 + c110 + c001 + c101 + c011 + c111;
      m[0] = c100 + c110 + c101 + c111;
      m[1] = c010 + c110 + c011 + c111;
      m[2] = c001 + c101 + c011 + c111;
      if (s != 0 && s != 8) cut[atomicAdd(&n_cut, 1)] = (uint16_t)tid;
      for (int d = 0; d < 3; d++)
        if (m[d] != 0 && m[d] != 4) face[atomicAdd(&n_face, 1)] = (uint16_t)(tid * 3 + d);
    }
    __syncthreads();
    const int cuts = 27 * n_cut, samples = cuts + 9 * n_face;
    for (int u = tid; u < samples; u += 256) {
      int c, d, a, b, e;  // cell (its thread), direction of the face or -1, sample numbers along x, y, z
      if (u < cuts) {
        c = cut[u / 27]; d = -1;
        const int r = u % 27;
        a = r / 9; b = r / 3 % 3; e = r % 3;
      } else {
        const int f = face[(u - cuts) / 9], r = (u - cuts) % 9;
        c = f / 3; d = f - 3 * c;
        a = r / 3; b = d == 0 ? r / 3 : r % 3; e = r % 3;
      }
      const int i = ijk[c][0], j = ijk[c][1], k = ijk[c][2];
      double x = g.Xf[i] + kSub[a] * (double)g.Xd[i], y = g.Yf[j] + kSub[b] * (double)g.Yd[j],
             z = g.Zf[k] + kSub[e] * (double)g.Zd[k];
      if (d == 0) x = g.Xf[i + 1];
      if (d == 1) y = g.Yf[j + 1];
      if (d == 2) z = g.Zf[k + 1];
      if (!solid_at(g, x, y, z)) atomicAdd(&open[c][d + 1], 1);
    }
    __syncthreads();
    if (q < N) {
      const float ph = s == 0 ? 1.f : s == 8 ? 0.f : (float)(open[tid][0] / 27.0);
      float ap[3];
      for (int d = 0; d < 3; d++) ap[d] = m[d] == 0 ? 1.f : m[d] == 4 ? 0.f : (float)(open[tid][d + 1] / 9.0);
      phi[q] = ph;
      ap0[q] = ap[0]; ap1[q] = ap[1]; ap2[q] = ap[2]; ap3[q] = 0.f;
      t[q] = ph < 0.2 ? T_SOLID : T_FLUID;
    }
    __syncthreads();  // (the lists and counts are used again)
  }
}

// Camber-surface height of a thin surface at (x, |y|), or false outside its planform
// (zMean, src/air_cfd.js:92).
__device__ bool camber_z(const a3d_surface& S, double sA, double x, double ay, double& z) {
  if (ay > S.semi || ay < sA) return false;
  const double c = s_chord(S, ay), xc = (x - s_xle(S, ay)) / c;
  if (xc < 0 || xc > 1) return false;
  z = S.z0 + (ay - sA) * S.tanD_deg + naca_c(S.camber, xc) * c - (xc - 0.25) * c * S.tanI_deg;
  return true;
}

// Baffle on the z face nearest the mean camber surface of column (i, j), of the wing and then of
// the tail: the face aperture is reduced by the planform coverage and the local slope dz/dx is
// stored in ap3 (src/air_cfd.js:94-111).  Nine lanes per column, one a sample; the first one sums
// them in the reference's order.  Columns never share a cell.  One thread a column and one launch
// a surface took 2 x 16 us at 1M cells, this takes 9.
__global__ void __launch_bounds__(256) k_baffle(GeoDev g, float* ap2, float* ap3) {
  const long NX = g.NX, columns = NX * g.NY;
  const int lane = threadIdx.x & 31, r = lane % 9, lead = lane - r;
  const long warps = (long)gridDim.x * (blockDim.x / 32);
  for (long w = blockIdx.x * (long)(blockDim.x / 32) + threadIdx.x / 32; 3 * w < columns; w += warps) {
    const long n = 3 * w + lane / 9;
    const bool mine = lane < 27 && n < columns;
    const int i = mine ? (int)(n % NX) : 0, j = mine ? (int)(n / NX) : 0;
    for (int which = 0; which < 2; which++) {
      const a3d_surface& S = which == 0 ? g.a->wing : g.a->htail;
      const double sA = S.sA;
      double zm = 0, sl = 0;
      bool hit = false;
      if (mine && !(g.Yf[j] > S.semi || g.Yf[j + 1] < sA)) {
        const double x = g.Xf[i] + kSub[r / 3] * (double)g.Xd[i], y = g.Yf[j] + kSub[r % 3] * (double)g.Yd[j];
        double z1, z0;
        hit = camber_z(S, sA, x, y, zm);
        if (hit) {
          const double e = 0.02 * s_chord(S, fmin(y, S.semi));
          const bool ok1 = camber_z(S, sA, x + e, y, z1), ok0 = camber_z(S, sA, x - e, y, z0);
          sl = (ok1 && ok0) ? (z1 - z0) / (2 * e) : ok1 ? (z1 - zm) / e : ok0 ? (zm - z0) / e : 0;
          if (which == 1) { zm -= (x - g.hp0) * g.tdR; sl -= g.tdR; }
        }
      }
      const unsigned hits = __ballot_sync(0xffffffffu, hit);
      if (!hits) continue;
      int cov = 0;
      double zs = 0, ss = 0;
      for (int o = 0; o < 9; o++) {
        const int from = min(lead + o, 31);
        const double zo = __shfl_sync(0xffffffffu, zm, from), so = __shfl_sync(0xffffffffu, sl, from);
        if (hits >> from & 1) { cov++; zs += zo; ss += so; }
      }
      if (!mine) cov = 0;
      // first k with a centre above the surface: nine candidates a turn
      const double zmean = zs / cov;
      int k = -1;
      for (int kb = 0; __any_sync(0xffffffffu, cov != 0 && k < 0); kb += 9) {
        const bool stop = !(kb + r < g.NZ - 2 && (double)g.Zc[kb + r + 1] <= zmean);
        const unsigned stops = __ballot_sync(0xffffffffu, stop) >> lead & 0x1ffu;
        if (k < 0 && stops) k = min(kb + __ffs(stops) - 1, max(g.NZ - 2, 0));
      }
      if (cov && r == 0) {
        const long q = ((long)k * g.NY + j) * NX + i;
        ap2[q] = (float)fmin((double)ap2[q], 1 - cov / 9.0);
        ap3[q] = (float)(ss / cov);
      }
    }
  }
}

// Fixed-state layers: cells of one x layer i whose centre lies in the ring [rin, rout] around an
// engine axis become type `ty` with phi = 1 (src/air_cfd.js:123, 128); a layer that catches no
// cell centre is marked with a padded ring instead (src/air_cfd.js:124, 129).
struct Ring {
  int i, ty;
  uint8_t bit;
  double ey, ez, rin, rout, rin_pad, rout_pad;
};
struct Rings {
  static constexpr int kMax = A3D_MAX_ENGINES * (A3D_MAX_EXITS + 1);
  int n;
  Ring r[kMax];
};

// Bit x of *caught: ring x catches a cell centre.
__global__ void k_ring_caught(GeoDev g, Rings rings, unsigned* caught) {
  const long NY = g.NY, NZ = g.NZ;
  unsigned got = 0;
  for (long n = blockIdx.x * (long)blockDim.x + threadIdx.x; n < NY * NZ; n += (long)gridDim.x * blockDim.x) {
    const int j = (int)(n % NY), k = (int)(n / NY);
    for (int x = 0; x < rings.n; x++) {
      const double r = hypot((double)g.Yc[j] - rings.r[x].ey, (double)g.Zc[k] - rings.r[x].ez);
      if (r <= rings.r[x].rout && r >= rings.r[x].rin) got |= 1u << x;
    }
  }
  if (got) atomicOr(caught, got);
}

// One thread marks a (j, k) column of all rings, in the reference's engine and exit order.
__global__ void k_mark(GeoDev g, Rings rings, const unsigned* caught, uint8_t* t, float* phi, uint8_t* mark) {
  const long NY = g.NY, NZ = g.NZ;
  const unsigned got = *caught;
  for (long n = blockIdx.x * (long)blockDim.x + threadIdx.x; n < NY * NZ; n += (long)gridDim.x * blockDim.x) {
    const int j = (int)(n % NY), k = (int)(n / NY);
    for (int x = 0; x < rings.n; x++) {
      const Ring& R = rings.r[x];
      const bool pad = !(got >> x & 1);
      const double r = hypot((double)g.Yc[j] - R.ey, (double)g.Zc[k] - R.ez);
      if (r <= (pad ? R.rout_pad : R.rout) && r >= (pad ? R.rin_pad : R.rin)) {
        const long q = ((long)k * NY + j) * g.NX + R.i;
        t[q] = (uint8_t)R.ty; phi[q] = 1.f; mark[q] |= R.bit;
      }
    }
  }
}

// A cell's finished faces, from the final types:
//   apertures of faces touching a solid closed; baffle slope dropped on domain-top faces, on
//   closed faces and around fixed cells (src/air_cfd.js:132-136);
//   jet cells open their +x face toward fluid, intake cells the -x neighbour's +x face
//   (src/air_cfd.js:138; the flat index q +- 1 is used as the reference does);
//   and the numbers of solid and of cut cells (src/air_cfd.js:139).
// Two passes and a counting one with two atomics a warp took 50 us for 1M cells, this takes 18.
__global__ void __launch_bounds__(256) k_finish(int NX, int NY, int NZ, const uint8_t* __restrict__ t,
                                                const float* __restrict__ phi, const uint8_t* __restrict__ mark,
                                                float* ap0, float* ap1, float* ap2, float* ap3,
                                                unsigned long long* out) {
  const long NXY = (long)NX * NY, N = NXY * NZ;
  unsigned ns = 0, nc = 0;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < N; q += (long)gridDim.x * blockDim.x) {
    const long row = q / NX;
    const int i = (int)(q - row * NX), k = (int)(row / NY), j = (int)(row - (long)k * NY);
    const uint8_t tq = t[q], tx = q + 1 < N ? t[q + 1] : (uint8_t)T_GHOST;
    const bool solid = tq == T_SOLID;
    const float p0 = ap0[q], p1 = ap1[q], p2 = ap2[q], p3 = ap3[q];
    float a0 = p0, a1 = p1, a2 = p2, a3 = p3;
    if (i + 1 < NX && (solid || tx == T_SOLID)) a0 = 0.f;
    if (j + 1 < NY && (solid || t[q + NX] == T_SOLID)) a1 = 0.f;
    if (k + 1 >= NZ) a3 = 0.f;
    else {
      const uint8_t tz = t[q + NXY];
      if (solid || tz == T_SOLID) { a2 = 0.f; a3 = 0.f; }
      if (tz >= T_SINK) a3 = 0.f;
    }
    if (tq >= T_SINK) a3 = 0.f;
    if (q + 1 < N && (((mark[q] & 1) && tx == T_FLUID) || ((mark[q + 1] & 2) && tq == T_FLUID))) a0 = 1.f;
    if (a0 != p0) ap0[q] = a0;
    if (a1 != p1) ap1[q] = a1;
    if (a2 != p2) ap2[q] = a2;
    if (a3 != p3) ap3[q] = a3;
    if (solid) ns++;
    else if (tq == T_FLUID && (phi[q] < 1.f || a0 < 1.f || a1 < 1.f || a2 < 1.f)) nc++;
  }
  __shared__ unsigned long long sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  ns = __reduce_add_sync(0xffffffffu, ns);
  nc = __reduce_add_sync(0xffffffffu, nc);
  if ((threadIdx.x & 31) == 0) {
    if (ns) atomicAdd(&sum[0], (unsigned long long)ns);
    if (nc) atomicAdd(&sum[1], (unsigned long long)nc);
  }
  __syncthreads();
  if (threadIdx.x < 2 && sum[threadIdx.x]) atomicAdd(out + threadIdx.x, sum[threadIdx.x]);
}

int grid_blocks(long work, int threads = 256) {
  long b = (work + threads - 1) / threads;
  return (int)std::max(1L, std::min(b, 148L * 32));
}

}  // namespace

int geom_build_device(const a3d_shape& shape, const GridDev& gd, double h, double delta_deg, const GeomDev& out,
                      cudaStream_t st, int64_t counts[2], int32_t vol[3]) {
  const int NX = gd.NX, NY = gd.NY, NZ = gd.NZ;
  const long N = (long)NX * NY * NZ;
  a3d_shape* d_shape = nullptr;
  uint8_t *cin = nullptr, *mark = nullptr;
  unsigned long long* d_cnt = nullptr;
  const long nodes = (long)(NX + 1) * (NY + 1) * (NZ + 1);
  int rc = A3D_OK;
  auto fail = [&](cudaError_t e, const char* what) {
    set_error("%s: %s", what, cudaGetErrorString(e));
    rc = e == cudaErrorMemoryAllocation ? A3D_ERR_NOMEM : A3D_ERR_CUDA;
  };
  cudaError_t e;
  if ((e = temp_alloc(&d_shape, sizeof(a3d_shape), st)) != cudaSuccess) { fail(e, "device memory (shape)"); return rc; }
  if ((e = temp_alloc(&cin, nodes, st)) != cudaSuccess) fail(e, "device memory (node flags)");
  if (rc == A3D_OK && (e = temp_alloc(&mark, N, st)) != cudaSuccess) fail(e, "device memory (marks)");
  if (rc == A3D_OK && (e = temp_alloc(&d_cnt, 3 * sizeof(unsigned long long), st)) != cudaSuccess) fail(e, "device memory (counts)");
  if (rc == A3D_OK) {
    GeoDev g;
    g.a = d_shape;
    g.Xf = gd.Xf; g.Yf = gd.Yf; g.Zf = gd.Zf; g.Xd = gd.Xd; g.Yd = gd.Yd; g.Zd = gd.Zd; g.Yc = gd.Yc; g.Zc = gd.Zc;
    g.NX = NX; g.NY = NY; g.NZ = NZ;
    const a3d_surface& ht = shape.htail;
    const double dR = delta_deg * kDeg;
    g.hp0 = ht.x0 + 0 * ht.tanL + 0.25 * ht.cr;  // htail.xLE(0) + 0.25 * cr
    g.hp1 = ht.z0;
    g.cR = std::cos(dR); g.sR = std::sin(dR); g.tdR = std::tan(dR);
    auto thick = [&](const a3d_surface& S) { return 0.5 * (S.tcR * S.cr + S.tcT * S.ct) >= 1.5 * h; };
    g.volW = thick(shape.wing); g.volH = thick(ht); g.volV = thick(shape.vtail);
    if (vol) { vol[0] = g.volW; vol[1] = g.volH; vol[2] = g.volV; }
    cudaMemcpyAsync(d_shape, &shape, sizeof(a3d_shape), cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(mark, 0, N, st);
    cudaMemsetAsync(d_cnt, 0, 3 * sizeof(unsigned long long), st);
    k_nodes<<<grid_blocks(nodes), 256, 0, st>>>(g, cin);
    k_cells<<<grid_blocks(N), 256, 0, st>>>(g, cin, out.phi, out.ap0, out.ap1, out.ap2, out.ap3, out.t);
    k_baffle<<<grid_blocks(((long)NX * NY + 2) / 3 * 32), 256, 0, st>>>(g, out.ap2, out.ap3);
    // fixed-state layers, in the reference's engine/exit order
    auto layer_at = [&](double xv) { int i = 0; while (i < NX - 1 && gd.hXf[i + 1] <= xv) i++; return i; };
    Rings rings;
    rings.n = 0;
    for (int en = 0; en < std::min<int>(shape.n_engines, A3D_MAX_ENGINES); en++) {
      const a3d_engine& E = shape.engines[en];
      const double pad = 0.55 * std::max(std::max((double)gd.hYd0, (double)gd.hZd0), h);
      for (int x = 0; x < std::min<int>(shape.n_exits, A3D_MAX_EXITS); x++) {
        const a3d_exit& ex = shape.exits[x];
        rings.r[rings.n++] = {layer_at(E.x0 + ex.x - 1e-3), ex.type, 1,           E.y, E.z, ex.Rin, ex.R,
                              ex.Rin - pad,                 ex.R + pad};
      }
      if (!E.internal) {  // ring test r <= 0.9 lip_r + pad with no inner bound
        const double r = 0.9 * shape.lip_r;
        rings.r[rings.n++] = {layer_at(E.x0 + shape.lip_x + 1e-3), T_SINK, 2, E.y, E.z, -1e300, r, -1e300, r + 0.55 * h};
      }
    }
    if (rings.n) {
      k_ring_caught<<<grid_blocks((long)NY * NZ), 256, 0, st>>>(g, rings, (unsigned*)(d_cnt + 2));
      k_mark<<<grid_blocks((long)NY * NZ), 256, 0, st>>>(g, rings, (unsigned*)(d_cnt + 2), out.t, out.phi, mark);
    }
    k_finish<<<(int)std::min<long>(grid_blocks(N), 148 * 8), 256, 0, st>>>(NX, NY, NZ, out.t, out.phi, mark, out.ap0,
                                                                           out.ap1, out.ap2, out.ap3, d_cnt);
    unsigned long long hc[2] = {0, 0};
    if (counts) cudaMemcpyAsync(hc, d_cnt, sizeof(hc), cudaMemcpyDeviceToHost, st);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) fail(e, "geometry kernels");
    else if ((e = cudaGetLastError()) != cudaSuccess) fail(e, "geometry launch");
    if (counts) { counts[0] = (int64_t)hc[0]; counts[1] = (int64_t)hc[1]; }
  }
  for (void* p : {(void*)d_cnt, (void*)mark, (void*)cin, (void*)d_shape})
    if (p) cudaFreeAsync(p, st);
  cudaStreamSynchronize(st);
  return rc;
}

}  // namespace a3d

extern "C" int a3d_geom_build(const a3d_shape* shape, const int32_t dims[3], const double* xf, const double* yf,
                              const double* zf, double h, double delta_deg, uint8_t* t, float* phi, float* ap0,
                              float* ap1, float* ap2, float* ap3, int64_t counts[2], int32_t vol[3]) {
  using namespace a3d;
  clear_error();
  A3D_ARG(shape && dims && xf && yf && zf, "null pointer");
  A3D_ARG(dims[0] >= 1 && dims[1] >= 2 && dims[2] >= 1, "grid dims (NY >= 2 for the symmetry mirror)");
  A3D_TRY(use_device(-1));
  const long N = (long)dims[0] * dims[1] * dims[2];
  GridDev gd;
  GeomDev g{};
  cudaStream_t st = nullptr;
  A3D_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  int rc = grid_upload(dims, xf, yf, zf, st, gd);
  if (rc == A3D_OK) rc = geom_alloc(N, g);
  if (rc == A3D_OK) rc = geom_build_device(*shape, gd, h, delta_deg, g, st, counts, vol);
  if (rc == A3D_OK) {
    cudaError_t e = cudaSuccess;
    if (t && e == cudaSuccess) e = cudaMemcpy(t, g.t, N, cudaMemcpyDeviceToHost);
    if (phi && e == cudaSuccess) e = cudaMemcpy(phi, g.phi, N * 4, cudaMemcpyDeviceToHost);
    if (ap0 && e == cudaSuccess) e = cudaMemcpy(ap0, g.ap0, N * 4, cudaMemcpyDeviceToHost);
    if (ap1 && e == cudaSuccess) e = cudaMemcpy(ap1, g.ap1, N * 4, cudaMemcpyDeviceToHost);
    if (ap2 && e == cudaSuccess) e = cudaMemcpy(ap2, g.ap2, N * 4, cudaMemcpyDeviceToHost);
    if (ap3 && e == cudaSuccess) e = cudaMemcpy(ap3, g.ap3, N * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { set_error("geometry copy-out: %s", cudaGetErrorString(e)); rc = A3D_ERR_CUDA; }
  }
  cudaStreamSynchronize(st);  // (after an error too: the grid may still be on its way up)
  geom_free(g);
  grid_free(gd);
  cudaStreamDestroy(st);
  return rc;
}
