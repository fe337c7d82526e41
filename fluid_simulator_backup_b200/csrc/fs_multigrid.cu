// Multigrid-preconditioned CG for the FP32 + FP64 refinement pressure solve
// of the corrected box projection (PROJECTION_3D.h:416, the system of
// POISSON_SOLVER_3D.h:1030-1214; the method has no counterpart in the
// reference, whose Jacobi-PCG is PCG_METHOD.cpp:4-126).
//
// Why.  At density ratio 1000 the red-black IC(0) iteration needs about 590
// iterations per projection at 256^3, growing with the grid.  One V-cycle as
// the preconditioner needs 8 to 15 on every grid (to 1e-6 relative; counted
// on the dam break, the rising bubble and the oil/water layers at 48^3 to
// 256^3), each costing about two of the red-black iterations.
//
// The cycle.  Cells are aggregated 2 x 2 x 2 (an odd extent leaves a half
// aggregate); restriction sums, prolongation copies, and a coarse coupling is
// half the sum of the fine couplings across the aggregates' common face.
// The Galerkin sum alone makes a smooth field twice too stiff per level in
// this piecewise-constant basis; the half restores the finite-volume
// coupling.  Every level is again a seven-point operator with zero couplings
// on the walls, two-coloured.  Smoothing is Gauss-Seidel by colours: red,
// black, red before the coarse correction (the first red sweep acts on zero,
// x = b/d, and is done by the kernel that writes b), the reverse after, so
// the cycle is symmetric and CG may use it.  Three half sweeps a side need
// 14, 10 and 7 iterations on the three scenes where two need 23, 17, 12 and
// four 12, 8, 5: the least traffic in total.  Levels of at most kMgCoarse
// cells a side run in one thread block in shared memory (four half sweeps a
// side there).
//
// Bytes.  The couplings (12 bytes per cell) are most of what a sweep would
// read, but away from the interface all faces of a cell carry its phase's
// 1/rho.  A byte per cell names that case (1: all neighbours in the phi <= 0
// phase, 2: in the other, 0: read the couplings), so that a half sweep moves
// about 6.5 bytes per cell instead of 18, the SpMV 9 instead of 20, and the
// FP64 residual 21 instead of 28 without a division.
//
// One iteration: q = A p and p.q (k_mg_spmv); x += alpha p in FP64, r -=
// alpha q, r.r (k_mg_update); the true residual b - A x in FP64 in place of
// r whenever the recursive one meets the tolerance or has dropped by
// reliable_delta (k_mg_defect, which alone decides convergence); the cycle
// z = M r; r.z (k_mg_dot); p = z + beta p (k_mg_direction).  All decisions
// are taken on the device: a solve is one graph launch and one host wait.
// Vectors are FP32 with FP64 sums, the iterate and the true residual FP64,
// as in the red-black solve.
//
// Measured (B200, CUDA events around whole calls, before: red-black IC(0)):
// a 256^3 rising-bubble timestep 646 -> 87 ms (its three solves 565 -> 30),
// a projection of 150 x 210 x 131 cells 87.2 -> 6.5 ms, of 40^3 4.8 -> 1.3 ms.
//
// r and z are stored by colour in the packed half layout of fs_redblack.cu
// (slot (h, j, k): red cell at i = 2h + ((j+k)&1), black at 2h + ((j+k+1)&1)),
// so that a half sweep reads and writes contiguous rows; x, p and q are in
// the cell layout.  The kernels of the iteration take one slot (two cells)
// per thread and move along z.
#include <cuda_bf16.h>

#include <algorithm>

#include "fs_kernels.h"

namespace fsb {

namespace {

constexpr int kBX = 32, kBY = 8;

// one level as the kernels see it
struct Lev {
  Lay L, H;
  const float *ax, *ay, *az;
  const unsigned char* cls[2];
  float* x[2];
  float* b[2];
  float a[3];   // the uniform coupling of class 1 and 2 (index 0 unused)
  float ia[3];  // its inverse
};

Lev lev_of(const MgLevel& m) {
  Lev v;
  v.L = m.L;
  v.H = m.H;
  v.ax = m.ax;
  v.ay = m.ay;
  v.az = m.az;
  for (int c = 0; c < 2; ++c) {
    v.cls[c] = m.cls[c];
    v.x[c] = m.x[c];
    v.b[c] = m.b[c];
  }
  v.a[0] = v.ia[0] = 0.0f;
  for (int c = 1; c < 3; ++c) {
    v.a[c] = m.a[c - 1];
    v.ia[c] = 1.0f / m.a[c - 1];
  }
  return v;
}

// planes per block: up to 8, fewer where that would leave the GPU idle
int chunk_of(const Lay& H) {
  const int64_t tiles = (int64_t)((H.nx + kBX - 1) / kBX) * ((H.ny + kBY - 1) / kBY);
  int c = (int)(tiles * H.nz / (148 * 8));
  return c < 1 ? 1 : (c > 8 ? 8 : c);
}
dim3 grid_of(const Lay& H, int chunk) {
  return dim3((H.nx + kBX - 1) / kBX, (H.ny + kBY - 1) / kBY, (H.nz + chunk - 1) / chunk);
}

__device__ __forceinline__ bool stopped(const MgState* st) { return ((const volatile MgState*)st)->done != 0; }

__device__ __forceinline__ int faces_inside(const Lay& L, int i, int j, int k) {
  return (i > 0) + (i < L.nx - 1) + (j > 0) + (j < L.ny - 1) + (k > 0) + (k < L.nz - 1);
}
__device__ __forceinline__ float over_faces(float v, int n) { return n == 6 ? v * (1.0f / 6.0f) : v / (float)n; }

struct Couplings {
  float xm, xp, ym, yp, zm, zp;
  __device__ __forceinline__ float sum() const { return ((xm + xp) + (ym + yp)) + (zm + zp); }
};
__device__ __forceinline__ Couplings couplings_at(const Lev& v, int64_t c) {
  return {v.ax[c], v.ax[c + 1], v.ay[c], v.ay[c + v.L.px], v.az[c], v.az[c + v.L.slab]};
}

// the first half sweep on zero: b/d
__device__ __forceinline__ float first_sweep(const Lev& v, int cl, float b, int i, int j, int k) {
  if (cl) return over_faces(b * v.ia[cl], faces_inside(v.L, i, j, k));
  const float d = couplings_at(v, v.L.at(i, j, k)).sum();
  return d > 0.0f ? b / d : 0.0f;
}

// the coarse value under fine cell (i, j, k)
__device__ __forceinline__ float coarse_at(const Lev& e, int i, int j, int k) {
  const int I = i >> 1, J = j >> 1, K = k >> 1;
  return e.x[(I + J + K) & 1][e.H.at(I >> 1, J, K)];
}

// ---------------------------------------------------------------------------
// Half sweep of one colour.  CORRECT: the first sweep after the coarse
// correction; the other colour's values are read as x + e, which is all the
// correction has to do (the swept colour's old values are not used, the
// other colour is swept next).
// ---------------------------------------------------------------------------
template <bool CORRECT>
__global__ void __launch_bounds__(kBX * kBY) k_mg_sweep(Lev v, Lev e, int color, const MgState* st, int kchunk) {
  if (stopped(st)) return;
  const Lay &L = v.L, &H = v.H;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  if (h >= H.nx || j >= H.ny) return;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  const float* __restrict__ xo = v.x[1 - color];
  const float* __restrict__ b = v.b[color];
  const unsigned char* __restrict__ cls = v.cls[color];
  float* __restrict__ x = v.x[color];
  int64_t s = H.at(h, j, k0);
  for (int k = k0; k < k1; ++k, s += H.slab) {
    const int par = (j + k + color) & 1, i = 2 * h + par;
    if (i >= L.nx) continue;
    const int cl = cls[s];
    const float bv = b[s];
    float xm = xo[s + par - 1], xp = xo[s + par];
    float ym = xo[s - H.px], yp = xo[s + H.px];
    float zm = xo[s - H.slab], zp = xo[s + H.slab];
    if (CORRECT) {
      if (i > 0) xm += coarse_at(e, i - 1, j, k);
      if (i < L.nx - 1) xp += coarse_at(e, i + 1, j, k);
      if (j > 0) ym += coarse_at(e, i, j - 1, k);
      if (j < L.ny - 1) yp += coarse_at(e, i, j + 1, k);
      if (k > 0) zm += coarse_at(e, i, j, k - 1);
      if (k < L.nz - 1) zp += coarse_at(e, i, j, k + 1);
    }
    float out;
    if (cl) {
      // neighbours beyond a wall hold 0 and are not counted
      out = over_faces(fmaf(bv, v.ia[cl], ((xm + xp) + (ym + yp)) + (zm + zp)), faces_inside(L, i, j, k));
    } else {
      const Couplings a = couplings_at(v, L.at(i, j, k));
      float num = a.xm * xm + a.xp * xp;
      num += a.ym * ym + a.yp * yp;
      num += a.zm * zm + a.zp * zp;
      const float d = a.sum();
      out = d > 0.0f ? (bv + num) / d : 0.0f;
    }
    x[s] = out;
  }
}

// residual of one cell (slot s of colour `color`) for the restriction
__device__ __forceinline__ float residual_at(const Lev& v, int color, int h, int j, int k) {
  const Lay &L = v.L, &H = v.H;
  const int par = (j + k + color) & 1, i = 2 * h + par;
  if (i >= L.nx || j >= L.ny || k >= L.nz) return 0.0f;
  const int64_t s = H.at(h, j, k);
  const float* __restrict__ xo = v.x[1 - color];
  const int cl = v.cls[color][s];
  const float xc = v.x[color][s], b = v.b[color][s];
  const float xm = xo[s + par - 1], xp = xo[s + par];
  const float ym = xo[s - H.px], yp = xo[s + H.px];
  const float zm = xo[s - H.slab], zp = xo[s + H.slab];
  if (cl) {
    const float n = (float)faces_inside(L, i, j, k);
    return fmaf(v.a[cl], (((xm + xp) + (ym + yp)) + (zm + zp)) - n * xc, b);
  }
  const Couplings a = couplings_at(v, L.at(i, j, k));
  float q = a.xm * (xm - xc) + a.xp * (xp - xc);
  // a wall's coupling is zero, so its neighbour value does not matter
  q += a.ym * (ym - xc) + a.yp * (yp - xc);
  q += a.zm * (zm - xc) + a.zp * (zp - xc);
  return b + q;
}

// Restriction: the residual of the colour that was not swept last (the other
// one's is zero) summed over each aggregate into the coarse right-hand side,
// and the coarse level's first red sweep.  The packed slots of coarse cell
// (I, J, K) are (I, 2J..2J+1, 2K..2K+1): contiguous across the warp.
__global__ void __launch_bounds__(kBX * kBY) k_mg_restrict(Lev v, Lev e, int color, const MgState* st, int kchunk) {
  if (stopped(st)) return;
  const int I = blockIdx.x * kBX + threadIdx.x, J = blockIdx.y * kBY + threadIdx.y;
  if (I >= e.L.nx || J >= e.L.ny) return;
  const int K0 = blockIdx.z * kchunk, K1 = min(e.L.nz, K0 + kchunk);
  for (int K = K0; K < K1; ++K) {
    float r = residual_at(v, color, I, 2 * J, 2 * K) + residual_at(v, color, I, 2 * J + 1, 2 * K);
    r += residual_at(v, color, I, 2 * J, 2 * K + 1) + residual_at(v, color, I, 2 * J + 1, 2 * K + 1);
    const int cc = (I + J + K) & 1;
    const int64_t s = e.H.at(I >> 1, J, K);
    e.b[cc][s] = r;
    // (the one-block levels start from zero themselves and have no classes)
    if (cc == 0 && e.cls[0]) e.x[0][s] = first_sweep(e, e.cls[0][s], r, I, J, K);
  }
}

// ---------------------------------------------------------------------------
// The small levels in one block: a whole V-cycle in shared memory.  Every
// level's arrays are padded by one cell (x and the couplings 0 there), five
// per level: x, b and the three couplings.
// ---------------------------------------------------------------------------
constexpr int kCoarseThreads = 1024;
constexpr int kCoarseSweeps = 4;

struct CoarseLev {
  int nx, ny, nz, sy, sz, n;  // extents; strides and size of the padded arrays
  int off;                    // of x in shared memory; b, ax, ay, az follow
  const float *ax, *ay, *az;
  Lay L;
};
struct CoarseArgs {
  int levels;
  CoarseLev l[kMgMaxLevels];
  float* x[2];
  float* b[2];
  Lay H;  // packed layout of the top level
};

__device__ __forceinline__ void coarse_sweep(const CoarseLev& v, float* sm, int color) {
  float* x = sm + v.off;
  const float *b = x + v.n, *ax = b + v.n, *ay = ax + v.n, *az = ay + v.n;
  const int hx = (v.nx + 1) >> 1, count = hx * v.ny * v.nz;
  for (int t = threadIdx.x; t < count; t += kCoarseThreads) {
    const int h = t % hx, row = t / hx, j = row % v.ny, k = row / v.ny;
    const int i = 2 * h + ((j + k + color) & 1);
    if (i >= v.nx) continue;
    const int c = (k + 1) * v.sz + (j + 1) * v.sy + i + 1;
    const float xm = ax[c], xp = ax[c + 1], ym = ay[c], yp = ay[c + v.sy], zm = az[c], zp = az[c + v.sz];
    const float d = ((xm + xp) + (ym + yp)) + (zm + zp);
    const float num = b[c] + (((xm * x[c - 1] + xp * x[c + 1]) + (ym * x[c - v.sy] + yp * x[c + v.sy])) +
                              (zm * x[c - v.sz] + zp * x[c + v.sz]));
    x[c] = d > 0.0f ? num / d : 0.0f;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kCoarseThreads) k_mg_coarse(CoarseArgs A, const MgState* st) {
  if (stopped(st)) return;
  extern __shared__ float sm[];
  const int tid = threadIdx.x;
  {
    const CoarseLev& last = A.l[A.levels - 1];
    const int total = last.off + 5 * last.n;
    for (int t = tid; t < total; t += kCoarseThreads) sm[t] = 0.0f;
  }
  __syncthreads();
  for (int q = 0; q < A.levels; ++q) {
    const CoarseLev& v = A.l[q];
    float* x = sm + v.off;
    const int count = v.nx * v.ny * v.nz;
    for (int t = tid; t < count; t += kCoarseThreads) {
      const int i = t % v.nx, row = t / v.nx, j = row % v.ny, k = row / v.ny;
      const int c = (k + 1) * v.sz + (j + 1) * v.sy + i + 1;
      const int64_t g = v.L.at(i, j, k);
      x[2 * v.n + c] = v.ax[g];  // the low faces; the high walls stay 0
      x[3 * v.n + c] = v.ay[g];
      x[4 * v.n + c] = v.az[g];
      if (q == 0) x[v.n + c] = A.b[(i + j + k) & 1][A.H.at(i >> 1, j, k)];
    }
  }
  __syncthreads();
  for (int q = 0; q < A.levels; ++q) {
    const CoarseLev& v = A.l[q];
    if (q == A.levels - 1) break;
    for (int m = 0; m < kCoarseSweeps; ++m) coarse_sweep(v, sm, m & 1);
    // restrict the residual
    const CoarseLev& w = A.l[q + 1];
    const float *x = sm + v.off, *b = x + v.n, *ax = b + v.n, *ay = ax + v.n, *az = ay + v.n;
    float* wb = sm + w.off + w.n;
    const int count = w.nx * w.ny * w.nz;
    for (int t = tid; t < count; t += kCoarseThreads) {
      const int I = t % w.nx, row = t / w.nx, J = row % w.ny, K = row / w.ny;
      float r = 0.0f;
      for (int m = 0; m < 8; ++m) {
        const int i = 2 * I + (m & 1), j = 2 * J + ((m >> 1) & 1), k = 2 * K + (m >> 2);
        if (i >= v.nx || j >= v.ny || k >= v.nz) continue;
        const int c = (k + 1) * v.sz + (j + 1) * v.sy + i + 1;
        const float xc = x[c];
        float s = b[c] + (ax[c] * (x[c - 1] - xc) + ax[c + 1] * (x[c + 1] - xc));
        s += ay[c] * (x[c - v.sy] - xc) + ay[c + v.sy] * (x[c + v.sy] - xc);
        s += az[c] * (x[c - v.sz] - xc) + az[c + v.sz] * (x[c + v.sz] - xc);
        r += s;
      }
      wb[(K + 1) * w.sz + (J + 1) * w.sy + I + 1] = r;
    }
    __syncthreads();
  }
  for (int q = A.levels - 1; q >= 0; --q) {
    const CoarseLev& v = A.l[q];
    if (q == A.levels - 1) {
      // the coarsest level (at most 2 cells a side): sweeps to a solve
      for (int m = 0; m < 8; ++m) coarse_sweep(v, sm, m & 1);
      for (int m = 7; m >= 0; --m) coarse_sweep(v, sm, m & 1);
      continue;
    }
    const CoarseLev& w = A.l[q + 1];
    float* x = sm + v.off;
    const float* wx = sm + w.off;
    const int count = v.nx * v.ny * v.nz;
    for (int t = tid; t < count; t += kCoarseThreads) {
      const int i = t % v.nx, row = t / v.nx, j = row % v.ny, k = row / v.ny;
      x[(k + 1) * v.sz + (j + 1) * v.sy + i + 1] += wx[((k >> 1) + 1) * w.sz + ((j >> 1) + 1) * w.sy + (i >> 1) + 1];
    }
    __syncthreads();
    for (int m = kCoarseSweeps - 1; m >= 0; --m) coarse_sweep(v, sm, m & 1);
  }
  {
    const CoarseLev& v = A.l[0];
    const float* x = sm + v.off;
    const int count = v.nx * v.ny * v.nz;
    for (int t = tid; t < count; t += kCoarseThreads) {
      const int i = t % v.nx, row = t / v.nx, j = row % v.ny, k = row / v.ny;
      A.x[(i + j + k) & 1][A.H.at(i >> 1, j, k)] = x[(k + 1) * v.sz + (j + 1) * v.sy + i + 1];
    }
  }
}

// ---------------------------------------------------------------------------
// Operator set-up
// ---------------------------------------------------------------------------

// Couplings of the low faces of each cell (FP64 from phi, stored FP32; the
// expression of the projection's coupling kernel) and the cell's class.
template <class T>
__global__ void __launch_bounds__(kBX * kBY) k_mg_build(const MgState* st, Lay L, Lay H, double rn, double rp,
                                                        double inv2, float* __restrict__ ax, float* __restrict__ ay,
                                                        float* __restrict__ az, unsigned char* __restrict__ cls0,
                                                        unsigned char* __restrict__ cls1, double* extra0, int kchunk) {
  const int i = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  if (i >= L.nx || j >= L.ny) return;
  const int k0 = blockIdx.z * kchunk, k1 = min(L.nz, k0 + kchunk);
  const T* __restrict__ phi = (const T*)st->phi;
  const double vneg = 1.0 / rn, vpos = 1.0 / rp;
  if (i == 0 && j == 0 && k0 == 0) *extra0 = 0.0;  // no deflation
  // the face between a cell and its low neighbour
  auto beta = [&](T low, T c) -> double {
    const bool nl = low <= T(0), nc = c <= T(0);
    if (nl == nc) return nc ? vneg : vpos;
    const double vl = nl ? vneg : vpos, vc = nc ? vneg : vpos, al = fabs((double)low), ac = fabs((double)c);
    return vl * vc * (ac + al) / (vc * al + vl * ac);
  };
  int64_t c = L.at(i, j, k0);
  T down = k0 > 0 ? phi[c - L.slab] : phi[c];
  T p = phi[c];
  for (int k = k0; k < k1; ++k, c += L.slab) {
    const T up = k + 1 < L.nz ? phi[c + L.slab] : p;
    const T xm = i > 0 ? phi[c - 1] : p, xp = i < L.nx - 1 ? phi[c + 1] : p;
    const T ym = j > 0 ? phi[c - L.px] : p, yp = j < L.ny - 1 ? phi[c + L.px] : p;
    ax[c] = i > 0 ? (float)(beta(xm, p) * inv2) : 0.0f;
    ay[c] = j > 0 ? (float)(beta(ym, p) * inv2) : 0.0f;
    az[c] = k > 0 ? (float)(beta(down, p) * inv2) : 0.0f;
    const bool n = p <= T(0);
    const bool same = (xm <= T(0)) == n && (xp <= T(0)) == n && (ym <= T(0)) == n && (yp <= T(0)) == n &&
                      (down <= T(0)) == n && (up <= T(0)) == n;
    (((i + j + k) & 1) ? cls1 : cls0)[H.at(i >> 1, j, k)] = same ? (n ? 1 : 2) : 0;
    down = p;
    p = up;
  }
}

// coarse couplings: half the sum of the fine couplings across the face
__global__ void __launch_bounds__(kBX * kBY) k_mg_coarsen(Lay Lf, const float* __restrict__ fx,
                                                          const float* __restrict__ fy, const float* __restrict__ fz,
                                                          Lay L, float* __restrict__ ax, float* __restrict__ ay,
                                                          float* __restrict__ az) {
  const int I = blockIdx.x * kBX + threadIdx.x, J = blockIdx.y * kBY + threadIdx.y, K = blockIdx.z;
  if (I >= L.nx || J >= L.ny) return;
  // cells past an odd extent are ghosts, whose couplings are zero
  const int64_t c = L.at(I, J, K), f = Lf.at(2 * I, 2 * J, 2 * K);
  ax[c] = 0.5f * ((fx[f] + fx[f + Lf.px]) + (fx[f + Lf.slab] + fx[f + Lf.slab + Lf.px]));
  ay[c] = 0.5f * ((fy[f] + fy[f + 1]) + (fy[f + Lf.slab] + fy[f + Lf.slab + 1]));
  az[c] = 0.5f * ((fz[f] + fz[f + 1]) + (fz[f + Lf.px] + fz[f + Lf.px + 1]));
}

// classes of a coarse level: every face inside the box carries the same
// phase's uniform coupling
__global__ void __launch_bounds__(kBX * kBY) k_mg_class(Lev v, unsigned char* __restrict__ cls0,
                                                        unsigned char* __restrict__ cls1) {
  const int i = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y, k = blockIdx.z;
  const Lay& L = v.L;
  if (i >= L.nx || j >= L.ny) return;
  const Couplings a = couplings_at(v, L.at(i, j, k));
  int cl = 0;
  for (int q = 1; q < 3; ++q) {
    const float u = v.a[q];
    if ((i == 0 || a.xm == u) && (i == L.nx - 1 || a.xp == u) && (j == 0 || a.ym == u) &&
        (j == L.ny - 1 || a.yp == u) && (k == 0 || a.zm == u) && (k == L.nz - 1 || a.zp == u))
      cl = q;
  }
  // a level of one cell has no face: read the (zero) couplings
  if (faces_inside(L, i, j, k) == 0) cl = 0;
  (((i + j + k) & 1) ? cls1 : cls0)[v.H.at(i >> 1, j, k)] = (unsigned char)cl;
}

// ---------------------------------------------------------------------------
// The iteration on the finest level: one packed slot (cells i0 = 2h, i0 + 1)
// per thread; red is cell i0 + ((j+k)&1).
// ---------------------------------------------------------------------------

// q = A p in flux form (FP32 arithmetic, each flux exact to 2 eps32 of
// itself), p.q and alpha = r.z / p.q.
__global__ void __launch_bounds__(kBX * kBY) k_mg_spmv(Lev v, const float* __restrict__ p, float* __restrict__ q,
                                                       MgState* st, double* partials, int kchunk) {
  if (stopped(st)) return;
  const Lay &L = v.L, &H = v.H;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  double pq = 0.0;
  if (h < H.nx && j < H.ny) {
    const int i0 = 2 * h;
    const bool two = i0 + 1 < L.nx;
    int64_t c = L.at(i0, j, k0), s = H.at(h, j, k0);
    auto ld2 = [&](int64_t o) { return *reinterpret_cast<const float2*>(p + o); };
    float2 dn = ld2(c - L.slab), pc = ld2(c);
    for (int k = k0; k < k1; ++k, c += L.slab, s += H.slab) {
      const float2 up = ld2(c + L.slab);
      float2 ym = ld2(c - L.px), yp = ld2(c + L.px);
      const float xl = p[c - 1], xr = p[c + 2];
      const int par = (j + k) & 1;
      const int c0 = v.cls[par][s], c1 = v.cls[1 - par][s];
      float q0, q1 = 0.0f;
      if (c0) {
        // a face on a wall carries no flux: its neighbour is read as p itself
        float f = (i0 > 0 ? pc.x - xl : 0.0f) + (two ? pc.x - pc.y : 0.0f);
        f += (j > 0 ? pc.x - ym.x : 0.0f) + (j < L.ny - 1 ? pc.x - yp.x : 0.0f);
        f += (k > 0 ? pc.x - dn.x : 0.0f) + (k < L.nz - 1 ? pc.x - up.x : 0.0f);
        q0 = v.a[c0] * f;
      } else {
        const Couplings a = couplings_at(v, c);
        q0 = a.xm * (pc.x - xl) + a.xp * (pc.x - pc.y);
        q0 += a.ym * (pc.x - ym.x) + a.yp * (pc.x - yp.x);
        q0 += a.zm * (pc.x - dn.x) + a.zp * (pc.x - up.x);
      }
      if (two) {
        if (c1) {
          float f = (pc.y - pc.x) + (i0 + 2 < L.nx ? pc.y - xr : 0.0f);
          f += (j > 0 ? pc.y - ym.y : 0.0f) + (j < L.ny - 1 ? pc.y - yp.y : 0.0f);
          f += (k > 0 ? pc.y - dn.y : 0.0f) + (k < L.nz - 1 ? pc.y - up.y : 0.0f);
          q1 = v.a[c1] * f;
        } else {
          const Couplings a = couplings_at(v, c + 1);
          q1 = a.xm * (pc.y - pc.x) + a.xp * (pc.y - xr);
          q1 += a.ym * (pc.y - ym.y) + a.yp * (pc.y - yp.y);
          q1 += a.zm * (pc.y - dn.y) + a.zp * (pc.y - up.y);
        }
        *reinterpret_cast<float2*>(q + c) = make_float2(q0, q1);
      } else {
        q[c] = q0;
      }
      pq += (double)pc.x * (double)q0 + (double)pc.y * (double)q1;  // q1 = 0 past an odd extent
      dn = pc;
      pc = up;
    }
  }
  pq = block_sum(pq);
  double tot;
  if (grid_reduce_sum(pq, partials, &st->ticket, &tot)) {
    const double alpha = st->rz / tot;
    if (!(tot > 0.0) || !isfinite(alpha)) {
      st->status = PCG_STAGNATED;  // lost its footing in this arithmetic; the caller decides
      st->done = 1;
    } else {
      st->alpha = alpha;
    }
  }
}

// x += alpha p (FP64), r -= alpha q, r.r and the first red half sweep of the
// next cycle.  The last block asks for the true residual (pause) when the
// recursive one meets the tolerance, has dropped by reliable_delta since the
// last true one, or the iteration cap is reached.
__global__ void __launch_bounds__(kBX * kBY) k_mg_update(Lev v, const float* __restrict__ p,
                                                         const float* __restrict__ q, MgState* st, double* partials,
                                                         int kchunk) {
  if (stopped(st)) return;
  const Lay &L = v.L, &H = v.H;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  const double alpha = ((const volatile MgState*)st)->alpha;
  const float al = (float)alpha;
  double* __restrict__ x = st->x;
  double rr = 0.0;
  if (h < H.nx && j < H.ny) {
    const int i0 = 2 * h;
    const bool two = i0 + 1 < L.nx;
    int64_t c = L.at(i0, j, k0), s = H.at(h, j, k0);
    for (int k = k0; k < k1; ++k, c += L.slab, s += H.slab) {
      const float2 pv = *reinterpret_cast<const float2*>(p + c), qv = *reinterpret_cast<const float2*>(q + c);
      double2 xv = *reinterpret_cast<const double2*>(x + c);
      xv.x += alpha * (double)pv.x;
      xv.y += alpha * (double)pv.y;
      if (two) *reinterpret_cast<double2*>(x + c) = xv;
      else x[c] = xv.x;
      const int par = (j + k) & 1;  // the colour of cell i0; cell i0 + 1 has the other
      float* r0 = v.b[par];
      float* r1 = v.b[1 - par];
      const float ra = r0[s] - al * qv.x;
      r0[s] = ra;
      rr += (double)ra * (double)ra;
      float rb = 0.0f;
      if (two) {
        rb = r1[s] - al * qv.y;
        r1[s] = rb;
        rr += (double)rb * (double)rb;
      }
      if (par == 0) v.x[0][s] = first_sweep(v, v.cls[0][s], ra, i0, j, k);
      else if (two) v.x[0][s] = first_sweep(v, v.cls[0][s], rb, i0 + 1, j, k);
    }
  }
  rr = block_sum(rr);
  double tot;
  if (grid_reduce_sum(rr, partials, &st->ticket, &tot)) {
    st->rr = tot;
    st->iter += 1;
    if (!isfinite(tot)) {
      st->status = PCG_STAGNATED;  // the FP32 recursion broke down; x may hold the bad step
      st->done = 1;
    } else if (tot <= st->tol2 || tot < st->delta * st->delta * st->max_rr || st->iter >= st->max_iter) {
      st->pause = 1;
    }
  }
}

// The true residual r = b - A x in FP64 (A from phi in FP64), its norm, the
// first red half sweep, and the decisions that rest on it.  INIT: the start
// of a solve (unconditional; also keeps the initial guess in st->bak).
template <class T, bool INIT>
__global__ void __launch_bounds__(kBX * kBY) k_mg_defect(Lev v, MgState* st, double* partials, double rn, double rp,
                                                         double inv2, int kchunk) {
  if (!INIT && (stopped(st) || !((const volatile MgState*)st)->pause)) return;
  const Lay &L = v.L, &H = v.H;
  const T* __restrict__ phi = (const T*)st->phi;
  const double* __restrict__ x = st->x;
  const double* __restrict__ b = st->b;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  const double vneg = 1.0 / rn, vpos = 1.0 / rp;
  double rr = 0.0;
  if (h < H.nx && j < H.ny) {
    const int i0 = 2 * h;
    const bool two = i0 + 1 < L.nx;
    int64_t c = L.at(i0, j, k0), s = H.at(h, j, k0);
    auto ld2 = [&](int64_t o) { return *reinterpret_cast<const double2*>(x + o); };
    double2 dn = ld2(c - L.slab), xc = ld2(c);
    // flux sum of one cell whose faces all carry its phase's 1/rho
    for (int k = k0; k < k1; ++k, c += L.slab, s += H.slab) {
      const double2 up = ld2(c + L.slab), ym = ld2(c - L.px), yp = ld2(c + L.px);
      const double xl = x[c - 1], xr = x[c + 2];
      const double2 bv = *reinterpret_cast<const double2*>(b + c);
      if (INIT) {
        if (two) *reinterpret_cast<double2*>(st->bak + c) = xc;
        else st->bak[c] = xc.x;
      }
      const int par = (j + k) & 1;
      double r[2] = {0.0, 0.0};
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if (m == 1 && !two) break;
        const int i = i0 + m;
        const int cl = v.cls[par ^ m][s];
        const double xv = m ? xc.y : xc.x;
        const bool okl = i > 0, okr = i < L.nx - 1, okb = j > 0, okt = j < L.ny - 1, okd = k > 0, oku = k < L.nz - 1;
        const double dl = okl ? xv - (m ? xc.x : xl) : 0.0, dr = okr ? xv - (m ? xr : xc.y) : 0.0;
        const double db = okb ? xv - (m ? ym.y : ym.x) : 0.0, dt = okt ? xv - (m ? yp.y : yp.x) : 0.0;
        const double dd = okd ? xv - (m ? dn.y : dn.x) : 0.0, du = oku ? xv - (m ? up.y : up.x) : 0.0;
        double flux;
        if (cl) {
          flux = (cl == 1 ? vneg : vpos) * (((dl + dr) + (db + dt)) + (dd + du));
        } else {
          const int64_t cc = c + m;
          const double pc = (double)phi[cc];
          flux = 0.0;
          if (okl) flux += face_coef(pc, (double)phi[cc - 1], vneg, vpos) * dl;
          if (okr) flux += face_coef(pc, (double)phi[cc + 1], vneg, vpos) * dr;
          if (okb) flux += face_coef(pc, (double)phi[cc - L.px], vneg, vpos) * db;
          if (okt) flux += face_coef(pc, (double)phi[cc + L.px], vneg, vpos) * dt;
          if (okd) flux += face_coef(pc, (double)phi[cc - L.slab], vneg, vpos) * dd;
          if (oku) flux += face_coef(pc, (double)phi[cc + L.slab], vneg, vpos) * du;
        }
        r[m] = (m ? bv.y : bv.x) - inv2 * flux;
        rr += r[m] * r[m];
        const float rf = (float)r[m];
        v.b[par ^ m][s] = rf;
        if ((par ^ m) == 0) v.x[0][s] = first_sweep(v, cl, rf, i, j, k);
      }
      dn = xc;
      xc = up;
    }
  }
  rr = block_sum(rr);
  double tot;
  if (grid_reduce_sum(rr, partials, &st->ticket, &tot)) {
    if (INIT) {
      const double bb = *st->bb_src;
      st->bb = bb;
      st->tol2 = st->tol * st->tol * bb;
      st->best = tot;
      st->rr0 = tot;
      st->rz = 0.0;
      st->beta = 0.0;
      st->iter = 0;
      st->stall = 0;
      st->outer = 1;
      st->batches = 0u;
      st->restart = 1;
      st->done = 0;
      st->status = PCG_RUNNING;
    } else {
      st->outer += 1;
      // the recursion has drifted far from the true residual: drop the direction
      st->restart = tot > 100.0 * st->rr;
    }
    st->pause = 0;
    st->rr_true = tot;
    st->max_rr = tot;
    if (!isfinite(tot) || !isfinite(st->bb)) {
      st->status = INIT ? PCG_NONFINITE : PCG_STAGNATED;
      st->done = 1;
    } else if (tot <= st->tol2 || !(st->bb > 0.0)) {
      st->status = PCG_CONVERGED;
      st->done = 1;
    } else if (st->iter >= st->max_iter) {
      st->status = PCG_MAXITER;
      st->done = 1;
    } else if (!INIT) {
      if (tot < 0.25 * st->best) st->stall = 0;
      else st->stall += 1;
      if (tot > 1.0e4 * st->best || st->stall >= 24) {
        st->status = PCG_STAGNATED;  // diverged, or no further progress
        st->done = 1;
      }
    }
    if (tot < st->best) st->best = tot;
  }
}

// r.z over both colours and beta.  The packed arrays are walked whole: z is
// zero in every slot without a cell.
__global__ void __launch_bounds__(256) k_mg_dot(Lev v, MgState* st, double* partials) {
  if (stopped(st)) return;
  const int64_t n4 = v.H.total >> 2;
  double rz = 0.0;
  for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < n4; t += (int64_t)gridDim.x * 256) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float4 a = reinterpret_cast<const float4*>(v.b[c])[t], z = reinterpret_cast<const float4*>(v.x[c])[t];
      rz += ((double)a.x * (double)z.x + (double)a.y * (double)z.y) +
            ((double)a.z * (double)z.z + (double)a.w * (double)z.w);
    }
  }
  rz = block_sum(rz);
  double tot;
  if (grid_reduce_sum(rz, partials, &st->ticket, &tot)) {
    const double old = st->rz;
    st->beta = (st->restart || !(old > 0.0)) ? 0.0 : tot / old;
    st->restart = 0;
    st->rz = tot;
    if (!isfinite(tot) || !(tot > 0.0)) {
      st->status = PCG_STAGNATED;
      st->done = 1;
    }
  }
}

// p = z + beta p.  With a loop handle one thread also continues the graph's
// loop while the solve runs (bounded by the iteration cap whatever the
// state says).
__global__ void __launch_bounds__(kBX * kBY) k_mg_direction(Lev v, float* __restrict__ p, MgState* st, int kchunk,
                                                            int loop, cudaGraphConditionalHandle handle) {
  const bool stop = stopped(st);
  if (loop && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
    const unsigned int n = st->batches + 1u;
    st->batches = n;
    cudaGraphSetConditional(handle, (!stop && n < (unsigned int)st->max_iter + 2u) ? 1u : 0u);
  }
  if (stop) return;
  const Lay &L = v.L, &H = v.H;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  if (h >= H.nx || j >= H.ny) return;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  const float beta = (float)((const volatile MgState*)st)->beta;
  const int i0 = 2 * h;
  const bool two = i0 + 1 < L.nx;
  int64_t c = L.at(i0, j, k0), s = H.at(h, j, k0);
  for (int k = k0; k < k1; ++k, c += L.slab, s += H.slab) {
    const int par = (j + k) & 1;
    float2 pv = make_float2(v.x[par][s], v.x[1 - par][s]);
    if (beta != 0.0f) {  // a restart does not read the old direction
      const float2 po = *reinterpret_cast<const float2*>(p + c);
      pv.x += beta * po.x;
      pv.y += beta * po.y;
    }
    if (two) *reinterpret_cast<float2*>(p + c) = pv;
    else p[c] = pv.x;
  }
}

// The pressure's constant.  The system is singular: CG moves the iterate in
// the range of its preconditioner, which fixes the constant of the result.
// The red-black solve conserves sum(x / dinv) over the black cells (z = dinv
// r and sum(r) = 0); the same sum is restored here, so that both solves give
// one pressure.
// Sums over the black cells: sum(x / dinv) and sum(1 / dinv), dinv the bf16
// 1/diag(S) of the red-black solve (fs_redblack.cu).
__global__ void __launch_bounds__(kBX * kBY) k_mg_anchor(Lay L, Lay H,
                                                         const unsigned short* __restrict__ dinv, MgState* st,
                                                         double* partials, int after, int kchunk) {
  if (after && ((const volatile MgState*)st)->status == PCG_STAGNATED) return;
  const double* __restrict__ x = st->x;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  double sx = 0.0, sw = 0.0;
  if (h < H.nx && j < H.ny) {
    int64_t s = H.at(h, j, k0);
    for (int k = k0; k < k1; ++k, s += H.slab) {
      const int i = 2 * h + ((j + k + 1) & 1);
      if (i >= L.nx) continue;
      const double w = (double)(1.0f / __uint_as_float((unsigned)dinv[s] << 16));
      sx += w * x[L.at(i, j, k)];
      sw += w;
    }
  }
  sx = block_sum(sx);
  sw = block_sum(sw);
  // two sums through one ticket
  __shared__ bool is_last;
  const int nb = num_blocks(), fb = flat_block();
  if (thread0()) {
    partials[fb] = sx;
    partials[nb + fb] = sw;
    __threadfence();
    is_last = atomicAdd(&st->ticket, 1u) == (unsigned int)(nb - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  const int tid = threadIdx.x + kBX * threadIdx.y;
  double a = 0.0, w = 0.0;
  for (int t = tid; t < nb; t += kBX * kBY) {
    a += __ldcg(partials + t);
    w += __ldcg(partials + nb + t);
  }
  a = block_sum(a);
  __syncthreads();
  w = block_sum(w);
  if (thread0()) {
    if (after) st->shift = w > 0.0 ? (st->anchor - a) / w : 0.0;
    else st->anchor = a;
    st->ticket = 0u;
  }
}

__global__ void __launch_bounds__(kBX * kBY) k_mg_shift(Lay L, Lay H, const MgState* st, int kchunk) {
  const double d = st->shift;
  if (st->status == PCG_STAGNATED || d == 0.0) return;
  double* __restrict__ x = st->x;
  const int h = blockIdx.x * kBX + threadIdx.x, j = blockIdx.y * kBY + threadIdx.y;
  if (h >= H.nx || j >= H.ny) return;
  const int k0 = blockIdx.z * kchunk, k1 = min(H.nz, k0 + kchunk);
  const bool two = 2 * h + 1 < L.nx;
  int64_t c = L.at(2 * h, j, k0);
  for (int k = k0; k < k1; ++k, c += L.slab) {
    if (two) {
      double2 v = *reinterpret_cast<double2*>(x + c);
      v.x += d;
      v.y += d;
      *reinterpret_cast<double2*>(x + c) = v;
    } else {
      x[c] += d;
    }
  }
}

size_t coarse_floats(int nx, int ny, int nz) { return (size_t)5 * (nx + 2) * (ny + 2) * (nz + 2); }
constexpr size_t kCoarseBytes = 220 * 1024;  // of the 227 KB a block may have

}  // namespace

// The grids of the hierarchy: halved (rounding up) until at most 2 cells a
// side; `top` is the first level from which on all fit one block.
int mg_plan(int nx, int ny, int nz, int ext[kMgMaxLevels][3], int* top) {
  int n = 0;
  for (;;) {
    ext[n][0] = nx;
    ext[n][1] = ny;
    ext[n][2] = nz;
    ++n;
    if ((nx <= 2 && ny <= 2 && nz <= 2) || n == kMgMaxLevels) break;
    nx = (nx + 1) / 2;
    ny = (ny + 1) / 2;
    nz = (nz + 1) / 2;
  }
  size_t floats = 0;
  int t = n;
  while (t > 1) {
    floats += coarse_floats(ext[t - 1][0], ext[t - 1][1], ext[t - 1][2]);
    if (floats * sizeof(float) > kCoarseBytes) break;
    --t;
  }
  *top = t;
  return n;
}

cudaError_t mg_prepare() {
  return cudaFuncSetAttribute(k_mg_coarse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseBytes);
}

int mg_max_blocks(const Lay& H) {
  const dim3 g = grid_of(H, chunk_of(H));
  return (int)std::max<int64_t>((int64_t)g.x * g.y * g.z, reduction_blocks((int64_t)1 << 40));
}

template <class T>
int mg_build(const Multigrid& M, const MgState* st, double dx, double rho_neg, double rho_pos, double* extra0,
             cudaStream_t s) {
  const MgLevel& f = M.level[0];
  {
    const int ch = chunk_of(f.L);
    k_mg_build<T><<<grid_of(f.L, ch), dim3(kBX, kBY, 1), 0, s>>>(st, f.L, f.H, rho_neg, rho_pos, 1.0 / (dx * dx),
                                                                 f.ax, f.ay, f.az, f.cls[0], f.cls[1], extra0, ch);
  }
  int launches = 1;
  for (int l = 1; l < M.levels; ++l) {
    const MgLevel &a = M.level[l - 1], &b = M.level[l];
    const dim3 g = grid_of(b.L, 1);
    k_mg_coarsen<<<g, dim3(kBX, kBY, 1), 0, s>>>(a.L, a.ax, a.ay, a.az, b.L, b.ax, b.ay, b.az);
    ++launches;
    if (l < M.top) {
      k_mg_class<<<g, dim3(kBX, kBY, 1), 0, s>>>(lev_of(b), b.cls[0], b.cls[1]);
      ++launches;
    }
  }
  return launches;
}

namespace {

// z = M r: the V-cycle on the residual in level 0's b (x's first red sweep done)
int cycle(const Multigrid& M, const MgState* st, cudaStream_t s) {
  int launches = 0;
  const dim3 blk(kBX, kBY, 1);
  for (int l = 0; l < M.top; ++l) {
    const Lev v = lev_of(M.level[l]), e = lev_of(M.level[l + 1]);
    const int ch = chunk_of(v.H);
    const dim3 g = grid_of(v.H, ch);
    k_mg_sweep<false><<<g, blk, 0, s>>>(v, e, 1, st, ch);
    k_mg_sweep<false><<<g, blk, 0, s>>>(v, e, 0, st, ch);
    const int ce = chunk_of(e.L);
    k_mg_restrict<<<grid_of(e.L, ce), blk, 0, s>>>(v, e, 1, st, ce);
    launches += 3;
  }
  CoarseArgs A{};
  size_t floats = 0;
  A.levels = M.levels - M.top;
  for (int q = 0; q < A.levels; ++q) {
    const MgLevel& m = M.level[M.top + q];
    CoarseLev& w = A.l[q];
    w.nx = m.L.nx;
    w.ny = m.L.ny;
    w.nz = m.L.nz;
    w.sy = w.nx + 2;
    w.sz = w.sy * (w.ny + 2);
    w.n = w.sz * (w.nz + 2);
    w.off = (int)floats;
    w.ax = m.ax;
    w.ay = m.ay;
    w.az = m.az;
    w.L = m.L;
    floats += 5 * (size_t)w.n;
  }
  const MgLevel& t = M.level[M.top];
  for (int c = 0; c < 2; ++c) {
    A.x[c] = t.x[c];
    A.b[c] = t.b[c];
  }
  A.H = t.H;
  k_mg_coarse<<<1, kCoarseThreads, floats * sizeof(float), s>>>(A, st);
  ++launches;
  for (int l = M.top - 1; l >= 0; --l) {
    const Lev v = lev_of(M.level[l]), e = lev_of(M.level[l + 1]);
    const int ch = chunk_of(v.H);
    const dim3 g = grid_of(v.H, ch);
    k_mg_sweep<true><<<g, blk, 0, s>>>(v, e, 0, st, ch);
    k_mg_sweep<false><<<g, blk, 0, s>>>(v, e, 1, st, ch);
    k_mg_sweep<false><<<g, blk, 0, s>>>(v, e, 0, st, ch);
    launches += 3;
  }
  return launches;
}

int direction(const Multigrid& M, float* p, MgState* st, double* partials, bool loop,
              cudaGraphConditionalHandle handle, cudaStream_t s) {
  const Lev v = lev_of(M.level[0]);
  const int ch = chunk_of(v.H);
  k_mg_dot<<<reduction_blocks(v.H.total >> 2), 256, 0, s>>>(v, st, partials);
  k_mg_direction<<<grid_of(v.H, ch), dim3(kBX, kBY, 1), 0, s>>>(v, p, st, ch, loop ? 1 : 0, handle);
  return 2;
}

}  // namespace

template <class T>
int mg_start(const Multigrid& M, float* p, MgState* st, double* partials, double dx, double rho_neg, double rho_pos,
             cudaStream_t s) {
  const Lev v = lev_of(M.level[0]);
  const int ch = chunk_of(v.H);
  k_mg_defect<T, true><<<grid_of(v.H, ch), dim3(kBX, kBY, 1), 0, s>>>(v, st, partials, rho_neg, rho_pos,
                                                                     1.0 / (dx * dx), ch);
  int n = 1 + cycle(M, st, s);
  return n + direction(M, p, st, partials, false, cudaGraphConditionalHandle{}, s);
}

template <class T>
int mg_iteration(const Multigrid& M, float* p, float* q, MgState* st, double* partials, double dx, double rho_neg,
                 double rho_pos, bool loop, cudaGraphConditionalHandle handle, cudaStream_t s) {
  const Lev v = lev_of(M.level[0]);
  const int ch = chunk_of(v.H);
  const dim3 g = grid_of(v.H, ch), blk(kBX, kBY, 1);
  k_mg_spmv<<<g, blk, 0, s>>>(v, p, q, st, partials, ch);
  k_mg_update<<<g, blk, 0, s>>>(v, p, q, st, partials, ch);
  k_mg_defect<T, false><<<g, blk, 0, s>>>(v, st, partials, rho_neg, rho_pos, 1.0 / (dx * dx), ch);
  int n = 3 + cycle(M, st, s);
  return n + direction(M, p, st, partials, loop, handle, s);
}

void mg_anchor(const Multigrid& M, const unsigned short* dinv, MgState* st, double* partials, bool after,
               cudaStream_t s) {
  const MgLevel& f = M.level[0];
  const int ch = chunk_of(f.H);
  const dim3 g = grid_of(f.H, ch), blk(kBX, kBY, 1);
  k_mg_anchor<<<g, blk, 0, s>>>(f.L, f.H, dinv, st, partials, after ? 1 : 0, ch);
  if (after) k_mg_shift<<<g, blk, 0, s>>>(f.L, f.H, st, ch);
}

__global__ void k_mg_loop_start(cudaGraphConditionalHandle handle, const MgState* st) {
  cudaGraphSetConditional(handle, stopped(st) ? 0u : 1u);
}
void mg_loop_start(cudaGraphConditionalHandle handle, const MgState* st, cudaStream_t s) {
  k_mg_loop_start<<<1, 1, 0, s>>>(handle, st);
}

template int mg_build<float>(const Multigrid&, const MgState*, double, double, double, double*, cudaStream_t);
template int mg_start<float>(const Multigrid&, float*, MgState*, double*, double, double, double, cudaStream_t);
template int mg_iteration<float>(const Multigrid&, float*, float*, MgState*, double*, double, double, double, bool,
                                 cudaGraphConditionalHandle, cudaStream_t);

}  // namespace fsb
