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
// four 12, 8, 5: the least traffic in total.  The levels that fit the
// shared memory of a cluster of blocks run in one kernel (four half sweeps a
// side there).
//
// Bytes.  The couplings (12 bytes per cell) are most of what a sweep would
// read, but away from the interface all faces of a cell carry its phase's
// 1/rho.  A byte per cell names that case (1: all neighbours in the phi <= 0
// phase, 2: in the other, 0: read the couplings), so that a half sweep moves
// about 6.5 bytes per cell instead of 18, the SpMV 9 instead of 20, and the
// FP64 residual 21 instead of 28 without a division.
//
// One iteration: the cycle z = M r, whose last two sweeps sum r.z; p = z + beta
// p (k_mg_direction); q = A p and p.q (k_mg_spmv); x += alpha p in FP64, r -=
// alpha q, r.r (k_mg_update); the true residual b - A x in FP64 in place of r
// whenever the recursive one meets the tolerance or has dropped by
// reliable_delta (k_mg_defect, which alone decides convergence and comes last, so
// that no cycle follows it, and none at all a guess that meets the tolerance).
// All decisions are taken on the device: a solve is one graph launch and one host
// wait.
// Vectors are FP32 with FP64 sums, the iterate and the true residual FP64,
// as in the red-black solve.
//
// Measured (B200, CUDA events around whole calls, before: red-black IC(0)): a
// projection of 150 x 210 x 131 cells to 1e-6 85.6 -> 5.0 ms, of 40^3 4.7 -> 1.0
// ms; the three solves of a 256^3 rising-bubble timestep 565 -> 22 ms.
//
// r and z are stored by colour in the packed half layout of fs_redblack.cu
// (slot (h, j, k): red cell at i = 2h + ((j+k)&1), black at 2h + ((j+k+1)&1)),
// so that a half sweep reads and writes contiguous rows; x, p and q are in
// the cell layout.
#include <cuda_bf16.h>

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "fs_kernels.h"

namespace cg = cooperative_groups;

namespace fsb {

namespace {

constexpr int kThreads = 256;

// one level as the kernels see it
struct Lev {
  Lay L, H;
  const float *ax, *ay, *az;
  const unsigned char* cls[2];
  const unsigned char* ccls;  // finest level: the same classes in the cell layout
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
  v.ccls = m.ccls;
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

// Launch of a kernel whose threads walk the columns of a plane (x fastest,
// `per` items along x each) up chunks of z planes.  Consecutive columns
// instead of tiles: no thread is left over at the row ends, and a thread's
// neighbours come from L1 either way.  Chunks of up to 8 planes, fewer where
// that would leave the GPU idle.
struct Columns {
  dim3 grid;
  int w, chunk;  // items per row, planes per block
};
Columns columns(int nx, int ny, int nz, int per) {
  Columns c;
  c.w = (nx + per - 1) / per;
  const int64_t bx = ((int64_t)c.w * ny + kThreads - 1) / kThreads;
  const int64_t ch = bx * nz / (148 * 12);
  c.chunk = (int)(ch < 1 ? 1 : (ch > 8 ? 8 : ch));
  c.grid = dim3((unsigned)bx, (unsigned)((nz + c.chunk - 1) / c.chunk), 1);
  return c;
}

struct Column {
  int i, j, k0, k1;  // i: the first of the thread's items, in items
  bool ok;
  __device__ __forceinline__ Column(int w, int ny, int nz, int chunk) {
    const unsigned t = blockIdx.x * (unsigned)kThreads + threadIdx.x;
    j = (int)(t / (unsigned)w);
    i = (int)(t - (unsigned)j * (unsigned)w);
    k0 = blockIdx.y * chunk;
    k1 = min(nz, k0 + chunk);
    ok = j < ny;
  }
};

__device__ __forceinline__ bool stopped(const MgState* st) { return state_read(&st->done) != 0; }

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

// W consecutive slots or cells of a thread
template <int W> struct FW {
  float v[W];
};
using F4 = FW<4>;
__device__ __forceinline__ F4 load4(const float* p) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  return {{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ void store4(float* p, const F4& a) {
  *reinterpret_cast<float4*>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}

template <int W> __device__ __forceinline__ FW<W> loadw(const float* p) {
  if constexpr (W == 4) return load4(p);
  else return {{*p}};
}
template <int W> __device__ __forceinline__ void storew(float* p, const FW<W>& a) {
  if constexpr (W == 4) store4(p, a);
  else *p = a.v[0];
}
template <int W> __device__ __forceinline__ unsigned classes(const unsigned char* p) {  // a byte each
  if constexpr (W == 4) return *reinterpret_cast<const unsigned*>(p);
  else return *p;
}

// The coarse values over slots h .. h+3 (coarse cells I = h .. h+3, h a
// multiple of 4) of a row in coarse row (J, K): two of each colour.  Coarse
// ghosts hold 0.
__device__ __forceinline__ F4 coarse4(const Lev& e, int h, int J, int K) {
  const int g = (J + K) & 1;  // the colour of the even ones
  const int64_t s = e.H.at(h >> 1, J, K);
  const float2 a = *reinterpret_cast<const float2*>(e.x[g] + s), b = *reinterpret_cast<const float2*>(e.x[1 - g] + s);
  return {{a.x, b.x, a.y, b.y}};
}
__device__ __forceinline__ float coarse1(const Lev& e, int I, int J, int K) {
  return e.x[(I + J + K) & 1][e.H.at(I >> 1, J, K)];
}

template <int W> __device__ __forceinline__ FW<W> coarsew(const Lev& e, int h, int J, int K) {
  if constexpr (W == 4) return coarse4(e, h, J, K);
  else return {{coarse1(e, h, J, K)}};
}

// ---------------------------------------------------------------------------
// Half sweep of one colour, four slots per thread (W).  The other colour's values
// in the thread's row are one vector (slot h holds the x neighbours of slots h
// and h -+ 1) and, plane by plane, also its z neighbours: marching up, a plane
// costs one new vector of them, the two y rows, b, one neighbouring slot and
// four class bytes.  Measured at 256^3 against one slot per thread (whose
// loads waited on the class byte, 30 % of HBM) and a dot product of its own:
// the last black and red sweep and r.z 41 + 41 + 39 -> 32 + 39 us, the
// restriction 71 -> 48, the SpMV (likewise four cells) 77 -> 52, the update
// 153 -> 112.
//
// W = 1 on grids where four would leave SMs idle (wide()): there the time is one
// chain of loads, four times as long at the interface.  A half sweep with four and
// with one: 48^3 5.4 -> 3.1 us, 75 x 105 x 66 8.8 -> 5.4, but on 96^3 (480 blocks with
// four, against the rule's 444) 9.3 -> 12.9 with r.z; a restriction onto 40^3 and
// smaller 7 -> 5.
//
// CORRECT: the first sweep after the coarse correction; the other colour's
// values are read as x + e, which is all the correction has to do (the swept
// colour's old values are not used, the other colour is swept next).  Values
// past the box stay 0.
// DOT: the last black (1) and red (2) sweep on the finest level also sum r.z;
// the red one's last block adds both up and sets beta.
// ---------------------------------------------------------------------------
template <int W, bool CORRECT, int DOT>
__global__ void __launch_bounds__(kThreads) k_mg_sweep(Lev v, Lev e, int color, MgState* st, double* partials, int w,
                                                       int chunk) {
  if (stopped(st)) return;
  const Lay &L = v.L, &H = v.H;
  const Column q(w, H.ny, H.nz, chunk);
  double rz = 0.0;
  if (q.ok) {
    const int h = W * q.i, j = q.j;
    const float* __restrict__ xo = v.x[1 - color];
    const float* __restrict__ b = v.b[color];
    const unsigned char* __restrict__ cls = v.cls[color];
    float* __restrict__ x = v.x[color];
    int64_t s = H.at(h, j, q.k0);
    const int fyz0 = (j > 0) + (j < L.ny - 1);
    // other colour's row at plane k: x + e, zero in slots without a cell.
    // Slot m's cell of that colour is at i = 2 (h + m) + (1 - par).
    auto correct = [&](FW<W>& r, int par, int k) {
      const FW<W> c = coarsew<W>(e, h, j >> 1, k >> 1);
#pragma unroll
      for (int m = 0; m < W; ++m)
        if (2 * (h + m) + 1 - par < L.nx) r.v[m] += c.v[m];
    };
    const int p0 = (j + q.k0 + color) & 1;
    FW<W> zm = loadw<W>(xo + s - H.slab), xc = loadw<W>(xo + s);
    if (CORRECT) {
      if (q.k0 > 0) correct(zm, 1 - p0, q.k0 - 1);
      correct(xc, p0, q.k0);
    }
    for (int k = q.k0; k < q.k1; ++k, s += H.slab) {
      const int par = (j + k + color) & 1;
      FW<W> zp = loadw<W>(xo + s + H.slab);
      FW<W> ym = loadw<W>(xo + s - H.px), yp = loadw<W>(xo + s + H.px);
      const FW<W> bv = loadw<W>(b + s);
      const unsigned cl = classes<W>(cls + s);
      float side = xo[par ? s + W : s - 1];
      if (CORRECT) {
        if (k < L.nz - 1) correct(zp, 1 - par, k + 1);
        const FW<W> cm = coarsew<W>(e, h, (j - 1) >> 1, k >> 1);
#pragma unroll
        for (int m = 0; m < W; ++m) ym.v[m] += cm.v[m];  // (a ghost row's coarse row is a ghost too)
        if (j < L.ny - 1) {
          const FW<W> cp = coarsew<W>(e, h, (j + 1) >> 1, k >> 1);
#pragma unroll
          for (int m = 0; m < W; ++m) yp.v[m] += cp.v[m];
        }
        if (par) {
          if (2 * (h + W) < L.nx) side += coarse1(e, h + W, j >> 1, k >> 1);
        } else if (h > 0) {
          side += coarse1(e, h - 1, j >> 1, k >> 1);
        }
      }
      const int fyz = fyz0 + (k > 0) + (k < L.nz - 1);
      FW<W> out;
      const int c0 = cl & 255u;
      if (c0 && cl == (W == 4 ? 0x01010101u : 1u) * c0) {
        const float ia = v.ia[c0];
#pragma unroll
        for (int m = 0; m < W; ++m) {
          const int i = 2 * (h + m) + par;
          const float xs = par ? (m < W - 1 ? xc.v[m + 1] : side) : (m > 0 ? xc.v[m - 1] : side);
          // neighbours beyond a wall hold 0 and are not counted
          const float sum = fmaf(bv.v[m], ia, ((xc.v[m] + xs) + (ym.v[m] + yp.v[m])) + (zm.v[m] + zp.v[m]));
          out.v[m] = over_faces(sum, fyz + (i > 0) + (i < L.nx - 1));
        }
      } else {
#pragma unroll
        for (int m = 0; m < W; ++m) {
          const int i = 2 * (h + m) + par;
          out.v[m] = 0.0f;
          if (i >= L.nx) continue;
          const float xs = par ? (m < W - 1 ? xc.v[m + 1] : side) : (m > 0 ? xc.v[m - 1] : side);
          const int cm = (cl >> (8 * m)) & 255u;
          if (cm) {
            const float sum = fmaf(bv.v[m], v.ia[cm], ((xc.v[m] + xs) + (ym.v[m] + yp.v[m])) + (zm.v[m] + zp.v[m]));
            out.v[m] = over_faces(sum, fyz + (i > 0) + (i < L.nx - 1));
          } else {
            const Couplings a = couplings_at(v, L.at(i, j, k));
            float num = par ? a.xm * xc.v[m] + a.xp * xs : a.xm * xs + a.xp * xc.v[m];
            num += a.ym * ym.v[m] + a.yp * yp.v[m];
            num += a.zm * zm.v[m] + a.zp * zp.v[m];
            const float d = a.sum();
            out.v[m] = d > 0.0f ? (bv.v[m] + num) / d : 0.0f;
          }
        }
      }
      storew<W>(x + s, out);
      if (DOT) {
#pragma unroll
        for (int m = 0; m < W; ++m) rz += (double)bv.v[m] * (double)out.v[m];
      }
      zm = xc;
      xc = zp;
    }
  }
  if (DOT) {
    rz = block_sum(rz);
    const int nb = num_blocks();
    if (DOT == 1) {
      if (thread0()) partials[flat_block()] = rz;
      return;
    }
    // two ranges of partial sums: the black sweep's, then this one's
    __shared__ bool is_last;
    if (thread0()) {
      partials[nb + flat_block()] = rz;
      __threadfence();
      is_last = atomicAdd(&st->ticket, 1u) == (unsigned)(nb - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double sum = 0.0;
#pragma unroll 4
    for (int t = threadIdx.x; t < 2 * nb; t += kThreads) sum += __ldcg(partials + t);
    sum = block_sum(sum);
    if (thread0()) {
      st->ticket = 0u;
      const double old = st->rz;
      st->beta = (st->restart || !(old > 0.0)) ? 0.0 : sum / old;
      st->restart = 0;
      st->rz = sum;
      if (!isfinite(sum) || !(sum > 0.0)) {
        st->status = PCG_STAGNATED;
        st->done = 1;
      }
    }
  }
}

// Residual of W slots of one row (colour `color`, the one not swept last),
// zero in slots without a cell.
template <int W>
__device__ __forceinline__ FW<W> residualw(const Lev& v, int color, int h, int j, int k) {
  FW<W> r{};
  const Lay &L = v.L, &H = v.H;
  if (j >= L.ny || k >= L.nz) return r;
  const int par = (j + k + color) & 1;
  const int64_t s = H.at(h, j, k);
  const float* __restrict__ xo = v.x[1 - color];
  const FW<W> xc = loadw<W>(xo + s), ym = loadw<W>(xo + s - H.px), yp = loadw<W>(xo + s + H.px), zm = loadw<W>(xo + s - H.slab),
           zp = loadw<W>(xo + s + H.slab), own = loadw<W>(v.x[color] + s), b = loadw<W>(v.b[color] + s);
  const unsigned cl = classes<W>(v.cls[color] + s);
  const float side = xo[par ? s + W : s - 1];
  const int fyz = (j > 0) + (j < L.ny - 1) + (k > 0) + (k < L.nz - 1);
#pragma unroll
  for (int m = 0; m < W; ++m) {
    const int i = 2 * (h + m) + par;
    if (i >= L.nx) continue;
    const float xs = par ? (m < W - 1 ? xc.v[m + 1] : side) : (m > 0 ? xc.v[m - 1] : side);
    const float o = own.v[m];
    const int cm = (cl >> (8 * m)) & 255u;
    if (cm) {
      const float n = (float)(fyz + (i > 0) + (i < L.nx - 1));
      r.v[m] = fmaf(v.a[cm], (((xc.v[m] + xs) + (ym.v[m] + yp.v[m])) + (zm.v[m] + zp.v[m])) - n * o, b.v[m]);
    } else {
      // a wall's coupling is zero, so its neighbour value does not matter
      const Couplings a = couplings_at(v, L.at(i, j, k));
      float q = par ? a.xm * (xc.v[m] - o) + a.xp * (xs - o) : a.xm * (xs - o) + a.xp * (xc.v[m] - o);
      q += a.ym * (ym.v[m] - o) + a.yp * (yp.v[m] - o);
      q += a.zm * (zm.v[m] - o) + a.zp * (zp.v[m] - o);
      r.v[m] = b.v[m] + q;
    }
  }
  return r;
}

// Restriction: the residual of the colour that was not swept last (the other
// one's is zero) summed over each aggregate into the coarse right-hand side,
// and the coarse level's first red sweep.  The packed slots of coarse cell
// (I, J, K) are (I, 2J..2J+1, 2K..2K+1): a thread takes W coarse cells.
template <int W>
__global__ void __launch_bounds__(kThreads) k_mg_restrict(Lev v, Lev e, int color, const MgState* st, int w,
                                                          int chunk) {
  if (stopped(st)) return;
  const Column q(w, e.L.ny, e.L.nz, chunk);
  if (!q.ok) return;
  const int I = W * q.i, J = q.j;
  for (int K = q.k0; K < q.k1; ++K) {
    const FW<W> a = residualw<W>(v, color, I, 2 * J, 2 * K), b = residualw<W>(v, color, I, 2 * J + 1, 2 * K),
             c = residualw<W>(v, color, I, 2 * J, 2 * K + 1), d = residualw<W>(v, color, I, 2 * J + 1, 2 * K + 1);
    FW<W> r;
#pragma unroll
    for (int m = 0; m < W; ++m) r.v[m] = (a.v[m] + b.v[m]) + (c.v[m] + d.v[m]);
    const int g = (J + K) & 1;  // the colour of the even coarse cells; cells past the box got 0
    const int64_t s = e.H.at(I >> 1, J, K);
    if constexpr (W == 4) {
      *reinterpret_cast<float2*>(e.b[g] + s) = make_float2(r.v[0], r.v[2]);
      *reinterpret_cast<float2*>(e.b[1 - g] + s) = make_float2(r.v[1], r.v[3]);
      // (the cluster's levels start from zero themselves and have no classes)
      if (e.cls[0]) {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int Ir = I + 2 * m + g;  // red: even when g = 0, odd when g = 1
          if (Ir < e.L.nx) e.x[0][s + m] = first_sweep(e, e.cls[0][s + m], g ? r.v[2 * m + 1] : r.v[2 * m], Ir, J, K);
        }
      }
    } else {
      const int own = (I + g) & 1;
      e.b[own][s] = r.v[0];
      if (own == 0 && e.cls[0]) e.x[0][s] = first_sweep(e, e.cls[0][s], r.v[0], I, J, K);
    }
  }
}

// ---------------------------------------------------------------------------
// The small levels in one cluster of thread blocks: a whole V-cycle in the
// shared memory of up to 16 SMs.  A level of more than kSplitSlots slots is
// split into slabs along z, one per block, whose x has a halo plane on each
// side: a block that relaxes a cell of its first or last plane writes the
// value into the neighbour's halo too, and the cluster's barrier after each
// half sweep makes it visible.  The levels below run in the first block, those
// of at most 32 cells a colour in its first warp, without block barriers.
// The arrays of a level (x, b, 1/d and the three couplings) share one zero
// cell between rows and one zero row between planes, which stand for the walls.
//
// What bounds it: latency (a barrier and a chain of shared reads per half sweep,
// about 0.3 us in one block, 1 us with the cluster's barrier) and the fetch of
// its instructions, which every launch repeats: with the sweeps unrolled it takes
// 37 us at 40^3, with loops 30 us; slabs of more than two slots a thread (38 x
// 53 x 33) are slower than the six grid kernels of a level.  Measured, a whole
// projection to 1e-6 with the levels above 16^3 as grid kernels and one block for
// the rest -> so: 40^3 1.21 -> 1.00 ms, 64^3 1.55 -> 1.26, 96^3 2.09 -> 1.94.
// ---------------------------------------------------------------------------
constexpr int kCoarseThreads = 1024;
constexpr int kCoarseSweeps = 4;
constexpr int kCoarseItems = 2;      // slots of one colour per thread: up to 2048 per slab, 1024 unsplit
constexpr int kWarpCells = 32;       // of one colour: levels of one warp
constexpr int kSplitSlots = 512;     // larger levels are split

struct CoarseLev {
  int nx, ny, nz, sy, sz;  // extents; strides of the arrays
  int split;               // over the cluster's blocks, else in the first one
  int off;                 // of x in shared memory (planes + 2 planes of it)
  int b, d, ax, ay, az;    // of the others from x, indexed as x is (no halo planes; az: the upper one)
  const float *gx, *gy, *gz;
  Lay L;
};
struct CoarseArgs {
  int levels, floats;
  CoarseLev l[kMgMaxLevels];
  float* x[2];
  float* b[2];
  Lay H;  // packed layout of the top level
};

__host__ __device__ __forceinline__ int coarse_slots(int nx, int ny, int nz) { return ((nx + 1) >> 1) * ny * nz; }

// the planes k0 .. k0 + n - 1 of a level that a block owns
struct Slab {
  int k0, n;
};
__device__ __forceinline__ Slab slab_of(const CoarseLev& v, int rank, int blocks) {
  if (!v.split) return {0, rank == 0 ? v.nz : 0};
  const int k0 = v.nz * rank / blocks;
  return {k0, v.nz * (rank + 1) / blocks - k0};
}
__device__ __forceinline__ int owner_of(const CoarseLev& v, int k, int blocks) {
  return v.split ? ((k + 1) * blocks - 1) / v.nz : 0;
}

__device__ __forceinline__ float coarse_relax(const CoarseLev& v, const float* x, int c) {
  const float *ax = x + v.ax, *ay = x + v.ay, *az = x + v.az;
  const float num = x[v.b + c] +
                    (((ax[c] * x[c - 1] + ax[c + 1] * x[c + 1]) + (ay[c] * x[c - v.sy] + ay[c + v.sy] * x[c + v.sy])) +
                     (az[c] * x[c - v.sz] + az[c + v.sz] * x[c + v.sz]));
  return num * x[v.d + c];
}
__device__ __forceinline__ float coarse_residual(const CoarseLev& v, const float* x, int c) {
  const float *ax = x + v.ax, *ay = x + v.ay, *az = x + v.az;
  const float xc = x[c];
  float s = x[v.b + c] + (ax[c] * (x[c - 1] - xc) + ax[c + 1] * (x[c + 1] - xc));
  s += ay[c] * (x[c - v.sy] - xc) + ay[c + v.sy] * (x[c + v.sy] - xc);
  s += az[c] * (x[c - v.sz] - xc) + az[c + v.sz] * (x[c + v.sz] - xc);
  return s;
}

// The slots a thread owns on a level: the index of the cell at i = 2h, and
// whether the slot's cells exist (a half slot at the end of an odd row has one
// cell only, marked).  below, above: where the neighbours' halo planes hold
// this slab's first and last plane (nullptr: none).
template <int N>
struct CoarseItems {
  int c[N];             // -1: none
  unsigned par, half;   // bit m: (j + k) & 1; cell 2h + 1 does not exist
  float *below, *above;
  int last;             // first index of the last plane
  __device__ __forceinline__ void init(const CoarseLev& v, const Slab& z, int tid, int threads) {
    const int hx = (v.nx + 1) >> 1, count = hx * v.ny * z.n;
    par = half = 0u;
    below = above = nullptr;
    last = z.n * v.sz;
#pragma unroll
    for (int m = 0; m < N; ++m) {
      const int t = tid + m * threads;
      c[m] = -1;
      if (t < count) {
        const int h = t % hx, row = t / hx, j = row % v.ny, k = row / v.ny;
        c[m] = (k + 1) * v.sz + j * v.sy + 2 * h;
        par |= (unsigned)((j + z.k0 + k) & 1) << m;
        half |= (unsigned)(2 * h + 1 >= v.nx) << m;
      }
    }
  }
  __device__ __forceinline__ void neighbours(const CoarseLev& v, const Slab& z, float* x, int blocks,
                                             const cg::cluster_group& cl) {
    if (!v.split || z.n == 0) return;
    if (z.k0 > 0) {
      const int r = owner_of(v, z.k0 - 1, blocks);
      below = cl.map_shared_rank(x, r) + slab_of(v, r, blocks).n * v.sz;
    }
    if (z.k0 + z.n < v.nz) above = cl.map_shared_rank(x, owner_of(v, z.k0 + z.n, blocks)) - z.n * v.sz;
  }
  __device__ __forceinline__ void store(const CoarseLev& v, float* x, int at, float value) const {
    x[at] = value;
    if (below && at < 2 * v.sz) below[at] = value;
    if (above && at >= last) above[at] = value;
  }
  __device__ __forceinline__ void sweep(const CoarseLev& v, float* x, int color) const {
#pragma unroll
    for (int m = 0; m < N; ++m) {
      if (c[m] < 0) continue;
      const int o = ((par >> m) ^ color) & 1;
      if (o && ((half >> m) & 1)) continue;
      store(v, x, c[m] + o, coarse_relax(v, x, c[m] + o));
    }
  }
};

// The residual of this block's planes of level v, summed into level w's b in
// the blocks that own it: each fine plane adds its two cells per coarse cell
// (two planes at most add to one, so the sum does not depend on their order).
// Black was swept last, its residual is zero: only the red cells count.
__device__ __forceinline__ void coarse_restrict(const CoarseLev& v, const CoarseLev& w, const Slab& z, float* sm,
                                                int blocks, const cg::cluster_group& cl, int tid, int threads) {
  const float* x = sm + v.off;
  const int plane = w.nx * w.ny, count = plane * z.n;
  for (int t = tid; t < count; t += threads) {
    const int lk = t / plane, k = z.k0 + lk, K = k >> 1, rest = t - lk * plane, J = rest / w.nx, I = rest - J * w.nx;
    float r = 0.0f;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int j = 2 * J + m, i = 2 * I + ((j + k) & 1);
      if (i < v.nx && j < v.ny) r += coarse_residual(v, x, (lk + 1) * v.sz + j * v.sy + i);
    }
    const int own = owner_of(w, K, blocks);
    float* wb = sm + w.off + w.b + (K - slab_of(w, own, blocks).k0 + 1) * w.sz + J * w.sy + I;
    atomicAdd(own == (int)cl.block_rank() ? wb : cl.map_shared_rank(wb, own), r);
  }
}
template <int N>
__device__ __forceinline__ void coarse_prolong(const CoarseLev& v, const CoarseLev& w, const Slab& z,
                                               const CoarseItems<N>& it, float* sm, int blocks,
                                               const cg::cluster_group& cl) {
  float* x = sm + v.off;
#pragma unroll
  for (int m = 0; m < N; ++m) {
    if (it.c[m] < 0) continue;
    const int lk = it.c[m] / v.sz - 1, rest = it.c[m] - (lk + 1) * v.sz, j = rest / v.sy, i = rest - j * v.sy;
    const int K = (z.k0 + lk) >> 1, own = owner_of(w, K, blocks);
    const float* wx = sm + w.off + (K - slab_of(w, own, blocks).k0 + 1) * w.sz + (j >> 1) * w.sy + (i >> 1);
    const float e = own == (int)cl.block_rank() ? *wx : *cl.map_shared_rank(wx, own);
    it.store(v, x, it.c[m], x[it.c[m]] + e);
    if (!((it.half >> m) & 1)) it.store(v, x, it.c[m] + 1, x[it.c[m] + 1] + e);
  }
}

__global__ void __launch_bounds__(kCoarseThreads) k_mg_coarse(const __grid_constant__ CoarseArgs A, const MgState* st) {
  if (stopped(st)) return;  // the same in every block
  extern __shared__ __align__(16) float sm[];
  const cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, rank = (int)cl.block_rank(), blocks = (int)cl.num_blocks();
  for (int t = tid; t < A.floats >> 2; t += kCoarseThreads)
    reinterpret_cast<float4*>(sm)[t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();
  // the operators of this block's planes (and the low faces of the plane above a
  // slab), all levels in one range of indices, so that their reads overlap
  {
    int q = 0, base = 0, plane = A.l[0].nx * A.l[0].ny;
    Slab z = slab_of(A.l[0], rank, blocks);
    auto count = [&]() { return z.n ? plane * (z.n + (z.k0 + z.n < A.l[q].nz ? 1 : 0)) : 0; };
#pragma unroll 1
    for (int t = tid;; t += kCoarseThreads) {
      while (t - base >= count()) {
        base += count();
        if (++q == A.levels) break;
        plane = A.l[q].nx * A.l[q].ny;
        z = slab_of(A.l[q], rank, blocks);
      }
      if (q == A.levels) break;
      const CoarseLev& v = A.l[q];
      float* x = sm + v.off;
      const int k = (t - base) / plane, rest = (t - base) - k * plane, j = rest / v.nx, i = rest - j * v.nx;
      const int c = (k + 1) * v.sz + j * v.sy + i;
      const int64_t g = v.L.at(i, j, z.k0 + k);
      const float zm = v.gz[g];
      if (k == z.n) {
        x[v.az + c] = zm;
        continue;
      }
      // the low faces, then 1/d (the high walls' couplings are ghosts, 0)
      const float xm = v.gx[g], ym = v.gy[g];
      const float d = ((xm + v.gx[g + 1]) + (ym + v.gy[g + v.L.px])) + (zm + v.gz[g + v.L.slab]);
      const float rhs = q == 0 ? A.b[(i + j + z.k0 + k) & 1][A.H.at(i >> 1, j, z.k0 + k)] : 0.0f;
      x[v.d + c] = d > 0.0f ? 1.0f / d : 0.0f;
      x[v.ax + c] = xm;
      x[v.ay + c] = ym;
      x[v.az + c] = zm;
      if (q == 0) x[v.b + c] = rhs;
    }
  }
  if (blocks > 1) cl.sync();
  else __syncthreads();
  int first = 0;  // the first level that is not split
#pragma unroll 1
  for (; first < A.levels && A.l[first].split; ++first) {
    const CoarseLev& v = A.l[first];
    const Slab z = slab_of(v, rank, blocks);
    CoarseItems<kCoarseItems> it;
    it.init(v, z, tid, kCoarseThreads);
    it.neighbours(v, z, sm + v.off, blocks, cl);
#pragma unroll 1
    for (int m = 0; m < kCoarseSweeps; ++m) {
      it.sweep(v, sm + v.off, m & 1);
      cl.sync();
    }
    coarse_restrict(v, A.l[first + 1], z, sm, blocks, cl, tid, kCoarseThreads);
    cl.sync();
  }
  if (rank == 0) {
    // by the block, the last ones by one warp
    int big = first;
    while (big < A.levels && coarse_slots(A.l[big].nx, A.l[big].ny, A.l[big].nz) > kWarpCells) ++big;
#pragma unroll 1
    for (int q = first; q < big; ++q) {
      const CoarseLev& v = A.l[q];
      const Slab z{0, v.nz};
      CoarseItems<1> it;
      it.init(v, z, tid, kCoarseThreads);
#pragma unroll 1
      for (int m = 0; m < kCoarseSweeps; ++m) {
        it.sweep(v, sm + v.off, m & 1);
        __syncthreads();
      }
      if (q + 1 < A.levels) {
        coarse_restrict(v, A.l[q + 1], z, sm, 1, cl, tid, kCoarseThreads);
        __syncthreads();
      }
    }
    if (tid < 32) {
#pragma unroll 1
      for (int q = big; q < A.levels; ++q) {
        const CoarseLev& v = A.l[q];
        const Slab z{0, v.nz};
        CoarseItems<1> it;
        it.init(v, z, tid, 32);
        // the coarsest level (at most 2 cells a side) is swept to a solve
        const int sweeps = q == A.levels - 1 ? 2 * kCoarseSweeps : kCoarseSweeps;
#pragma unroll 1
        for (int m = 0; m < sweeps; ++m) {
          it.sweep(v, sm + v.off, m & 1);
          __syncwarp();
        }
        if (q + 1 < A.levels) coarse_restrict(v, A.l[q + 1], z, sm, 1, cl, tid, 32);
        __syncwarp();
      }
#pragma unroll 1
      for (int q = A.levels - 1; q >= big; --q) {
        const CoarseLev& v = A.l[q];
        const Slab z{0, v.nz};
        CoarseItems<1> it;
        it.init(v, z, tid, 32);
        if (q + 1 < A.levels) coarse_prolong(v, A.l[q + 1], z, it, sm, 1, cl);
        __syncwarp();
        const int sweeps = q == A.levels - 1 ? 2 * kCoarseSweeps : kCoarseSweeps;
#pragma unroll 1
        for (int m = sweeps - 1; m >= 0; --m) {
          it.sweep(v, sm + v.off, m & 1);
          __syncwarp();
        }
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int q = big - 1; q >= first; --q) {
      const CoarseLev& v = A.l[q];
      const Slab z{0, v.nz};
      CoarseItems<1> it;
      it.init(v, z, tid, kCoarseThreads);
      if (q + 1 < A.levels) {
        coarse_prolong(v, A.l[q + 1], z, it, sm, 1, cl);
        __syncthreads();
      }
#pragma unroll 1
      for (int m = kCoarseSweeps - 1; m >= 0; --m) {
        it.sweep(v, sm + v.off, m & 1);
        __syncthreads();
      }
    }
  }
  if (first > 0) cl.sync();
#pragma unroll 1
  for (int q = first - 1; q >= 0; --q) {
    const CoarseLev& v = A.l[q];
    const Slab z = slab_of(v, rank, blocks);
    CoarseItems<kCoarseItems> it;
    it.init(v, z, tid, kCoarseThreads);
    it.neighbours(v, z, sm + v.off, blocks, cl);
    coarse_prolong(v, A.l[q + 1], z, it, sm, blocks, cl);
    cl.sync();
#pragma unroll 1
    for (int m = kCoarseSweeps - 1; m >= 0; --m) {
      it.sweep(v, sm + v.off, m & 1);
      cl.sync();  // (the last one: no block leaves while another writes into it)
    }
  }
  {
    const CoarseLev& v = A.l[0];
    const Slab z = slab_of(v, rank, blocks);
    const float* x = sm + v.off;
    const int plane = v.nx * v.ny;
    for (int t = tid; t < plane * z.n; t += kCoarseThreads) {
      const int k = t / plane, rest = t - k * plane, j = rest / v.nx, i = rest - j * v.nx;
      A.x[(i + j + z.k0 + k) & 1][A.H.at(i >> 1, j, z.k0 + k)] = x[(k + 1) * v.sz + j * v.sy + i];
    }
  }
}

// ---------------------------------------------------------------------------
// Operator set-up
// ---------------------------------------------------------------------------

// Couplings of the low faces of each cell (FP64 from phi, stored FP32; the
// expression of the projection's coupling kernel) and the cell's class.
template <class T>
__global__ void __launch_bounds__(kThreads) k_mg_build(const MgState* st, Lay L, Lay H, double rn, double rp,
                                                       double inv2, float* __restrict__ ax, float* __restrict__ ay,
                                                       float* __restrict__ az, unsigned char* __restrict__ cls0,
                                                       unsigned char* __restrict__ cls1,
                                                       unsigned char* __restrict__ ccls, double* extra0, int w,
                                                       int chunk) {
  const Column col(w, L.ny, L.nz, chunk);
  if (!col.ok) return;
  const int i = col.i, j = col.j, k0 = col.k0, k1 = col.k1;
  const T* __restrict__ phi = (const T*)st->phi;
  const double vneg = 1.0 / rn, vpos = 1.0 / rp;
  if (i == 0 && j == 0 && k0 == 0) *extra0 = 0.0;  // no deflation
  // the face between a cell and its low neighbour
  auto beta = [&](T low, T c) -> double {
    const bool nl = low <= T(0), nc = c <= T(0);
    if (nl == nc && low == low && c == c) return nc ? vneg : vpos;  // (a NaN goes on into the coupling)
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
    const bool same = p == p && (xm <= T(0)) == n && (xp <= T(0)) == n && (ym <= T(0)) == n && (yp <= T(0)) == n &&
                      (down <= T(0)) == n && (up <= T(0)) == n;
    const unsigned char cl = same ? (n ? 1 : 2) : 0;
    (((i + j + k) & 1) ? cls1 : cls0)[H.at(i >> 1, j, k)] = cl;
    ccls[c] = cl;
    down = p;
    p = up;
  }
}

// coarse couplings: half the sum of the fine couplings across the face
__global__ void __launch_bounds__(kThreads) k_mg_coarsen(Lay Lf, const float* __restrict__ fx,
                                                         const float* __restrict__ fy, const float* __restrict__ fz,
                                                         Lay L, float* __restrict__ ax, float* __restrict__ ay,
                                                         float* __restrict__ az) {
  const Column col(L.nx, L.ny, L.nz, 1);
  if (!col.ok) return;
  const int I = col.i, J = col.j, K = col.k0;
  // cells past an odd extent are ghosts, whose couplings are zero
  const int64_t c = L.at(I, J, K), f = Lf.at(2 * I, 2 * J, 2 * K);
  ax[c] = 0.5f * ((fx[f] + fx[f + Lf.px]) + (fx[f + Lf.slab] + fx[f + Lf.slab + Lf.px]));
  ay[c] = 0.5f * ((fy[f] + fy[f + 1]) + (fy[f + Lf.slab] + fy[f + Lf.slab + 1]));
  az[c] = 0.5f * ((fz[f] + fz[f + 1]) + (fz[f + Lf.px] + fz[f + Lf.px + 1]));
}

// classes of a coarse level: every face inside the box carries the same
// phase's uniform coupling
__global__ void __launch_bounds__(kThreads) k_mg_class(Lev v, unsigned char* __restrict__ cls0,
                                                       unsigned char* __restrict__ cls1) {
  const Lay& L = v.L;
  const Column col(L.nx, L.ny, L.nz, 1);
  if (!col.ok) return;
  const int i = col.i, j = col.j, k = col.k0;
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
// The iteration on the finest level.  x, p and q are in the cell layout; four
// cells i0 .. i0+3 per thread (slots i0/2, i0/2 + 1 of each colour; cell i0 +
// m is red when (m + j + k) is even), two in the FP64 residual.
// ---------------------------------------------------------------------------

// r, z or the red iterate of four cells from / to the packed colours.
__device__ __forceinline__ F4 unpack4(const float* const a[2], int64_t s, int par) {
  const float2 e = *reinterpret_cast<const float2*>(a[par] + s), o = *reinterpret_cast<const float2*>(a[1 - par] + s);
  return {{e.x, o.x, e.y, o.y}};
}

// q = A p in flux form (FP32 arithmetic, each flux exact to 2 eps32 of
// itself), p.q and alpha = r.z / p.q.
__global__ void __launch_bounds__(kThreads) k_mg_spmv(Lev v, const float* __restrict__ p, float* __restrict__ q,
                                                      MgState* st, double* partials, int w, int chunk) {
  if (stopped(st)) return;
  const Lay& L = v.L;
  const Column col(w, L.ny, L.nz, chunk);
  double pq = 0.0;
  if (col.ok) {
    const int i0 = 4 * col.i, j = col.j;
    const int valid = min(4, L.nx - i0);
    int64_t c = L.at(i0, j, col.k0);
    F4 dn = load4(p + c - L.slab), pc = load4(p + c);
    for (int k = col.k0; k < col.k1; ++k, c += L.slab) {
      const F4 up = load4(p + c + L.slab), ym = load4(p + c - L.px), yp = load4(p + c + L.px);
      const float xl = p[c - 1], xr = p[c + 4];
      const unsigned cl = *reinterpret_cast<const unsigned*>(v.ccls + c);
      const bool b0 = j > 0, b1 = j < L.ny - 1, d0 = k > 0, d1 = k < L.nz - 1;
      F4 out;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        out.v[m] = 0.0f;
        if (m >= valid) continue;
        const int cm = (cl >> (8 * m)) & 255u;
        const float pm = pc.v[m], l = m ? pc.v[m - 1] : xl, r = m < 3 ? pc.v[m + 1] : xr;
        if (cm) {
          // a face on a wall carries no flux
          float f = (i0 + m > 0 ? pm - l : 0.0f) + (i0 + m < L.nx - 1 ? pm - r : 0.0f);
          f += (b0 ? pm - ym.v[m] : 0.0f) + (b1 ? pm - yp.v[m] : 0.0f);
          f += (d0 ? pm - dn.v[m] : 0.0f) + (d1 ? pm - up.v[m] : 0.0f);
          out.v[m] = v.a[cm] * f;
        } else {
          const Couplings a = couplings_at(v, c + m);
          float f = a.xm * (pm - l) + a.xp * (pm - r);
          f += a.ym * (pm - ym.v[m]) + a.yp * (pm - yp.v[m]);
          f += a.zm * (pm - dn.v[m]) + a.zp * (pm - up.v[m]);
          out.v[m] = f;
        }
        pq += (double)pm * (double)out.v[m];
      }
      store4(q + c, out);  // (0 in ghosts past the row's end)
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
// last true one, has not for kCheckEvery iterations (at the floor of the
// arithmetic, where x only drifts), or the iteration cap is reached.
//
// x is kept in st->bak before it leaves the place of the smallest true residual
// so far (st->save, set by k_mg_defect): a solve that ends elsewhere goes back
// there.  x is read here anyway, so a save costs 8 bytes per cell: 43 instead of 35
// in the iterations that follow a true residual (a 256^3 timestep 41.33 -> 41.42
// ms, a projection of 150 x 210 x 131 cells 4.96 ms with and without).
constexpr int kCheckEvery = 8;
__global__ void __launch_bounds__(kThreads) k_mg_update(Lev v, const float* __restrict__ p,
                                                        const float* __restrict__ q, MgState* st, double* partials,
                                                        int w, int chunk) {
  if (stopped(st)) return;
  const Lay &L = v.L, &H = v.H;
  const Column col(w, L.ny, L.nz, chunk);
  const double alpha = state_read(&st->alpha);
  const float al = (float)alpha;
  const bool save = state_read(&st->save) != 0;
  double* __restrict__ x = st->x;
  double* __restrict__ bak = st->bak;
  float* __restrict__ rr_ = v.b[0];
  float* __restrict__ rb_ = v.b[1];
  float* __restrict__ xr_ = v.x[0];
  double rr = 0.0;
  if (col.ok) {
    const int i0 = 4 * col.i, j = col.j;
    const int valid = min(4, L.nx - i0);
    int64_t c = L.at(i0, j, col.k0), s = H.at(i0 >> 1, j, col.k0);
    for (int k = col.k0; k < col.k1; ++k, c += L.slab, s += H.slab) {
      const int par = (j + k) & 1;
      const F4 pv = load4(p + c), qv = load4(q + c);
      double2 x0 = *reinterpret_cast<const double2*>(x + c), x1 = *reinterpret_cast<const double2*>(x + c + 2);
      const float2 red = *reinterpret_cast<const float2*>(rr_ + s), black = *reinterpret_cast<const float2*>(rb_ + s);
      const unsigned cl = *reinterpret_cast<const unsigned*>(v.ccls + c);
      if (save) {  // (ghosts past the row's end: 0 in both)
        *reinterpret_cast<double2*>(bak + c) = x0;
        *reinterpret_cast<double2*>(bak + c + 2) = x1;
      }
      x0.x += alpha * (double)pv.v[0];
      x0.y += alpha * (double)pv.v[1];
      x1.x += alpha * (double)pv.v[2];
      x1.y += alpha * (double)pv.v[3];
      if (valid == 4) {
        *reinterpret_cast<double2*>(x + c) = x0;
        *reinterpret_cast<double2*>(x + c + 2) = x1;
      } else {
        x[c] = x0.x;
        if (valid > 1) x[c + 1] = x0.y;
        if (valid > 2) x[c + 2] = x1.x;
      }
      // past the row's end q and r are 0
      float2 nr, nb;  // red: cells par and par + 2
      nr.x = red.x - al * (par ? qv.v[1] : qv.v[0]);
      nr.y = red.y - al * (par ? qv.v[3] : qv.v[2]);
      nb.x = black.x - al * (par ? qv.v[0] : qv.v[1]);
      nb.y = black.y - al * (par ? qv.v[2] : qv.v[3]);
      *reinterpret_cast<float2*>(rr_ + s) = nr;
      *reinterpret_cast<float2*>(rb_ + s) = nb;
      rr += ((double)nr.x * (double)nr.x + (double)nr.y * (double)nr.y) +
            ((double)nb.x * (double)nb.x + (double)nb.y * (double)nb.y);
      float2 xr = make_float2(0.0f, 0.0f);
      if (par < valid) xr.x = first_sweep(v, (cl >> (8 * par)) & 255u, nr.x, i0 + par, j, k);
      if (par + 2 < valid) xr.y = first_sweep(v, (cl >> (8 * par + 16)) & 255u, nr.y, i0 + par + 2, j, k);
      *reinterpret_cast<float2*>(xr_ + s) = xr;
    }
  }
  rr = block_sum(rr);
  double tot;
  if (grid_reduce_sum(rr, partials, &st->ticket, &tot)) {
    st->rr = tot;
    st->iter += 1;
    st->save = 0;
    if (!isfinite(tot)) {
      st->status = PCG_STAGNATED;  // the FP32 recursion broke down; x may hold the bad step (the caller goes back)
      st->done = 1;
    } else if (tot <= st->tol2 || tot < st->delta * st->delta * st->max_rr || st->iter >= st->max_iter ||
               st->iter - st->checked >= kCheckEvery) {
      st->pause = 1;
    }
  }
}

// Flux sum of a cell near the interface, its face coefficients from phi in
// FP64; d holds x_c - x_nb per face (l, r, b, t, d, u), 0 on walls.
template <class T>
__device__ __noinline__ double mixed_flux(const T* phi, const Lay& L, int64_t c, int i, int j, int k, double vneg,
                                          double vpos, double dl, double dr, double db, double dt, double dd,
                                          double du) {
  const double pc = (double)phi[c];
  double flux = 0.0;
  if (i > 0) flux += face_coef(pc, (double)phi[c - 1], vneg, vpos) * dl;
  if (i < L.nx - 1) flux += face_coef(pc, (double)phi[c + 1], vneg, vpos) * dr;
  if (j > 0) flux += face_coef(pc, (double)phi[c - L.px], vneg, vpos) * db;
  if (j < L.ny - 1) flux += face_coef(pc, (double)phi[c + L.px], vneg, vpos) * dt;
  if (k > 0) flux += face_coef(pc, (double)phi[c - L.slab], vneg, vpos) * dd;
  if (k < L.nz - 1) flux += face_coef(pc, (double)phi[c + L.slab], vneg, vpos) * du;
  return flux;
}

// Whether the solve's loop goes on: bounded by the iteration cap whatever the
// state says.  Called by one thread after each iteration.
__device__ __forceinline__ void loop_next(MgState* st, cudaGraphConditionalHandle handle, bool stop) {
  const unsigned int n = st->batches + 1u;
  st->batches = n;
  cudaGraphSetConditional(handle, !stop && n < (unsigned int)st->max_iter + 2u ? 1u : 0u);
}

// The true residual r = b - A x in FP64 (A from phi in FP64), its norm, the
// first red half sweep, and the decisions that rest on it.  INIT: the start
// of a solve (unconditional; also keeps the initial guess in st->bak).  Else the
// last kernel of an iteration: with `loop` it also continues the graph's loop.
template <class T, bool INIT>
__global__ void __launch_bounds__(kThreads, 3) k_mg_defect(Lev v, MgState* st, double* partials, double rn, double rp,
                                                           double inv2, int w, int chunk, int loop,
                                                           cudaGraphConditionalHandle handle) {
  if (!INIT) {
    const bool stop = stopped(st);
    if (stop || !state_read(&st->pause)) {
      if (loop && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) loop_next(st, handle, stop);
      return;
    }
  }
  const Lay &L = v.L, &H = v.H;
  const Column col(w, H.ny, H.nz, chunk);
  const T* __restrict__ phi = (const T*)st->phi;
  const double* __restrict__ x = st->x;
  const double* __restrict__ b = st->b;
  const double vneg = 1.0 / rn, vpos = 1.0 / rp;
  double rr = 0.0;
  if (col.ok) {
    const int h = col.i, i0 = 2 * h, j = col.j;
    const bool two = i0 + 1 < L.nx;
    int64_t c = L.at(i0, j, col.k0), s = H.at(h, j, col.k0);
    auto ld2 = [&](const double* a, int64_t o) { return *reinterpret_cast<const double2*>(a + o); };
    double2 dn = ld2(x, c - L.slab), xc = ld2(x, c);
    const bool okl = i0 > 0, okr = i0 + 2 < L.nx, okb = j > 0, okt = j < L.ny - 1;
    for (int k = col.k0; k < col.k1; ++k, c += L.slab, s += H.slab) {
      const double2 up = ld2(x, c + L.slab), ym = ld2(x, c - L.px), yp = ld2(x, c + L.px);
      const double xl = x[c - 1], xr = x[c + 2];
      const double2 bv = ld2(b, c);
      const uchar2 cl = *reinterpret_cast<const uchar2*>(v.ccls + c);
      const int par = (j + k) & 1;
      const bool okd = k > 0, oku = k < L.nz - 1;
      if (INIT) {
        if (two) *reinterpret_cast<double2*>(st->bak + c) = xc;
        else st->bak[c] = xc.x;
      }
      const double dx = two ? xc.x - xc.y : 0.0;  // across the pair
      double f0, f1;
      {
        const double dl = okl ? xc.x - xl : 0.0, db = okb ? xc.x - ym.x : 0.0, dt = okt ? xc.x - yp.x : 0.0,
                     dd = okd ? xc.x - dn.x : 0.0, du = oku ? xc.x - up.x : 0.0;
        if (cl.x) f0 = (cl.x == 1 ? vneg : vpos) * (((dl + dx) + (db + dt)) + (dd + du));
        else f0 = mixed_flux<T>(phi, L, c, i0, j, k, vneg, vpos, dl, dx, db, dt, dd, du);
      }
      const double r0 = bv.x - inv2 * f0;
      rr += r0 * r0;
      const float a0 = (float)r0;
      v.b[par][s] = a0;
      if (par == 0) v.x[0][s] = first_sweep(v, cl.x, a0, i0, j, k);
      if (two) {
        const double dr = okr ? xc.y - xr : 0.0, db = okb ? xc.y - ym.y : 0.0, dt = okt ? xc.y - yp.y : 0.0,
                     dd = okd ? xc.y - dn.y : 0.0, du = oku ? xc.y - up.y : 0.0;
        if (cl.y) f1 = (cl.y == 1 ? vneg : vpos) * (((dr - dx) + (db + dt)) + (dd + du));
        else f1 = mixed_flux<T>(phi, L, c + 1, i0 + 1, j, k, vneg, vpos, -dx, dr, db, dt, dd, du);
        const double r1 = bv.y - inv2 * f1;
        rr += r1 * r1;
        const float a1 = (float)r1;
        v.b[1 - par][s] = a1;
        if (par == 1) v.x[0][s] = first_sweep(v, cl.y, a1, i0 + 1, j, k);
      } else {
        // the slot past an odd row's end has no cell: the red-black solve, which
        // shares these vectors, may have kept a value of its own in it
        v.b[1 - par][s] = 0.0f;
        if (par == 1) v.x[0][s] = 0.0f;
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
      st->save = 0;  // kept above
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
    st->checked = st->iter;
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
      if (tot < 0.9 * st->best) st->flat = 0;
      else st->flat += 1;
      if (tot > 1.0e4 * st->best || st->stall >= 24 || st->flat >= 4) {
        st->status = PCG_STAGNATED;  // diverged, or no further progress
        st->done = 1;
      }
    }
    if (!INIT && tot < st->best) {
      st->best = tot;
      st->save = 1;
    }
    if (!INIT && loop) loop_next(st, handle, st->done != 0);
  }
}

// p = z + beta p
__global__ void __launch_bounds__(kThreads) k_mg_direction(Lev v, float* __restrict__ p, const MgState* st, int w,
                                                           int chunk) {
  if (stopped(st)) return;
  const Lay &L = v.L, &H = v.H;
  const Column col(w, L.ny, L.nz, chunk);
  if (!col.ok) return;
  const float beta = (float)state_read(&st->beta);
  const int i0 = 4 * col.i, j = col.j;
  int64_t c = L.at(i0, j, col.k0), s = H.at(i0 >> 1, j, col.k0);
  const float* const z[2] = {v.x[0], v.x[1]};
  for (int k = col.k0; k < col.k1; ++k, c += L.slab, s += H.slab) {
    F4 pv = unpack4(z, s, (j + k) & 1);  // (0 past the row's end)
    if (beta != 0.0f) {  // a restart does not read the old direction
      const F4 po = load4(p + c);
#pragma unroll
      for (int m = 0; m < 4; ++m) pv.v[m] += beta * po.v[m];
    }
    store4(p + c, pv);
  }
}

// The pressure's constant.  The system is singular: CG moves the iterate in
// the range of its preconditioner, which fixes the constant of the result.
// The red-black solve conserves sum(x / dinv) over the black cells (z = dinv
// r and sum(r) = 0); the same sum is restored here, so that both solves give
// one pressure.
// Sums over the black cells: sum(x / dinv) and sum(1 / dinv), dinv the bf16
// 1/diag(S) of the red-black solve (fs_redblack.cu).
__global__ void __launch_bounds__(kThreads) k_mg_anchor(Lay L, Lay H, const unsigned short* __restrict__ dinv,
                                                        MgState* st, double* partials, int after, int w, int chunk) {
  if (after && state_read(&st->status) == PCG_STAGNATED) return;
  const double* __restrict__ x = st->x;
  const Column col(w, H.ny, H.nz, chunk);
  double sx = 0.0, sw = 0.0;
  if (col.ok) {
    const int h = col.i, j = col.j;
    int64_t s = H.at(h, j, col.k0);
    for (int k = col.k0; k < col.k1; ++k, s += H.slab) {
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
  double a = 0.0, ws = 0.0;
  for (int t = threadIdx.x; t < nb; t += kThreads) {
    a += __ldcg(partials + t);
    ws += __ldcg(partials + nb + t);
  }
  a = block_sum(a);
  __syncthreads();
  ws = block_sum(ws);
  if (thread0()) {
    if (after) st->shift = ws > 0.0 ? (st->anchor - a) / ws : 0.0;
    else st->anchor = a;
    st->ticket = 0u;
  }
}

__global__ void __launch_bounds__(kThreads) k_mg_shift(Lay L, const MgState* st, int w, int chunk) {
  const double d = st->shift;
  if (st->status == PCG_STAGNATED || d == 0.0) return;
  const Column col(w, L.ny, L.nz, chunk);
  if (!col.ok) return;
  double* __restrict__ x = st->x;
  const bool two = 2 * col.i + 1 < L.nx;
  int64_t c = L.at(2 * col.i, col.j, col.k0);
  for (int k = col.k0; k < col.k1; ++k, c += L.slab) {
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

constexpr size_t kCoarseBytes = 224 * 1024;  // of the 227 KB a block may have
// blocks of a cluster that k_mg_coarse may have (mg_prepare)
std::atomic<int> cluster_blocks{1};

cudaLaunchConfig_t coarse_launch(int blocks, size_t bytes, cudaLaunchAttribute* at, cudaStream_t s) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = blocks;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(blocks);
  c.blockDim = dim3(kCoarseThreads);
  c.dynamicSmemBytes = bytes;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 1;
  return c;
}

bool coarse_split(int nx, int ny, int nz, int blocks) { return blocks > 1 && coarse_slots(nx, ny, nz) > kSplitSlots; }
// shared floats of one level in one block, rounded up to a float4
size_t coarse_floats(int nx, int ny, int nz, int blocks) {
  const size_t p = coarse_split(nx, ny, nz, blocks) ? (nz + blocks - 1) / blocks : nz;
  return ((6 * p + 3) * (size_t)(nx + 1) * (ny + 1) + 3) / 4 * 4;
}

}  // namespace

// The grids of the hierarchy: halved (rounding up) until at most 2 cells a
// side; `top` is the first level from which on all fit a cluster of *cluster blocks.
int mg_plan(int nx, int ny, int nz, int ext[kMgMaxLevels][3], int* top, int* cluster) {
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
  const int blocks = *cluster = cluster_blocks;
  size_t floats = 0;
  int t = n;
  while (t > 1) {
    const int *e = ext[t - 1], planes = coarse_split(e[0], e[1], e[2], blocks) ? (e[2] + blocks - 1) / blocks : e[2];
    floats += coarse_floats(e[0], e[1], e[2], blocks);
    if (floats * sizeof(float) > kCoarseBytes || coarse_slots(e[0], e[1], planes) > (planes < e[2] ? kCoarseItems : 1) * kCoarseThreads)
      break;
    --t;
  }
  *top = t;
  return n;
}

// The largest cluster that the device runs: 16 blocks (of one GPC; more than the
// portable 8), else 8, else one block.
cudaError_t mg_prepare() {
  const cudaError_t e =
      cudaFuncSetAttribute(k_mg_coarse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseBytes);
  if (e != cudaSuccess) return e;
  for (int blocks : {16, 8, 1}) {
    if (blocks > 8 && cudaFuncSetAttribute(k_mg_coarse, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = coarse_launch(blocks, kCoarseBytes, &at, 0);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_mg_coarse, &cfg) == cudaSuccess && n > 0) {
      cluster_blocks = blocks;
      break;
    }
    cudaGetLastError();
  }
  return cudaSuccess;
}

int mg_max_blocks(const Lay& L) {
  int64_t most = 0;
  for (int per : {1, 2, 4}) {
    const Columns c = columns(L.nx, L.ny, L.nz, per);
    most = std::max(most, (int64_t)c.grid.x * c.grid.y);
  }
  return (int)most;
}

template <class T>
int mg_build(const Multigrid& M, const MgState* st, double dx, double rho_neg, double rho_pos, double* extra0,
             cudaStream_t s) {
  const MgLevel& f = M.level[0];
  const Columns g = columns(f.L.nx, f.L.ny, f.L.nz, 1);
  k_mg_build<T><<<g.grid, kThreads, 0, s>>>(st, f.L, f.H, rho_neg, rho_pos, 1.0 / (dx * dx), f.ax, f.ay, f.az,
                                            f.cls[0], f.cls[1], f.ccls, extra0, g.w, g.chunk);
  int launches = 1;
  for (int l = 1; l < M.levels; ++l) {
    const MgLevel &a = M.level[l - 1], &b = M.level[l];
    const dim3 grid((unsigned)(((int64_t)b.L.nx * b.L.ny + kThreads - 1) / kThreads), (unsigned)b.L.nz, 1);
    k_mg_coarsen<<<grid, kThreads, 0, s>>>(a.L, a.ax, a.ay, a.az, b.L, b.ax, b.ay, b.az);
    ++launches;
    if (l < M.top) {
      k_mg_class<<<grid, kThreads, 0, s>>>(lev_of(b), b.cls[0], b.cls[1]);
      ++launches;
    }
  }
  return launches;
}

namespace {

// slots of one colour per thread of a level's sweeps and restriction
int wide(const MgLevel& m) {
  const Columns g = columns(m.H.nx, m.H.ny, m.H.nz, 4);
  return (int64_t)g.grid.x * g.grid.y < 3 * 148 ? 1 : 4;
}
template <bool CORRECT, int DOT>
void sweep(const MgLevel& m, const MgLevel& coarse, int color, MgState* st, double* partials, cudaStream_t s) {
  const int w = wide(m);
  const Columns g = columns(m.H.nx, m.H.ny, m.H.nz, w);
  auto* kernel = w == 4 ? k_mg_sweep<4, CORRECT, DOT> : k_mg_sweep<1, CORRECT, DOT>;
  kernel<<<g.grid, kThreads, 0, s>>>(lev_of(m), lev_of(coarse), color, st, partials, g.w, g.chunk);
}

// z = M r: the V-cycle on the residual in level 0's b (x's first red sweep
// done), and r.z with beta
int cycle(const Multigrid& M, MgState* st, double* partials, cudaStream_t s) {
  int launches = 0;
  for (int l = 0; l < M.top; ++l) {
    const MgLevel &m = M.level[l], &c = M.level[l + 1];
    sweep<false, 0>(m, c, 1, st, partials, s);
    sweep<false, 0>(m, c, 0, st, partials, s);
    const int w = wide(c);
    const Columns g = columns(c.L.nx, c.L.ny, c.L.nz, w);
    auto* restriction = w == 4 ? k_mg_restrict<4> : k_mg_restrict<1>;
    restriction<<<g.grid, kThreads, 0, s>>>(lev_of(m), lev_of(c), 1, st, g.w, g.chunk);
    launches += 3;
  }
  CoarseArgs A{};
  size_t floats = 0;
  A.levels = M.levels - M.top;
  const Lay& tl = M.level[M.top].L;
  const int blocks = coarse_split(tl.nx, tl.ny, tl.nz, M.blocks) ? M.blocks : 1;
  for (int q = 0; q < A.levels; ++q) {
    const MgLevel& m = M.level[M.top + q];
    CoarseLev& w = A.l[q];
    w.nx = m.L.nx;
    w.ny = m.L.ny;
    w.nz = m.L.nz;
    w.sy = w.nx + 1;
    w.sz = w.sy * (w.ny + 1);
    w.split = coarse_split(w.nx, w.ny, w.nz, blocks);
    const int p = w.split ? (w.nz + blocks - 1) / blocks : w.nz;
    w.off = (int)floats;
    w.b = (p + 1) * w.sz;
    w.d = w.b + p * w.sz;
    w.ax = w.d + p * w.sz;
    w.ay = w.ax + p * w.sz;
    w.az = w.ay + p * w.sz;
    w.gx = m.ax;
    w.gy = m.ay;
    w.gz = m.az;
    w.L = m.L;
    floats += coarse_floats(w.nx, w.ny, w.nz, blocks);
  }
  A.floats = (int)floats;
  const MgLevel& t = M.level[M.top];
  for (int c = 0; c < 2; ++c) {
    A.x[c] = t.x[c];
    A.b[c] = t.b[c];
  }
  A.H = t.H;
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = coarse_launch(blocks, floats * sizeof(float), &at, s);
  cudaLaunchKernelEx(&cfg, k_mg_coarse, A, (const MgState*)st);
  ++launches;
  for (int l = M.top - 1; l >= 0; --l) {
    const MgLevel &m = M.level[l], &c = M.level[l + 1];
    sweep<true, 0>(m, c, 0, st, partials, s);
    if (l == 0) {
      sweep<false, 1>(m, c, 1, st, partials, s);
      sweep<false, 2>(m, c, 0, st, partials, s);
    } else {
      sweep<false, 0>(m, c, 1, st, partials, s);
      sweep<false, 0>(m, c, 0, st, partials, s);
    }
    launches += 3;
  }
  return launches;
}

}  // namespace

template <class T>
int mg_start(const Multigrid& M, MgState* st, double* partials, double dx, double rho_neg, double rho_pos,
             cudaStream_t s) {
  const Lev v = lev_of(M.level[0]);
  const Columns g = columns(v.H.nx, v.H.ny, v.H.nz, 1);
  k_mg_defect<T, true><<<g.grid, kThreads, 0, s>>>(v, st, partials, rho_neg, rho_pos, 1.0 / (dx * dx), g.w, g.chunk, 0,
                                                   cudaGraphConditionalHandle{});
  return 1;
}

template <class T>
int mg_iteration(const Multigrid& M, float* p, float* q, MgState* st, double* partials, double dx, double rho_neg,
                 double rho_pos, bool loop, cudaGraphConditionalHandle handle, cudaStream_t s) {
  const Lev v = lev_of(M.level[0]);
  const Columns g = columns(v.L.nx, v.L.ny, v.L.nz, 4), gd = columns(v.H.nx, v.H.ny, v.H.nz, 1);
  const int n = cycle(M, st, partials, s);
  k_mg_direction<<<g.grid, kThreads, 0, s>>>(v, p, st, g.w, g.chunk);
  k_mg_spmv<<<g.grid, kThreads, 0, s>>>(v, p, q, st, partials, g.w, g.chunk);
  k_mg_update<<<g.grid, kThreads, 0, s>>>(v, p, q, st, partials, g.w, g.chunk);
  k_mg_defect<T, false><<<gd.grid, kThreads, 0, s>>>(v, st, partials, rho_neg, rho_pos, 1.0 / (dx * dx), gd.w,
                                                     gd.chunk, loop ? 1 : 0, handle);
  return n + 4;
}

void mg_anchor(const Multigrid& M, const unsigned short* dinv, MgState* st, double* partials, bool after,
               cudaStream_t s) {
  const MgLevel& f = M.level[0];
  const Columns g = columns(f.H.nx, f.H.ny, f.H.nz, 1);
  k_mg_anchor<<<g.grid, kThreads, 0, s>>>(f.L, f.H, dinv, st, partials, after ? 1 : 0, g.w, g.chunk);
  if (after) k_mg_shift<<<g.grid, kThreads, 0, s>>>(f.L, st, g.w, g.chunk);
}

__global__ void k_mg_loop_start(cudaGraphConditionalHandle handle, const MgState* st) {
  cudaGraphSetConditional(handle, stopped(st) ? 0u : 1u);
}
void mg_loop_start(cudaGraphConditionalHandle handle, const MgState* st, cudaStream_t s) {
  k_mg_loop_start<<<1, 1, 0, s>>>(handle, st);
}

template int mg_build<float>(const Multigrid&, const MgState*, double, double, double, double*, cudaStream_t);
template int mg_start<float>(const Multigrid&, MgState*, double*, double, double, double, cudaStream_t);
template int mg_iteration<float>(const Multigrid&, float*, float*, MgState*, double*, double, double, double, bool,
                                 cudaGraphConditionalHandle, cudaStream_t);

}  // namespace fsb
