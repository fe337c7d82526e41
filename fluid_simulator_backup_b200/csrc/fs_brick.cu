// The FP64 Jacobi-PCG of the pressure (PCG_METHOD.cpp:4-126) as one resident
// kernel, for grids whose vectors fit the GPU's shared memory and registers.
//
// What bounds it.  At 64^3 and 96^3 an iteration of three kernels (fs_krylov.cu)
// takes 20 to 31 us, nearly all of it launches, grid-wide reductions and cold
// starts: the vectors are a few MB.  Here one block per SM keeps a brick of the
// box: r and q in registers, p (with a one-cell halo) and x in shared memory.
// The couplings are not kept: away from the interface every face carries its
// phase's 1/rho, and a byte per cell says which (and which faces lie on a
// wall).  The cells next to the interface are a list of their own, worked off
// by all threads before the rest (inline, each of a thread's 24 cells would wait
// for its couplings in turn: 41 us per iteration at 96^3), with their couplings
// in shared memory as far as it reaches and in global memory beyond.
//
// One iteration exchanges twice: p.q, then r.z with r.r.  The sums are also
// the barrier, and every block adds them in the same order, so alpha, beta and
// the decisions are the same everywhere.  The halo of p follows from p = z + beta p with the neighbours' z, which they
// store before the second exchange; no third one is needed.  The blocks wait
// on one another, so the launch is cooperative; every wait has a limit, after
// which the solve ends with PCG_TIMEOUT.
//
// Measured (B200), per iteration, three kernels in a graph -> this one: 32^3
// 17.8 -> 6.2 us, 64^3 22.9 -> 7.9, 96^3 46.9 -> 16.7, 112^3 62.8 -> 35.8.  The
// two exchanges take 3.7 us of it; the rest is instruction issue and latency at
// 16 warps per SM (the registers hold r and q).
#include <algorithm>

#include "fs_kernels.h"

namespace fsb {

namespace {

constexpr int kT = 512;                    // threads of a block
constexpr int kMaxBlocks = 256;            // one poller per block
constexpr unsigned kSpin = 1u << 22;       // polls before a wait gives up (seconds)
constexpr size_t kSmem = 227 * 1024 - 2048;  // dynamic shared memory of a block (static: the reductions)

struct BrickArgs {
  Lay L;
  int gx, gy, gz;
  const double *ax, *ay, *az, *diag, *phi, *b, *extra0;
  double *x, *zx;
  double* sums;       // [2][2][kMaxBlocks]: turn, value, block
  unsigned* count;    // blocks that have stored their sums, over all turns
  int cap;            // mixed cells whose couplings fit in shared memory
  PcgState* st;
  double a[3];           // uniform coupling of a phase (1: phi <= 0, 2: phi > 0)
  int64_t c_extra;       // cell that carries extra0, -1: none
};

// Sums of two values over the grid, the same in every block (two: whether the
// second one is wanted), and a barrier: what a block stored before is visible
// after it (through L2) in every block.  Each block stores its partial sums
// and counts itself in; one thread per block waits for the count, then all
// read the sums and add them in the same order.  Measured with 144 blocks:
// 1.8 us, against 4.5 us where every block polls the 144 sums themselves (the
// polls queue in front of the stores they wait for).  `turn` counts the
// exchanges of the solve from 1.  Returns false when a wait ran out.
__device__ __forceinline__ bool exchange(const BrickArgs& A, int nb, unsigned turn, bool two, double& v0, double& v1) {
  __shared__ double part[2][kT / 32];
  __shared__ int bad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double w0 = warp_sum(v0), w1 = two ? warp_sum(v1) : 0.0;
  if (lane == 0) {
    part[0][warp] = w0;
    part[1][warp] = w1;
  }
  if (tid == 0) bad = 0;
  __syncthreads();
  double* sums = A.sums + (turn & 1u) * 2 * kMaxBlocks;  // the other half may still be read
  if (warp == 0) {
    const double s0 = warp_sum(lane < kT / 32 ? part[0][lane] : 0.0);
    const double s1 = two ? warp_sum(lane < kT / 32 ? part[1][lane] : 0.0) : 0.0;
    if (lane == 0) {
      __stcg(sums + blockIdx.x, s0);
      if (two) __stcg(sums + kMaxBlocks + blockIdx.x, s1);
      // release: cumulative over the block's stores (after the barrier above)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(A.count) : "memory");
      const unsigned want = turn * (unsigned)nb;
      unsigned got = 0, n = 0;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(A.count) : "memory");
        if ((int)(got - want) >= 0) break;
        if (++n >= kSpin) {
          bad = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
  // warps 0 .. 7 gather the first value, 8 .. 15 the second
  const int from = tid & 255, value = tid >> 8;
  double g = from < nb && (value == 0 || two) ? __ldcg(sums + value * kMaxBlocks + from) : 0.0;
  g = warp_sum(g);
  if (lane == 0) part[0][warp] = g;
  __syncthreads();
  v0 = v1 = 0.0;
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    v0 += part[0][m];
    v1 += part[0][8 + m];
  }
  const bool ok = bad == 0;
  __syncthreads();  // before the next exchange writes part[] and bad
  return ok;
}

__device__ __forceinline__ bool brick_stop(const PcgState& s, double rz, double rr, double bb) {
  switch (s.criterion) {
    case 1: return rz < s.tol * s.tol;
    case 2: return rr < s.tol * s.tol;
    default: return sqrt(rr) <= s.tol * sqrt(bb);
  }
}

// A mixed cell that the list has no room for.
__device__ __noinline__ double unlisted_apply(const BrickArgs& A, int64_t g, const double* c, int sy, int sz) {
  const double v = c[0];
  double acc = A.ax[g] * (v - c[-1]) + A.ax[g + 1] * (v - c[1]);
  acc += A.ay[g] * (v - c[-sy]) + A.ay[g + A.L.px] * (v - c[sy]);
  acc += A.az[g] * (v - c[-sz]) + A.az[g + A.L.slab] * (v - c[sz]);
  if (g == A.c_extra) acc += *A.extra0 * v;
  return acc;
}

// K: cells per thread.  XG: x stays in global memory (bricks too large for it).
template <int K, bool XG>
__global__ void __launch_bounds__(kT, 1) k_pcg_brick(const __grid_constant__ BrickArgs A) {
  extern __shared__ double smem[];
  const Lay& L = A.L;
  const int nb = gridDim.x, tid = threadIdx.x;
  const int qx = blockIdx.x % A.gx, qy = (blockIdx.x / A.gx) % A.gy, qz = blockIdx.x / (A.gx * A.gy);
  const int i0 = (int)((int64_t)qx * L.nx / A.gx), i1 = (int)((int64_t)(qx + 1) * L.nx / A.gx);
  const int j0 = (int)((int64_t)qy * L.ny / A.gy), j1 = (int)((int64_t)(qy + 1) * L.ny / A.gy);
  const int k0 = (int)((int64_t)qz * L.nz / A.gz), k1 = (int)((int64_t)(qz + 1) * L.nz / A.gz);
  const int bx = i1 - i0, by = j1 - j0, bz = k1 - k0, cells = bx * by * bz;
  const int sy = bx + 2, sz = sy * (by + 2), padded = sz * (bz + 2);
  const int halo = 2 * (by * bz + bx * bz + bx * by);
  double* p = smem;
  double* xs = p + padded;
  double* inv = xs + (XG ? 0 : cells);  // 1/(n a) of n faces: [phase][n]
  // the list of mixed cells: q, 1/diag, the six couplings
  double* mq = inv + 24;
  double* mdi = mq + A.cap;
  double* ma = mdi + A.cap;
  int* go = (int*)(ma + 6 * (size_t)A.cap);  // offset of each cell in global memory
  int* hp = go + cells;
  int* hg = hp + halo;
  unsigned short* mt = (unsigned short*)(hg + halo);  // the cell of a list entry
  unsigned short* mp = mt + A.cap;                    // its index in p
  unsigned short* me = mp + A.cap;                    // a mixed cell's entry (>= cap: not in the list)
  unsigned char* kind = (unsigned char*)(me + cells);
  __shared__ int mixed;
  if (tid == 0) mixed = 0;
  if (tid < 24) inv[tid] = tid % 8 && tid / 8 ? 1.0 / (A.a[tid / 8] * (double)(tid % 8)) : 0.0;
  __syncthreads();
  const PcgState par = *A.st;  // tol, criterion, max_iter

  // this thread's cells tid + m kT: index in p
  int pi[K];
  unsigned edge = 0u;  // bit m: on the brick's surface
  double r[K], q[K];
  const int64_t base = L.at(i0, j0, k0);
#pragma unroll
  for (int m = 0; m < K; ++m) {
    const int t = tid + m * kT;
    pi[m] = -1;
    if (t < cells) {
      const int lx = t % bx, row = t / bx, ly = row % by, lz = row / by;
      pi[m] = (lz + 1) * sz + (ly + 1) * sy + lx + 1;
      const int o = (int)(lx + (int64_t)ly * L.px + (int64_t)lz * L.slab);
      go[t] = o;
      if (lx == 0 || lx == bx - 1 || ly == 0 || ly == by - 1 || lz == 0 || lz == bz - 1) edge |= 1u << m;
      // bits 0..5: the face lies inside the box; 6, 7: the phase whose 1/rho
      // all faces carry (0: read the couplings)
      const int i = i0 + lx, j = j0 + ly, k = k0 + lz;
      const int f = (i > 0) | (i < L.nx - 1) << 1 | (j > 0) << 2 | (j < L.ny - 1) << 3 | (k > 0) << 4 |
                    (k < L.nz - 1) << 5;
      const double* ph = A.phi + base + o;
      const bool n = ph[0] <= 0.0;
      const bool same = ph[0] == ph[0] && (!(f & 1) || (ph[-1] <= 0.0) == n) && (!(f & 2) || (ph[1] <= 0.0) == n) &&
                        (!(f & 4) || (ph[-L.px] <= 0.0) == n) && (!(f & 8) || (ph[L.px] <= 0.0) == n) &&
                        (!(f & 16) || (ph[-L.slab] <= 0.0) == n) && (!(f & 32) || (ph[L.slab] <= 0.0) == n);
      const bool extra = base + o == A.c_extra;
      kind[t] = (unsigned char)(f | (same && !extra ? (n ? 64 : 128) : 0));
      if (!same || extra) {
        const int e = atomicAdd(&mixed, 1);
        const int64_t g = base + o;
        me[t] = (unsigned short)e;
        if (e < A.cap) {
          mt[e] = (unsigned short)t;
          mp[e] = (unsigned short)pi[m];
          mdi[e] = 1.0 / A.diag[g];
          ma[e] = A.ax[g];
          ma[A.cap + e] = A.ax[g + 1];
          ma[2 * A.cap + e] = A.ay[g];
          ma[3 * A.cap + e] = A.ay[g + L.px];
          ma[4 * A.cap + e] = A.az[g];
          ma[5 * A.cap + e] = A.az[g + L.slab];
        }
      }
    }
  }
  // the halo: index in p and offset in global memory of each cell inside the box
  const int fx = by * bz, fy = bx * bz, fz = bx * by;
  for (int h = tid; h < halo; h += kT) {
    int t = h, lx, ly, lz;
    if (t < 2 * fx) {
      lx = t < fx ? -1 : bx;
      t -= t < fx ? 0 : fx;
      ly = t % by;
      lz = t / by;
    } else if (t < 2 * (fx + fy)) {
      t -= 2 * fx;
      ly = t < fy ? -1 : by;
      t -= t < fy ? 0 : fy;
      lx = t % bx;
      lz = t / bx;
    } else {
      t -= 2 * (fx + fy);
      lz = t < fz ? -1 : bz;
      t -= t < fz ? 0 : fz;
      lx = t % bx;
      ly = t / bx;
    }
    const int i = i0 + lx, j = j0 + ly, k = k0 + lz;
    const bool in = i >= 0 && i < L.nx && j >= 0 && j < L.ny && k >= 0 && k < L.nz;
    hp[h] = in ? (lz + 1) * sz + (ly + 1) * sy + lx + 1 : -1;
    hg[h] = (int)(lx + (int64_t)ly * L.px + (int64_t)lz * L.slab);
  }

  // A p of the mixed cells into mq, in flux form.  A wall's coupling is zero
  // and its halo entry of p stays finite.
  auto apply_mixed = [&]() {
    const int n = min(mixed, A.cap);
    for (int e = tid; e < n; e += kT) {
      const double* c = p + mp[e];
      const double v = c[0];
      double acc = ma[e] * (v - c[-1]) + ma[A.cap + e] * (v - c[1]);
      acc += ma[2 * A.cap + e] * (v - c[-sy]) + ma[3 * A.cap + e] * (v - c[sy]);
      acc += ma[4 * A.cap + e] * (v - c[-sz]) + ma[5 * A.cap + e] * (v - c[sz]);
      if (base + go[mt[e]] == A.c_extra) acc += *A.extra0 * v;
      mq[e] = acc;
    }
    __syncthreads();
  };
  // (A p)_c of this thread's cell m, after apply_mixed
  auto apply = [&](int m) -> double {
    const double* c = p + pi[m];
    const int t = tid + m * kT, f = kind[t];
    if (!(f >> 6)) return me[t] < A.cap ? mq[me[t]] : unlisted_apply(A, base + go[t], c, sy, sz);
    const double v = c[0];
    if ((f & 63) == 63)
      return A.a[f >> 6] * ((((v - c[-1]) + (v - c[1])) + ((v - c[-sy]) + (v - c[sy]))) + ((v - c[-sz]) + (v - c[sz])));
    const double dl = f & 1 ? v - c[-1] : 0.0, dr = f & 2 ? v - c[1] : 0.0, db = f & 4 ? v - c[-sy] : 0.0,
                 dt = f & 8 ? v - c[sy] : 0.0, dd = f & 16 ? v - c[-sz] : 0.0, du = f & 32 ? v - c[sz] : 0.0;
    return A.a[f >> 6] * (((dl + dr) + (db + dt)) + (dd + du));
  };
  // p = z + beta p on the halo, with the neighbours' z; eight fetches in flight
  auto update_halo = [&](double beta) {
    constexpr int kFetch = 8;
    for (int h0 = tid; h0 < halo; h0 += kFetch * kT) {
      int at[kFetch];
      double z[kFetch];
#pragma unroll
      for (int m = 0; m < kFetch; ++m) {
        const int h = h0 + m * kT;
        at[m] = h < halo ? hp[h] : -1;
        z[m] = at[m] >= 0 ? __ldcg(A.zx + base + hg[h]) : 0.0;
      }
#pragma unroll
      for (int m = 0; m < kFetch; ++m)
        if (at[m] >= 0) p[at[m]] = z[m] + (beta != 0.0 ? beta * p[at[m]] : 0.0);
    }
  };
  // z = r / diag
  auto precondition = [&](int m, double v) -> double {
    const int t = tid + m * kT, f = kind[t];
    if (f >> 6) return v * inv[(f >> 6) * 8 + __popc(f & 63)];
    return me[t] < A.cap ? v * mdi[me[t]] : v / A.diag[base + go[t]];
  };

  // r = b - A x, p = z (halo entries beyond a wall: 0)
  unsigned turn = 0;
  for (int t = tid; t < padded; t += kT) p[t] = 0.0;
  __syncthreads();
#pragma unroll
  for (int m = 0; m < K; ++m)
    if (pi[m] >= 0) {
      const double v = A.x[base + go[tid + m * kT]];
      p[pi[m]] = v;
      if (!XG) xs[tid + m * kT] = v;
    }
  __syncthreads();
  for (int h = tid; h < halo; h += kT)
    if (hp[h] >= 0) p[hp[h]] = A.x[base + hg[h]];
  __syncthreads();
  apply_mixed();
  double rz = 0.0, rr = 0.0, bb = 0.0, zero = 0.0;
#pragma unroll
  for (int m = 0; m < K; ++m)
    if (pi[m] >= 0) {
      const double bv = A.b[base + go[tid + m * kT]];
      r[m] = bv - apply(m);
      const double z = precondition(m, r[m]);
      q[m] = z;
      if (edge >> m & 1u) A.zx[base + go[tid + m * kT]] = z;
      rz += r[m] * z;
      rr += r[m] * r[m];
      bb += bv * bv;
    }
  bool alive = exchange(A, nb, ++turn, true, rz, rr);
  alive = exchange(A, nb, ++turn, false, bb, zero) && alive;
  int iter = 0, status = PCG_RUNNING;
  if (!alive) status = PCG_TIMEOUT;
  else if (!isfinite(rz) || !isfinite(rr)) status = PCG_NONFINITE;
  else if (bb == 0.0 || rr == 0.0 || (par.criterion != 1 && brick_stop(par, rz, rr, bb))) status = PCG_CONVERGED;
  else if (par.max_iter <= 0) status = PCG_MAXITER;
  if (status == PCG_RUNNING) {
    __syncthreads();
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (pi[m] >= 0) p[pi[m]] = q[m];
    update_halo(0.0);
    __syncthreads();
  }
  // every block takes the same decisions from the same sums
  while (status == PCG_RUNNING) {
    apply_mixed();
    double pq = 0.0;
    zero = 0.0;
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (pi[m] >= 0) {
        q[m] = apply(m);
        pq += p[pi[m]] * q[m];
      }
    if (!exchange(A, nb, ++turn, false, pq, zero)) {
      status = PCG_TIMEOUT;
      break;
    }
    const double alpha = rz / pq;
    if (!(pq > 0.0) || !isfinite(alpha)) {
      status = PCG_STAGNATED;
      break;
    }
    double rz1 = 0.0, rr1 = 0.0;
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (pi[m] >= 0) {
        r[m] -= alpha * q[m];
        const double z = precondition(m, r[m]);
        q[m] = z;
        if (edge >> m & 1u) A.zx[base + go[tid + m * kT]] = z;
        rz1 += r[m] * z;
        rr1 += r[m] * r[m];
      }
    if (!exchange(A, nb, ++turn, true, rz1, rr1)) {
      status = PCG_TIMEOUT;
      break;
    }
    const double beta = rz1 / rz;
    rz = rz1;
    rr = rr1;
    if (!isfinite(rz) || !isfinite(rr)) {
      status = PCG_NONFINITE;  // x is not moved along that step
      break;
    }
    if (brick_stop(par, rz, rr, bb)) {
      status = PCG_CONVERGED;
    } else {
      ++iter;
      if (iter >= par.max_iter) status = PCG_MAXITER;
    }
    if (XG) {
      constexpr int kFetch = 5;  // x values in flight
#pragma unroll
      for (int m0 = 0; m0 < K; m0 += kFetch) {
        double xv[kFetch];
#pragma unroll
        for (int m = 0; m < kFetch; ++m)
          xv[m] = m0 + m < K && pi[m0 + m] >= 0 ? A.x[base + go[tid + (m0 + m) * kT]] : 0.0;
#pragma unroll
        for (int m = 0; m < kFetch; ++m)
          if (m0 + m < K && pi[m0 + m] >= 0) A.x[base + go[tid + (m0 + m) * kT]] = xv[m] + alpha * p[pi[m0 + m]];
      }
    }
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (pi[m] >= 0) {
        const double pv = p[pi[m]];
        if (!XG) xs[tid + m * kT] += alpha * pv;
        p[pi[m]] = q[m] + beta * pv;
      }
    update_halo(beta);
    __syncthreads();
  }
  if (!XG && iter + (status == PCG_CONVERGED) > 0) {
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (pi[m] >= 0) A.x[base + go[tid + m * kT]] = xs[tid + m * kT];
  }
  if (blockIdx.x == 0 && tid == 0) {
    A.st->rz = rz;
    A.st->rr = rr;
    A.st->bb = bb;
    A.st->iter = iter;
    A.st->status = status;
    A.st->done = 1;
  }
}

// shared memory of a brick without its list of mixed cells, and of one entry
size_t brick_bytes(int bx, int by, int bz, bool xg) {
  const size_t cells = (size_t)bx * by * bz, padded = (size_t)(bx + 2) * (by + 2) * (bz + 2);
  const size_t halo = 2 * ((size_t)by * bz + (size_t)bx * bz + (size_t)bx * by);
  return (padded + (xg ? 0 : cells) + 24) * 8 + (cells + 2 * halo) * 4 + cells * 2 + (cells + 7) / 8 * 8;
}
constexpr size_t kEntryBytes = 8 * 8 + 2 * 2;

template <int K, bool XG>
bool prepare(const BrickPlan& P, int* most) {
  if (cudaFuncSetAttribute(k_pcg_brick<K, XG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess)
    return false;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(most, k_pcg_brick<K, XG>, kT, P.smem) == cudaSuccess;
}

const void* kernel_of(const BrickPlan& P) {
  if (P.xg) return (const void*)k_pcg_brick<20, true>;
  switch (P.per_thread) {
    case 2: return (const void*)k_pcg_brick<2, false>;
    case 4: return (const void*)k_pcg_brick<4, false>;
    case 8: return (const void*)k_pcg_brick<8, false>;
    case 12: return (const void*)k_pcg_brick<12, false>;
    default: return (const void*)k_pcg_brick<16, false>;
  }
}

}  // namespace

// The division of the box into at most `sms` bricks: the smallest largest
// brick, counting a halo cell as a third of a cell and one on an x face (a
// strided access) as a whole one.
BrickPlan brick_plan(const Lay& L, int sms) {
  BrickPlan best;
  double least = 1e300;
  sms = std::min(sms, kMaxBlocks);
  for (int gz = 1; gz <= std::min(sms, L.nz); ++gz)
    for (int gy = 1; gy <= std::min(sms / gz, L.ny); ++gy)
      for (int gx = 1; gx <= std::min(sms / gz / gy, L.nx); ++gx) {
        const int bx = (L.nx + gx - 1) / gx, by = (L.ny + gy - 1) / gy, bz = (L.nz + gz - 1) / gz;
        const double cost = (double)bx * by * bz + 2.0 * by * bz * (gx > 1) +
                            (2.0 / 3.0) * ((double)bx * bz * (gy > 1) + (double)bx * by * (gz > 1));
        if (cost >= least) continue;
        const int64_t cells = (int64_t)bx * by * bz;
        BrickPlan P;
        if (cells <= 16 * kT && brick_bytes(bx, by, bz, false) <= kSmem) {
          P.xg = false;
          for (int k : {16, 12, 8, 4, 2})
            if (cells <= (int64_t)k * kT) P.per_thread = k;
        } else if (cells <= 20 * kT && brick_bytes(bx, by, bz, true) <= kSmem) {
          P.xg = true;
          P.per_thread = 20;
        } else {
          continue;
        }
        P.gx = gx;
        P.gy = gy;
        P.gz = gz;
        P.smem = brick_bytes(bx, by, bz, P.xg);
        P.cap = (int)std::min<int64_t>(cells, (int64_t)((kSmem - P.smem) / kEntryBytes) / 4 * 4);
        P.smem += P.cap * kEntryBytes;
        best = P;
        least = cost;
      }
  if (best.gx == 0) return best;
  // a cooperative launch needs every block resident
  int most = 0, dev = 0, coop = 0;
  bool ok = false;
  if (best.xg) ok = prepare<20, true>(best, &most);
  else if (best.per_thread == 2) ok = prepare<2, false>(best, &most);
  else if (best.per_thread == 4) ok = prepare<4, false>(best, &most);
  else if (best.per_thread == 8) ok = prepare<8, false>(best, &most);
  else if (best.per_thread == 12) ok = prepare<12, false>(best, &most);
  else ok = prepare<16, false>(best, &most);
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess)
    ok = false;
  if (!ok || !coop || most < 1) {
    cudaGetLastError();
    return BrickPlan{};
  }
  return best;
}

size_t brick_slots_bytes() { return sizeof(double) * 4 * kMaxBlocks + 16; }

cudaError_t brick_solve(const BrickPlan& P, const Op7<double>& A, const double* phi, const double* b, double* x,
                        double* zx, void* slots, PcgState* st, double dx, double rho_neg, double rho_pos,
                        cudaStream_t s) {
  BrickArgs B{};
  B.L = A.L;
  B.gx = P.gx;
  B.gy = P.gy;
  B.gz = P.gz;
  B.ax = A.ax;
  B.ay = A.ay;
  B.az = A.az;
  B.diag = A.diag;
  B.phi = phi;
  B.b = b;
  B.extra0 = A.extra0;
  B.x = x;
  B.zx = zx;
  B.sums = (double*)slots;
  B.count = (unsigned*)(B.sums + 4 * kMaxBlocks);
  B.st = st;
  const double inv2 = 1.0 / (dx * dx);
  B.a[1] = (1.0 / rho_neg) * inv2;
  B.a[2] = (1.0 / rho_pos) * inv2;
  B.cap = P.cap;
  B.c_extra = A.c_extra >= 0 ? A.c_extra : A.L.at(0, 0, 0);
  cudaError_t e = cudaMemsetAsync(B.count, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  void* args[] = {&B};
  return cudaLaunchCooperativeKernel(kernel_of(P), dim3(P.gx * P.gy * P.gz), dim3(kT), args, P.smem, s);
}

}  // namespace fsb
