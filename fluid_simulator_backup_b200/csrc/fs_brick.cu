// Pressure solves of small boxes as one resident kernel: the FP64 Jacobi-PCG
// (PCG_METHOD.cpp:4-126) below, the red-black iteration of the FP32 contexts after
// it, for grids whose vectors fit the SMs' shared memory and registers.
//
// What bounds it.  At 64^3 and 96^3 an iteration of three kernels (fs_krylov.cu)
// takes 20 to 31 us, nearly all of it launches, grid-wide reductions and cold
// starts: the vectors are a few MB.  Here one block per SM (fewer in the smallest
// boxes) keeps a brick of the box: r and q in registers, p (with a one-cell halo)
// and x in shared memory.  The couplings are not kept: away from the interface
// every face carries its phase's 1/rho, and a byte per cell says which (and which
// faces lie on a wall).  The cells next to the interface are a list of their own, worked off
// by all threads before the rest (inline, each of a thread's 12 cells would wait
// for its couplings in turn: 41 us per iteration at 96^3), with their couplings
// in shared memory as far as it reaches and in global memory beyond.  The list
// is in the order of the cells, not in that of the warps' arrival: a listed cell
// and one beyond the list's end round alike only as far as the compiler
// contracts their expressions alike, and a solve has to repeat bit for bit.
//
// One iteration exchanges twice: p.q, then r.z with r.r.  The sums are also
// the barrier, and every block adds them in the same order, so alpha, beta and
// the decisions are the same everywhere.  The halo of p follows from p = z + beta
// p with the neighbours' z, which they store before the second exchange; no third
// one is needed.  The blocks wait
// on one another, so the launch is cooperative; every wait has a limit.  A block
// whose wait ran out sets timed_out, whatever the others made of that exchange,
// and leaves; the waits of those that go on then run out too.
//
// Measured (B200), per iteration, three kernels in a graph -> this one: 32^3
// 17.8 -> 5.8 us, 64^3 22.9 -> 7.7, 96^3 46.9 -> 14.6, 112^3 62.8 -> 29.9.  The
// two exchanges take 3.7 us of it (144 blocks); the rest is instruction issue and
// latency at 16 warps per SM (the registers hold r and q).
#include <algorithm>

#include "fs_kernels.h"

namespace fsb {

namespace {

constexpr int kT = 512;                    // threads of a block
constexpr int kMaxBlocks = 256;            // one poller per block
constexpr size_t kSmem = 227 * 1024 - 2048;  // dynamic shared memory of a block (static: the reductions)

// At least this many cells per block: a box of 24^3 or less leaves most SMs to
// the solves of other contexts.  One context does not notice (FP64 projection to
// 1e-8, one block per SM -> so: 16^3 0.88 -> 0.79 ms, 24^3 1.19 -> 1.25, 32^3 1.53
// -> 1.57; 1024 cells a block: 0.85, 1.37, 1.66), sixteen do (each: 16^3 0.65 ->
// 0.12, 24^3 0.97 -> 0.23, 32^3 1.26 -> 0.65).
constexpr int64_t kBlockCells = 512;

struct BrickArgs {
  Lay L;
  int gx, gy, gz;
  const double *ax, *ay, *az, *diag, *phi, *b, *extra0;
  double *x, *zx;
  double* sums;       // [2][2][kMaxBlocks]: turn, value, block
  unsigned* count;    // blocks that have stored their sums, over all turns
  int cap;            // mixed cells whose couplings fit in shared memory
  unsigned polls;     // before a wait gives up
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
// exchanges of the solve from 1.  Returns false when this block's wait ran out
// after `polls` polls; the others' may not have.
__device__ __forceinline__ bool exchange(double* all_sums, unsigned* count, unsigned polls, int nb, unsigned turn,
                                         bool two, double& v0, double& v1) {
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
  double* sums = all_sums + (turn & 1u) * 2 * kMaxBlocks;  // the other half may still be read
  if (warp == 0) {
    const double s0 = warp_sum(lane < kT / 32 ? part[0][lane] : 0.0);
    const double s1 = two ? warp_sum(lane < kT / 32 ? part[1][lane] : 0.0) : 0.0;
    if (lane == 0) {
      __stcg(sums + blockIdx.x, s0);
      if (two) __stcg(sums + kMaxBlocks + blockIdx.x, s1);
      // release: cumulative over the block's stores (after the barrier above)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      const unsigned want = turn * (unsigned)nb;
      unsigned got = 0, n = 0;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(count) : "memory");
        if ((int)(got - want) >= 0) break;
        if (++n >= polls) {
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

// Numbers the mixed ones of the places 0 .. n-1 in their order, by ballots over a
// range of places per warp: put(t, e) for the e-th.  Called by all threads;
// returns how many there are.
template <class Mixed, class Put>
__device__ __forceinline__ int number_mixed(int n, Mixed mixed, Put put) {
  __shared__ int count[kT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int range = (n + kT - 1) / kT * 32, t0 = warp * range, t1 = min(n, t0 + range);
  int own = 0;
  for (int t = t0; t < t1; t += 32) own += __popc(__ballot_sync(0xffffffffu, t + lane < t1 && mixed(t + lane)));
  if (lane == 0) count[warp] = own;
  __syncthreads();
  int e = 0, all = 0;
  for (int w = 0; w < kT / 32; ++w) {
    if (w < warp) e += count[w];
    all += count[w];
  }
  for (int t = t0; t < t1; t += 32) {
    const bool m = t + lane < t1 && mixed(t + lane);
    const unsigned b = __ballot_sync(0xffffffffu, m);
    if (m) put(t + lane, e + __popc(b & ((1u << lane) - 1u)));
    e += __popc(b);
  }
  return all;
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
    }
  }
  __syncthreads();
  const int listed = min(A.cap, number_mixed(cells, [&](int t) { return kind[t] < 64; }, [&](int t, int e) {
    me[t] = (unsigned short)e;
    if (e >= A.cap) return;
    const int lx = t % bx, row = t / bx, ly = row % by, lz = row / by;
    const int64_t g = base + go[t];
    mt[e] = (unsigned short)t;
    mp[e] = (unsigned short)((lz + 1) * sz + (ly + 1) * sy + lx + 1);
    mdi[e] = 1.0 / A.diag[g];
    ma[e] = A.ax[g];
    ma[A.cap + e] = A.ax[g + 1];
    ma[2 * A.cap + e] = A.ay[g];
    ma[3 * A.cap + e] = A.ay[g + L.px];
    ma[4 * A.cap + e] = A.az[g];
    ma[5 * A.cap + e] = A.az[g + L.slab];
  }));
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
    for (int e = tid; e < listed; e += kT) {
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
    return v * (me[t] < A.cap ? mdi[me[t]] : 1.0 / A.diag[base + go[t]]);
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
  bool alive = exchange(A.sums, A.count, A.polls, nb, ++turn, true, rz, rr);
  alive = exchange(A.sums, A.count, A.polls, nb, ++turn, false, bb, zero) && alive;
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
    if (!exchange(A.sums, A.count, A.polls, nb, ++turn, false, pq, zero)) {
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
    if (!exchange(A.sums, A.count, A.polls, nb, ++turn, true, rz1, rr1)) {
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
  if (tid == 0 && status == PCG_TIMEOUT) A.st->timed_out = 1;
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

// ---------------------------------------------------------------------------
// The red-black iteration of fs_redblack.cu (CG on the black Schur complement:
// FP32 vectors, FP64 iterate, bf16 pivots) between two reliable updates, as
// one resident kernel in the manner of the one above.
//
// What bounds it: at 96^3 the five kernels of an iteration move a few MB that L2
// holds, and 26.5 us go into their launches, cold starts and grid-wide
// reductions.  Here a brick's p and the tau of its red cells live in shared
// memory, one array per colour (neighbouring threads read neighbouring words; one
// array of both colours would be read two words apart), p with a halo of two
// cells and tau with one: each brick computes the tau of the red cells around it
// itself, so that an iteration still exchanges only twice.  r and q are
// registers, the FP64 iterate is in shared memory.  Every value is computed by the
// expressions of fs_redblack.cu and fs_krylov.cu in the same order; only the
// sums over the grid add in another one.  Measured, a whole projection to 1e-8 with five
// kernels per iteration -> with this one: 32^3 (120 iterations) 4.0 -> 1.5 ms,
// 64^3 (218) 7.2 -> 2.6, 96^3 (327) 14.2 -> 5.6, 120^3 (396) 25.3 -> 14.3.
// ---------------------------------------------------------------------------
struct RbBrickArgs {
  Lay L, H;
  int gx, gy, gz;
  const float *ax, *ay, *az, *phi;
  const double* extra0;
  float *r, *p, *z;
  const unsigned short* dinv;
  double* sums;
  unsigned* count;
  unsigned polls;
  PcgState* st;
  float a[3];  // uniform coupling of a phase
  int cap;     // mixed cells listed in shared memory
};

struct Six {
  float xm, xp, ym, yp, zm, zp;
};

// tau of the red cell in place c of its colour's array; o: its column is the
// second of its pair; first: it lies in column 0 of the box
__device__ __forceinline__ float brick_tau(const float* PB, int c, int o, int hy, int hz, bool first, const Six& a,
                                           float e0) {
  const float xm = PB[c + o - 1], xp = PB[c + o], ym = PB[c - hy], yp = PB[c + hy], zm = PB[c - hz], zp = PB[c + hz];
  const float b0 = first ? xp : xm;
  float num = a.xm * (xm - b0) + a.xp * (xp - b0);
  num += a.ym * (ym - b0) + a.yp * (yp - b0);
  num += a.zm * (zm - b0) + a.zp * (zp - b0);
  float d = ((a.xm + a.xp) + (a.ym + a.yp)) + (a.zm + a.zp);
  if (e0 != 0.0f) {
    num -= e0 * b0;
    d += e0;
  }
  return d > 0.0f ? num / d : 0.0f;
}

// (S p) of the black cell in place c; column: 0, 1 or 2 (any later one)
__device__ __forceinline__ float brick_schur(const float* PB, const float* PR, int c, int o, int hy, int hz, int column,
                                             const Six& a) {
  const float pc = PB[c];
  const float txm = PR[c + o - 1], txp = PR[c + o], tym = PR[c - hy], typ = PR[c + hy], tzm = PR[c - hz],
              tzp = PR[c + hz];
  const int b = column > 0 ? o - 1 : 0;
  const float dxm = column > 1 ? pc - PB[c - 1] : 0.0f;
  const float dym = pc - PB[c - hy + b], dyp = pc - PB[c + hy + b];
  const float dzm = pc - PB[c - hz + b], dzp = pc - PB[c + hz + b];
  float acc = a.xm * (dxm - txm) + a.xp * (0.0f - txp);
  acc += a.ym * (dym - tym) + a.yp * (dyp - typ);
  acc += a.zm * (dzm - tzm) + a.zp * (dzp - tzp);
  return acc;
}

// black cells of the halo (two layers on each face, the twelve edges between
// them; half of each, rounded up) and red cells of the first layer
__host__ __device__ inline int rb_halo(int bx, int by, int bz) {
  return 2 * (by * bz + bx * bz + bx * by) + 2 * (bx + by + bz) + 24;
}
__host__ __device__ inline int rb_ring(int bx, int by, int bz) { return by * bz + bx * bz + bx * by + 6; }

constexpr int kNotListed = 255;

// K: packed slots (a black and a red cell) per thread
template <int K>
__global__ void __launch_bounds__(kT, 1) k_rb_brick(const __grid_constant__ RbBrickArgs A) {
  extern __shared__ double smem[];
  const Lay &L = A.L, &H = A.H;
  const int nb = gridDim.x, tid = threadIdx.x;
  const int qx = blockIdx.x % A.gx, qy = (blockIdx.x / A.gx) % A.gy, qz = blockIdx.x / (A.gx * A.gy);
  const int h0 = (int)((int64_t)qx * H.nx / A.gx), h1 = (int)((int64_t)(qx + 1) * H.nx / A.gx);
  const int j0 = (int)((int64_t)qy * L.ny / A.gy), j1 = (int)((int64_t)(qy + 1) * L.ny / A.gy);
  const int k0 = (int)((int64_t)qz * L.nz / A.gz), k1 = (int)((int64_t)(qz + 1) * L.nz / A.gz);
  const int i0 = 2 * h0, bh = h1 - h0, bx = 2 * bh, by = j1 - j0, bz = k1 - k0, slots = bh * by * bz;
  const int sy = bx + 4, sz = sy * (by + 4), padded = sz * (bz + 4), hy = sy / 2, hz = sz / 2;
  double* xs = smem;
  float* PB = (float*)(xs + slots);
  float* PR = PB + padded / 2;
  float* ma = PR + padded / 2;  // the list of mixed cells: couplings, q, place
  float* mq = ma + 6 * (size_t)A.cap;
  int* list = (int*)(mq + A.cap);
  int* hp = list + A.cap;  // black halo cells: place and packed offset
  int* hg = hp + rb_halo(bx, by, bz);
  int* ring = hg + rb_halo(bx, by, bz);
  int* go = ring + rb_ring(bx, by, bz);                // a slot's packed offset
  unsigned short* me = (unsigned short*)(go + slots);  // a listed black cell's entry
  unsigned short* dv = me + slots;
  unsigned char* kind = (unsigned char*)(dv + slots);
  __shared__ int nhalo, nring;
  const PcgState in = *A.st;
  if (in.done) return;  // the same in every block
  double* x = (double*)in.x;
  if (tid == 0) nhalo = nring = 0;
  for (int t = tid; t < padded; t += kT) kind[t] = 0;
  for (int t = tid; t < padded / 2; t += kT) PB[t] = PR[t] = 0.0f;
  __syncthreads();
  const int64_t hbase = H.at(h0, j0, k0);
  // Every cell of the padded brick that takes part: its place in the lists, and
  // for a red cell of the brick or its first layer and a black cell of the brick
  // its kind: bits 0..5 the face lies inside the box, 6 and 7 the phase whose
  // 1/rho all faces carry.  0: listed (or no cell), kNotListed: the list is full.
  for (int t = tid; t < padded; t += kT) {
    const int lz = t / sz - 2, ly = t % sz / sy - 2, lx = t % sy - 2;
    const int i = i0 + lx, j = j0 + ly, k = k0 + lz;
    if (i < 0 || i >= L.nx || j < 0 || j >= L.ny || k < 0 || k >= L.nz) continue;
    const int ox = lx < 0 ? -lx : (lx >= bx ? lx - bx + 1 : 0), oy = ly < 0 ? -ly : (ly >= by ? ly - by + 1 : 0),
              oz = lz < 0 ? -lz : (lz >= bz ? lz - bz + 1 : 0);
    const int off = ox + oy + oz;
    const bool black = (i + j + k) & 1;
    if (off > (black ? 2 : 1)) continue;
    if (black && off > 0) {
      const int e = atomicAdd(&nhalo, 1);
      hp[e] = t >> 1;
      hg[e] = (int)(((i >> 1) - h0) + (int64_t)(j - j0) * H.px + (int64_t)(k - k0) * H.slab);
      continue;
    }
    if (off > 0) ring[atomicAdd(&nring, 1)] = t;
    const int f = (i > 0) | (i < L.nx - 1) << 1 | (j > 0) << 2 | (j < L.ny - 1) << 3 | (k > 0) << 4 | (k < L.nz - 1) << 5;
    const float* ph = A.phi + L.at(i, j, k);
    const bool n = ph[0] <= 0.0f;
    auto alike = [&](int64_t o) { return n ? ph[o] <= 0.0f : ph[o] > 0.0f; };  // NaN: of no phase
    const bool same = alike(0) && !(i == 0 && j == 0 && k == 0) && (!(f & 1) || alike(-1)) && (!(f & 2) || alike(1)) &&
                      (!(f & 4) || alike(-L.px)) && (!(f & 8) || alike(L.px)) && (!(f & 16) || alike(-L.slab)) &&
                      (!(f & 32) || alike(L.slab));
    kind[t] = same ? (unsigned char)(f | (n ? 64 : 128)) : kNotListed;
  }
  __syncthreads();
  const int mixed = number_mixed(padded, [&](int t) { return kind[t] == kNotListed; }, [&](int t, int e) {
    if (e >= A.cap) return;
    kind[t] = 0;
    const int lz = t / sz - 2, ly = t % sz / sy - 2, lx = t % sy - 2;
    const int i = i0 + lx, j = j0 + ly, k = k0 + lz;
    const bool black = (i + j + k) & 1;
    list[e] = t | (black ? 1 << 30 : 0) | min(i, 2) << 28;
    if (black) me[(lz * by + ly) * bh + (lx >> 1)] = (unsigned short)e;
    const int64_t g = L.at(i, j, k);
    ma[e] = A.ax[g];
    ma[A.cap + e] = A.ax[g + 1];
    ma[2 * A.cap + e] = A.ay[g];
    ma[3 * A.cap + e] = A.ay[g + L.px];
    ma[4 * A.cap + e] = A.az[g];
    ma[5 * A.cap + e] = A.az[g + L.slab];
  });
  // this thread's slots: index of the cell in the pair's first column, which
  // of the two is black, whether that one exists and its column
  int base[K];
  unsigned second = 0u, have = 0u, col0 = 0u, col1 = 0u;
  float r[K], q[K];
#pragma unroll
  for (int m = 0; m < K; ++m) {
    const int t = tid + m * kT;
    base[m] = -1;
    r[m] = q[m] = 0.0f;
    if (t < slots) {
      const int h = t % bh, row = t / bh, ly = row % by, lz = row / by;
      base[m] = (lz + 2) * sz + (ly + 2) * sy + 2 * h + 2;
      const int o = (j0 + ly + k0 + lz + 1) & 1, i = i0 + 2 * h + o;
      second |= (unsigned)o << m;
      if (i < L.nx) have |= 1u << m;
      if (i == 0) col0 |= 1u << m;
      if (i == 1) col1 |= 1u << m;
      go[t] = (int)(h + (int64_t)ly * H.px + (int64_t)lz * H.slab);
      const int64_t g = hbase + go[t];
      r[m] = A.r[g];
      dv[t] = A.dinv[g];
      xs[t] = x[g];
      PB[base[m] >> 1] = A.p[g];
    }
  }
  __syncthreads();
  const int halos = nhalo, rings = nring, listed = min(mixed, A.cap);
  for (int e = tid; e < halos; e += kT) PB[hp[e]] = A.p[hbase + hg[e]];
  // the first cell of the box, which carries the deflation term, where this brick needs its tau
  const int origin = i0 == 0 && j0 <= 1 && k0 <= 1 ? (2 - k0) * sz + (2 - j0) * sy + 2 : -1;
  const float e0 = (float)*A.extra0;
  __syncthreads();

  auto uniform = [&](int f) -> Six {
    const float a = A.a[f >> 6];
    if ((f & 63) == 63) return {a, a, a, a, a, a};
    return {f & 1 ? a : 0.0f, f & 2 ? a : 0.0f, f & 4 ? a : 0.0f, f & 8 ? a : 0.0f, f & 16 ? a : 0.0f, f & 32 ? a : 0.0f};
  };
  auto entry = [&](int e) -> Six {
    return {ma[e], ma[A.cap + e], ma[2 * A.cap + e], ma[3 * A.cap + e], ma[4 * A.cap + e], ma[5 * A.cap + e]};
  };
  auto fetched = [&](int t) -> Six {
    const int64_t g = L.at(i0 + t % sy - 2, j0 + t % sz / sy - 2, k0 + t / sz - 2);
    return {A.ax[g], A.ax[g + 1], A.ay[g], A.ay[g + L.px], A.az[g], A.az[g + L.slab]};
  };
  auto tau = [&](int t) {  // of a red cell that is not listed
    const int f = kind[t];
    if (f == kNotListed)
      PR[t >> 1] = brick_tau(PB, t >> 1, t & 1, hy, hz, i0 + t % sy - 2 == 0, fetched(t), t == origin ? e0 : 0.0f);
    else if (f)
      PR[t >> 1] = brick_tau(PB, t >> 1, t & 1, hy, hz, !(f & 1), uniform(f), 0.0f);
  };
  double rz = in.rz, rr = in.rr, rz_prev = in.rz_prev, best = in.best_rr, alpha = in.alpha, beta = in.beta;
  int iter = in.iter, stall = in.stall, status = PCG_RUNNING;
  unsigned turn = 0;
  while (status == PCG_RUNNING) {
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (base[m] >= 0) tau(base[m] + 1 - (int)(second >> m & 1u));
    for (int e = tid; e < rings; e += kT) tau(ring[e]);
    for (int e = tid; e < listed; e += kT)
      if (!(list[e] >> 30)) {
        const int t = list[e] & 0xfffffff;
        PR[t >> 1] = brick_tau(PB, t >> 1, t & 1, hy, hz, list[e] >> 28 == 0, entry(e), t == origin ? e0 : 0.0f);
      }
    __syncthreads();
    for (int e = tid; e < listed; e += kT)
      if (list[e] >> 30) {
        const int t = list[e] & 0xfffffff;
        mq[e] = brick_schur(PB, PR, t >> 1, t & 1, hy, hz, list[e] >> 28 & 3, entry(e));
      }
    __syncthreads();
    double pq = 0.0, none = 0.0;
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (have >> m & 1u) {
        const int o = (int)(second >> m & 1u), t = base[m] + o, f = kind[t];
        const int column = col0 >> m & 1u ? 0 : (col1 >> m & 1u ? 1 : 2);
        if (f == 0)
          q[m] = mq[me[tid + m * kT]];
        else
          q[m] = brick_schur(PB, PR, t >> 1, o, hy, hz, column, f == kNotListed ? fetched(t) : uniform(f));
        pq += (double)PB[t >> 1] * (double)q[m];
      }
    if (!exchange(A.sums, A.count, A.polls, nb, ++turn, false, pq, none)) {
      status = PCG_TIMEOUT;
      break;
    }
    alpha = rz / pq;
    if (!(pq > 0.0) || !isfinite(alpha)) {
      status = PCG_STAGNATED;
      break;
    }
    const float al = (float)alpha;
    double rz1 = 0.0, rr1 = 0.0;
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (have >> m & 1u) {
        const int t = tid + m * kT;
        r[m] -= al * q[m];
        const float z = r[m] * __uint_as_float((unsigned)dv[t] << 16);
        __stcg(A.z + hbase + go[t], z);
        q[m] = z;
        rz1 += (double)r[m] * (double)z;
        rr1 += (double)r[m] * (double)r[m];
      }
    if (!exchange(A.sums, A.count, A.polls, nb, ++turn, true, rz1, rr1)) {
      status = PCG_TIMEOUT;
      break;
    }
    // the decisions of k_cg_update, the same in every block
    rz_prev = rz;
    rz = rz1;
    rr = rr1;
    if (rr < 0.99 * best) {
      best = rr;
      stall = 0;
    } else {
      ++stall;
    }
    if (!isfinite(rz) || !isfinite(rr)) {
      status = PCG_NONFINITE;  // x is not moved along that step
      break;
    }
    if (in.criterion == 2 ? rr < in.tol * in.tol : (in.criterion == 1 ? rz < in.tol * in.tol : sqrt(rr) <= in.tol * sqrt(in.bb))) {
      status = PCG_CONVERGED;
    } else {
      beta = rz / rz_prev;
      ++iter;
      if (iter >= in.max_iter) status = PCG_MAXITER;
      else if (in.stall_limit > 0 && stall >= in.stall_limit) status = PCG_STAGNATED;
      else if (in.reliable_delta > 0.0 && rr < in.reliable_delta * in.reliable_delta * in.max_rr)
        status = PCG_RELIABLE_UPDATE;
    }
    const float be = (float)beta;
#pragma unroll
    for (int m = 0; m < K; ++m)
      if (have >> m & 1u) {
        const float pv = PB[base[m] >> 1];
        xs[tid + m * kT] += alpha * (double)pv;
        if (status == PCG_RUNNING) PB[base[m] >> 1] = pv * be + q[m];
      }
    if (status == PCG_RUNNING) {
      constexpr int kFetch = 6;  // neighbours' z in flight
      for (int f0 = tid; f0 < halos; f0 += kFetch * kT) {
        int at[kFetch];
        float z[kFetch];
#pragma unroll
        for (int m = 0; m < kFetch; ++m) {
          const int e = f0 + m * kT;
          at[m] = e < halos ? hp[e] : -1;
          z[m] = at[m] >= 0 ? __ldcg(A.z + hbase + hg[e]) : 0.0f;
        }
#pragma unroll
        for (int m = 0; m < kFetch; ++m)
          if (at[m] >= 0) PB[at[m]] = PB[at[m]] * be + z[m];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < K; ++m)
    if (have >> m & 1u) {
      const int t = tid + m * kT;
      const int64_t g = hbase + go[t];
      A.r[g] = r[m];
      A.p[g] = PB[base[m] >> 1];
      x[g] = xs[t];
    }
  if (tid == 0 && status == PCG_TIMEOUT) A.st->timed_out = 1;
  if (blockIdx.x == 0 && tid == 0) {
    PcgState* st = A.st;
    st->rz = rz;
    st->rr = rr;
    st->rz_prev = rz_prev;
    st->best_rr = best;
    st->stall = stall;
    st->alpha = alpha;
    st->beta = beta;
    st->iter = iter;
    st->x_pending = 0;
    st->status = status;
    st->done = status == PCG_RELIABLE_UPDATE ? 2 : 1;
  }
}

// blocks that a box may have
int blocks_for(const Lay& L, int sms) {
  const int64_t cells = (int64_t)L.nx * L.ny * L.nz;
  return (int)std::min<int64_t>(std::min(sms, kMaxBlocks), (cells + kBlockCells - 1) / kBlockCells);
}

size_t rb_brick_bytes(int bh, int by, int bz) {
  const int bx = 2 * bh;
  const size_t slots = (size_t)bh * by * bz, padded = (size_t)(bx + 4) * (by + 4) * (bz + 4);
  return slots * 8 + padded * 4 + (2 * (size_t)rb_halo(bx, by, bz) + rb_ring(bx, by, bz)) * 4 + slots * 8 +
         (padded + 7) / 8 * 8;
}
constexpr size_t kRbEntryBytes = 6 * 4 + 4 + 4;

const void* rb_kernel_of(int per_thread) {
  switch (per_thread) {
    case 2: return (const void*)k_rb_brick<2>;
    case 4: return (const void*)k_rb_brick<4>;
    case 6: return (const void*)k_rb_brick<6>;
    case 8: return (const void*)k_rb_brick<8>;
    default: return (const void*)k_rb_brick<12>;
  }
}

}  // namespace

// The division of the box into at most blocks_for() bricks: the smallest largest
// brick, counting a halo cell as a third of a cell and one on an x face (a
// strided access) as a whole one.
BrickPlan brick_plan(const Lay& L, int sms) {
  BrickPlan best;
  double least = 1e300;
  sms = blocks_for(L, sms);
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
  B.polls = P.polls;
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

// The same for the red-black iteration: bricks of whole pairs of columns.
BrickPlan rb_brick_plan(const Lay& L, const Lay& H, int sms) {
  BrickPlan best;
  double least = 1e300;
  sms = blocks_for(L, sms);
  for (int gz = 1; gz <= std::min(sms, L.nz); ++gz)
    for (int gy = 1; gy <= std::min(sms / gz, L.ny); ++gy)
      for (int gx = 1; gx <= std::min(sms / gz / gy, H.nx); ++gx) {
        const int bh = (H.nx + gx - 1) / gx, by = (L.ny + gy - 1) / gy, bz = (L.nz + gz - 1) / gz;
        const double cost = 2.0 * bh * by * bz + 3.0 * by * bz * (gx > 1) +
                            2.0 * ((double)bh * bz * (gy > 1) + (double)bh * by * (gz > 1));
        const int64_t slots = (int64_t)bh * by * bz;
        if (cost >= least || slots > 12 * kT || rb_brick_bytes(bh, by, bz) > kSmem) continue;
        BrickPlan P;
        for (int k : {12, 8, 6, 4, 2})
          if (slots <= (int64_t)k * kT) P.per_thread = k;
        P.gx = gx;
        P.gy = gy;
        P.gz = gz;
        P.smem = rb_brick_bytes(bh, by, bz);
        P.cap = (int)std::min<int64_t>(3 * slots, (int64_t)((kSmem - P.smem) / kRbEntryBytes) / 4 * 4);
        P.smem += P.cap * kRbEntryBytes;
        best = P;
        least = cost;
      }
  if (best.gx == 0) return best;
  int most = 0, dev = 0, coop = 0;
  const void* k = rb_kernel_of(best.per_thread);
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, k, kT, best.smem) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      !coop || most < 1) {
    cudaGetLastError();
    return BrickPlan{};
  }
  return best;
}

cudaError_t rb_brick_iterate(const BrickPlan& P, const RbOp& A, const float* phi, float* rh, float* ph, float* zh,
                             const unsigned short* dinv, void* slots, PcgState* st, double dx, double rho_neg,
                             double rho_pos, cudaStream_t s) {
  RbBrickArgs B{};
  B.L = A.L;
  B.H = A.Lh;
  B.gx = P.gx;
  B.gy = P.gy;
  B.gz = P.gz;
  B.ax = A.ax;
  B.ay = A.ay;
  B.az = A.az;
  B.phi = phi;
  B.extra0 = A.extra0;
  B.r = rh;
  B.p = ph;
  B.z = zh;
  B.dinv = dinv;
  B.sums = (double*)slots;
  B.count = (unsigned*)(B.sums + 4 * kMaxBlocks);
  B.polls = P.polls;
  B.st = st;
  const double inv2 = 1.0 / (dx * dx);
  B.a[1] = (float)((1.0 / rho_neg) * inv2);
  B.a[2] = (float)((1.0 / rho_pos) * inv2);
  B.cap = P.cap;
  cudaError_t e = cudaMemsetAsync(B.count, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  void* args[] = {&B};
  return cudaLaunchCooperativeKernel(rb_kernel_of(P.per_thread), dim3(P.gx * P.gy * P.gz), dim3(kT), args, P.smem, s);
}

}  // namespace fsb
