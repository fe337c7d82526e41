// The level-set and velocity updates and the Sussman step of a TAPED forward:
// the recomputed forward of fs_step_adjoint and of the operator adjoints.
//
// The adjoint freezes the Godunov branch of every Sussman step at its forward
// value.  Where the gradient of phi vanishes (the ridges of a distance field)
// that branch, and with it an O(1) part of the gradient in those cells, hangs
// on the last bit of phi.  The kernels here keep one evaluation order, term by
// term (ADVECTION_METHOD_3D.h:42-279, 745-1637), so that gradients do not move
// when the forward kernels of fs_stencil.cu are rearranged: with the faster
// form there the bar of phi of a 96^3 dam-break step differs by 4e-3 of its
// norm, all of it in such cells; the velocity update, whose upwind sides and
// 1/density weights amplify its last bits less, moves the velocities' bars by
// 5e-6.  They cost 39 us against 20 us per Sussman step at 96^3, about 1 ms of
// a 58 ms adjoint step.  Level-set ghosts are read (the caller fills them).
#include <algorithm>

#include "fs_kernels.h"

namespace fsb {

namespace {

template <class T>
__device__ __forceinline__ T weno_side(T r1, T r2, T r3, T r4, T r5, T eps) {
  const T c1312 = T(13.0 / 12.0);
  T t = (r1 - T(2) * r2) + r3, q = (r1 - T(4) * r2) + T(3) * r3;
  const T s1 = (c1312 * t) * t + (T(0.25) * q) * q;
  t = (r2 - T(2) * r3) + r4; q = r2 - r4;
  const T s2 = (c1312 * t) * t + (T(0.25) * q) * q;
  t = (r3 - T(2) * r4) + r5; q = (T(3) * r3 - T(4) * r4) + r5;
  const T s3 = (c1312 * t) * t + (T(0.25) * q) * q;
  const T e1 = eps + s1, e2 = eps + s2, e3 = eps + s3;
  const T q1 = e1 * e1, q2 = e2 * e2, q3 = e3 * e3;
  const T b1 = T(0.1) * (q2 * q3), b2 = T(0.6) * (q1 * q3), b3 = T(0.3) * (q1 * q2);
  const T inv = T(1) / ((b1 + b2) + b3);
  const T third = T(1.0 / 3.0), sixth = T(1.0 / 6.0);
  const T u1 = (r1 * third - r2 * T(7.0 / 6.0)) + r3 * T(11.0 / 6.0);
  const T u2 = (r2 * (-sixth) + r3 * T(5.0 / 6.0)) + r4 * third;
  const T u3 = (r3 * third + r4 * T(5.0 / 6.0)) - r5 * sixth;
  return ((b1 * u1 + b2 * u2) + b3 * u3) * inv;
}

// D- and D+ from the 7 samples v[0..6] = f[-3..3] along one axis.
template <class T>
__device__ __forceinline__ void weno_pair7(const T v[7], T inv_h, T eps, T& dm, T& dp) {
  const T d1 = inv_h * (v[1] - v[0]), d2 = inv_h * (v[2] - v[1]), d3 = inv_h * (v[3] - v[2]),
          d4 = inv_h * (v[4] - v[3]), d5 = inv_h * (v[5] - v[4]), d6 = inv_h * (v[6] - v[5]);
  dm = weno_side(d1, d2, d3, d4, d5, eps);
  dp = weno_side(d6, d5, d4, d3, d2, eps);
}

// ---------------------------------------------------------------------------
// shared-memory plane ring of the staged stencil kernels
// ---------------------------------------------------------------------------
constexpr int kTX = 32, kTY = 8;                     // tile (threads) in x and y
constexpr int kRW = kTX + 2 * GH, kRH = kTY + 2 * GH;  // staged plane: tile + halo
constexpr int kRing = 2 * GH + 1;                    // planes k-3 .. k+3

__device__ __forceinline__ int ring_slot(int k) { return ((k % kRing) + kRing) % kRing; }

// Plane k of f (halo included) into its ring slot: row-contiguous loads of
// the (32+6) x (8+6) window; halo cells beyond the ghost ring (i >= nx+3 or
// j >= ny+3, only at the tile past the box edge) are not needed and skipped.
template <class T>
__device__ __forceinline__ void stage_plane(T* ring, const T* __restrict__ f, const Lay& L, int i0, int j0, int k) {
  T* dst = ring + ring_slot(k) * (kRW * kRH);
  const int tid = threadIdx.x + kTX * threadIdx.y;
  for (int t = tid; t < kRW * kRH; t += kTX * kTY) {
    const int x = t % kRW, y = t / kRW;
    const int gi = i0 - GH + x, gj = j0 - GH + y;
    if (gi < L.nx + GH && gj < L.ny + GH) dst[t] = f[L.at(gi, gj, k)];
  }
}

// The seven samples of (tx, ty) in plane k along x, y and z from the ring.
template <class T>
__device__ __forceinline__ void ring_samples(const T* ring, int k, T vx[7], T vy[7], T vz[7]) {
  const int tx = threadIdx.x + GH, ty = threadIdx.y + GH;
  const T* pc = ring + ring_slot(k) * (kRW * kRH);
#pragma unroll
  for (int o = 0; o < 7; ++o) {
    vx[o] = pc[ty * kRW + tx + o - GH];
    vy[o] = pc[(ty + o - GH) * kRW + tx];
    vz[o] = ring[ring_slot(k + o - GH) * (kRW * kRH) + ty * kRW + tx];
  }
}

// Grid of a staged kernel: xy tiles times z chunks, enough blocks to fill
// the GPU a few times over (each chunk re-stages six halo planes).
struct StagedGrid {
  dim3 grid;
  int kchunk;
};
inline StagedGrid staged_grid(const Lay& L) {
  static int sms = 0;
  if (sms <= 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  }
  const int tx = (L.nx + kTX - 1) / kTX, ty = (L.ny + kTY - 1) / kTY;
  const int want = 8 * sms;
  const int chunks = std::max(1, std::min(L.nz, (want + tx * ty - 1) / (tx * ty)));
  const int kchunk = (L.nz + chunks - 1) / chunks;
  StagedGrid g;
  g.grid = dim3(tx, ty, (L.nz + kchunk - 1) / kchunk);
  g.kchunk = kchunk;
  return g;
}

// out = c0*base + c1*(src - dt*(u.grad src)), the level-set update at cell
// centres; u, v, w are the MAC faces (zero ghosts).  With c0 == 0 the
// combination is skipped and out is the forward-Euler value.
template <class T>
__global__ void __launch_bounds__(kTX * kTY) k_taped_levelset(const T* __restrict__ src, const T* __restrict__ base,
                                                           T* __restrict__ out, const T* __restrict__ u,
                                                           const T* __restrict__ v, const T* __restrict__ w, Lay L,
                                                           Lay Lu, Lay Lv, Lay Lw, T inv_h, T eps, T dt, T c0, T c1,
                                                           int kchunk) {
  __shared__ T ring[kRing * kRW * kRH];
  const int i0 = blockIdx.x * kTX, j0 = blockIdx.y * kTY;
  const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(L.nz, k0 + kchunk);
  const bool valid = i < L.nx && j < L.ny;
  for (int kk = k0 - GH; kk < k0 + GH; ++kk) stage_plane(ring, src, L, i0, j0, kk);
  for (int k = k0; k < k1; ++k) {
    stage_plane(ring, src, L, i0, j0, k + GH);
    __syncthreads();
    if (valid) {
      T vx[7], vy[7], vz[7];
      ring_samples(ring, k, vx, vy, vz);
      T dxm, dxp, dym, dyp, dzm, dzp;
      weno_pair7(vx, inv_h, eps, dxm, dxp);
      weno_pair7(vy, inv_h, eps, dym, dyp);
      weno_pair7(vz, inv_h, eps, dzm, dzp);
      const int64_t c = L.at(i, j, k);
      const T uc = (u[Lu.at(i + 1, j, k)] + u[Lu.at(i, j, k)]) * T(0.5);
      const T vc = (v[Lv.at(i, j + 1, k)] + v[Lv.at(i, j, k)]) * T(0.5);
      const T wc = (w[Lw.at(i, j, k + 1)] + w[Lw.at(i, j, k)]) * T(0.5);
      const T fe =
          vx[3] - dt * ((uc * (uc > T(0) ? dxm : dxp) + vc * (vc > T(0) ? dym : dyp)) + wc * (wc > T(0) ? dzm : dzp));
      out[c] = c0 == T(0) ? fe : c0 * base[c] + c1 * fe;
    }
    __syncthreads();
  }
}

// The velocities that advect face (i,j,k) of component `axis`: its own
// component, the four-face averages of the other two.
template <class T>
__device__ __forceinline__ void mac_velocity(const T* __restrict__ u, const T* __restrict__ v,
                                             const T* __restrict__ w, const Lay& Lu, const Lay& Lv, const Lay& Lw,
                                             int axis, int i, int j, int k, T& uvel, T& vvel, T& wvel) {
  if (axis == 0) {
    uvel = u[Lu.at(i, j, k)];
    vvel = (((v[Lv.at(i, j, k)] + v[Lv.at(i, j + 1, k)]) + v[Lv.at(i - 1, j, k)]) + v[Lv.at(i - 1, j + 1, k)]) * T(0.25);
    wvel = (((w[Lw.at(i, j, k)] + w[Lw.at(i, j, k + 1)]) + w[Lw.at(i - 1, j, k)]) + w[Lw.at(i - 1, j, k + 1)]) * T(0.25);
  } else if (axis == 1) {
    uvel = (((u[Lu.at(i, j, k)] + u[Lu.at(i + 1, j, k)]) + u[Lu.at(i, j - 1, k)]) + u[Lu.at(i + 1, j - 1, k)]) * T(0.25);
    vvel = v[Lv.at(i, j, k)];
    wvel = (((w[Lw.at(i, j, k)] + w[Lw.at(i, j, k + 1)]) + w[Lw.at(i, j - 1, k)]) + w[Lw.at(i, j - 1, k + 1)]) * T(0.25);
  } else {
    uvel = (((u[Lu.at(i, j, k)] + u[Lu.at(i + 1, j, k)]) + u[Lu.at(i, j, k - 1)]) + u[Lu.at(i + 1, j, k - 1)]) * T(0.25);
    vvel = (((v[Lv.at(i, j, k)] + v[Lv.at(i, j + 1, k)]) + v[Lv.at(i, j, k - 1)]) + v[Lv.at(i, j + 1, k - 1)]) * T(0.25);
    wvel = w[Lw.at(i, j, k)];
  }
}

// MAC component self-advection on every face of component `axis` (wall
// faces included, as the reference's loop covers the whole face grid).
template <class T>
__global__ void __launch_bounds__(kTX * kTY) k_taped_mac(const T* __restrict__ comp, T* __restrict__ out,
                                                      const T* __restrict__ u, const T* __restrict__ v,
                                                      const T* __restrict__ w, Lay Lc, Lay Lu, Lay Lv, Lay Lw,
                                                      int axis, T inv_h, T eps, T dt, int kchunk) {
  __shared__ T ring[kRing * kRW * kRH];
  const int i0 = blockIdx.x * kTX, j0 = blockIdx.y * kTY;
  const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(Lc.nz, k0 + kchunk);
  const bool valid = i < Lc.nx && j < Lc.ny;
  for (int kk = k0 - GH; kk < k0 + GH; ++kk) stage_plane(ring, comp, Lc, i0, j0, kk);
  for (int k = k0; k < k1; ++k) {
    stage_plane(ring, comp, Lc, i0, j0, k + GH);
    __syncthreads();
    if (valid) {
      T uvel, vvel, wvel;
      mac_velocity(u, v, w, Lu, Lv, Lw, axis, i, j, k, uvel, vvel, wvel);
      T vx[7], vy[7], vz[7];
      ring_samples(ring, k, vx, vy, vz);
      T dxm, dxp, dym, dyp, dzm, dzp;
      weno_pair7(vx, inv_h, eps, dxm, dxp);
      weno_pair7(vy, inv_h, eps, dym, dyp);
      weno_pair7(vz, inv_h, eps, dzm, dzp);
      out[Lc.at(i, j, k)] = vx[3] - dt * ((uvel * (uvel > T(0) ? dxm : dxp) + vvel * (vvel > T(0) ? dym : dyp)) +
                                          wvel * (wvel > T(0) ? dzm : dzp));
    }
    __syncthreads();
  }
}

// Per-axis Godunov choice of the reference's case tree.  code: 0 D-, 1 D+,
// 2 dropped (expansion fan).
template <class T>
__device__ __forceinline__ T godunov(T s, T dm, T dp, int& code, bool& shock) {
  const T sm = s * dm, sp = s * dp;
  shock = false;
  if (sp >= T(0) && sm >= T(0)) { code = 0; return dm; }
  if (sp <= T(0) && sm <= T(0)) { code = 1; return dp; }
  if (sp > T(0) && sm < T(0)) { code = 2; return T(0); }
  shock = true;  // sp < 0 < sm
  const T ss = s * (fabs(dp) - fabs(dm)) / (dp - dm);
  if (ss > T(0)) { code = 0; return dm; }
  code = 1;
  return dp;
}

// One pseudo-step phi - dtau*S*(|grad phi|_G - 1) with the sign-preserving
// clamp; out = c0*base + c1*(that) when c0 != 0 (RK block combination).
template <class T>
__global__ void __launch_bounds__(kTX * kTY) k_taped_sussman(const T* __restrict__ src, const T* __restrict__ sgn,
                                                    const T* __restrict__ base, T* __restrict__ out, Lay L, T inv_h,
                                                    T eps, T dtau, T c0, T c1, int typo, int kchunk) {
  __shared__ T ring[kRing * kRW * kRH];
  const int i0 = blockIdx.x * kTX, j0 = blockIdx.y * kTY;
  const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
  const int k0 = blockIdx.z * kchunk, k1 = min(L.nz, k0 + kchunk);
  const bool valid = i < L.nx && j < L.ny;
  for (int kk = k0 - GH; kk < k0 + GH; ++kk) stage_plane(ring, src, L, i0, j0, kk);
  for (int k = k0; k < k1; ++k) {
    stage_plane(ring, src, L, i0, j0, k + GH);
    __syncthreads();
    if (valid) {
      const int64_t c = L.at(i, j, k);
      T vx[7], vy[7], vz[7];
      ring_samples(ring, k, vx, vy, vz);
      T dxm, dxp, dym, dyp, dzm, dzp;
      weno_pair7(vx, inv_h, eps, dxm, dxp);
      weno_pair7(vy, inv_h, eps, dym, dyp);
      weno_pair7(vz, inv_h, eps, dzm, dzp);
      const T s = sgn[c];
      int cx, cy, cz;
      bool shx, shy, shz;
      const T gx = godunov(s, dxm, dxp, cx, shx);
      const T gy = godunov(s, dym, dyp, cy, shy);
      const T gz = godunov(s, dzm, dzp, cz, shz);
      T mag = sqrt((gx * gx + gy * gy) + gz * gz) - T(1);
      if (typo && shx && shy && cy == 1 && cz == 2) mag = (sqrt(gx * gx) + gy * gy) - T(1);
      T r = vx[3] - dtau * s * mag;
      if (s * r < T(0)) {
        if (s < T(0)) r = -eps;
        if (s > T(0)) r = eps;
      }
      out[c] = c0 == T(0) ? r : c0 * base[c] + c1 * r;
    }
    __syncthreads();
  }
}

}  // namespace

template <class T>
void taped_levelset(const T* src, const T* base, T* out, const T* u, const T* v, const T* w, const Lay& L,
                    const Lay& Lu, const Lay& Lv, const Lay& Lw, double dx, double eps, double dt, double c0, double c1,
                    cudaStream_t s) {
  const StagedGrid g = staged_grid(L);
  k_taped_levelset<T><<<g.grid, dim3(kTX, kTY, 1), 0, s>>>(src, base, out, u, v, w, L, Lu, Lv, Lw, T(1.0 / dx),
                                                           T(eps), T(dt), T(c0), T(c1), g.kchunk);
}

template <class T>
void taped_mac(const T* comp, T* out, const T* u, const T* v, const T* w, const Lay& Lc, const Lay& Lu, const Lay& Lv,
               const Lay& Lw, int axis, double dx, double eps, double dt, cudaStream_t s) {
  const StagedGrid g = staged_grid(Lc);
  k_taped_mac<T><<<g.grid, dim3(kTX, kTY, 1), 0, s>>>(comp, out, u, v, w, Lc, Lu, Lv, Lw, axis, T(1.0 / dx), T(eps),
                                                      T(dt), g.kchunk);
}

template <class T>
void taped_sussman(const T* src, const T* sgn, const T* base, T* out, const Lay& L, double dx, double eps, double dtau,
                   double c0, double c1, int typo, cudaStream_t s) {
  const StagedGrid g = staged_grid(L);
  k_taped_sussman<T><<<g.grid, dim3(kTX, kTY, 1), 0, s>>>(src, sgn, base, out, L, T(1.0 / dx), T(eps), T(dtau), T(c0),
                                                          T(c1), typo, g.kchunk);
}

#define FS_TAPED(T)                                                                                                 \
  template void taped_levelset<T>(const T*, const T*, T*, const T*, const T*, const T*, const Lay&, const Lay&,     \
                                  const Lay&, const Lay&, double, double, double, double, double, cudaStream_t);    \
  template void taped_mac<T>(const T*, T*, const T*, const T*, const T*, const Lay&, const Lay&, const Lay&,        \
                             const Lay&, int, double, double, double, cudaStream_t);                                \
  template void taped_sussman<T>(const T*, const T*, const T*, T*, const Lay&, double, double, double, double,      \
                                 double, int, cudaStream_t);
FS_TAPED(float)
FS_TAPED(double)

}  // namespace fsb
