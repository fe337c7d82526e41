// Level-set and velocity stencil kernels: ghost fills, WENO5 advection
// (ADVECTION_METHOD_3D.h:42-279), Sussman reinitialisation
// (ADVECTION_METHOD_3D.h:745-1637) and the RK stage combiners
// (EULERIAN_FLUID_SOLVER_3D.h:886-1109), templated on the storage/arithmetic
// type (double for the FP64 path, float for FP32_REFINE).
//
// The seven-point stencil kernels (WENO5 level set, WENO5 and ENO3 MAC
// components, Sussman) take one column of a z chunk per thread and march up
// it.  The seven samples along z slide through registers (one new load per
// cell); the x and y samples are read at fixed offsets and hit L1, where the
// neighbouring threads of the block have just read them.  A shared-memory
// ring of seven planes, as these kernels used before, spends more on staging
// the planes, two barriers per plane and the ring's index arithmetic than it
// saves: they are bound by instruction issue, not by HBM (12 to 20 bytes per
// cell in FP32).  What cut the time is fewer instructions per cell:
//   - the two one-sided WENO5 derivatives share their differences, second
//     differences and the squares of these; an advection, which uses only the
//     upwind side, evaluates only that one;
//   - each side is its middle difference plus a weighted correction,
//     D = r3 + (b1 v1 + b2 v2 + b3 v3)/(b1 + b2 + b3), b_k = d_k prod_{j!=k}
//     q_j, q = (eps + IS)^2: algebraically the reference's
//     sum (d_k/q_k) u_k / sum (d_k/q_k) with one reciprocal per side, which in
//     FP32 may be the hardware's (1 ulp, of a term that only corrects r3);
//   - level-set ghosts are the linear extrapolation the ghost fill would
//     store, formed in registers by the threads next to a wall, so no fill
//     precedes the kernel (and the first Sussman step writes the sign field
//     it is the first to need).
// Measured (B200), before -> after, per launch with its ghost fill: Sussman
// step 256^3 FP32 516 -> 256 us, 33 x 47 x 29 FP64 17.8 -> 4.3 us; level set
// 256^3 FP32 533 -> 239 us; WENO5, three components, 200 x 136 x 267 FP32 855 ->
// 305 us; ENO3, three components, 65 x 97 x 41 FP64 76 -> 19 us.
#include <algorithm>

#include "fs_kernels.h"

namespace fsb {

// ---------------------------------------------------------------------------
// ghost fills
// ---------------------------------------------------------------------------

// m-th ghost layer (m = 1..3) of the outward linear extrapolation
// ghost(-m) = 2 ghost(-m+1) - ghost(-m+2), evaluated recursively from the
// two boundary values f0 (on the wall) and f1 (one inside) as the reference
// does (FIELD_STRUCTURE_3D.h:1776-1895).
template <class T>
__device__ __forceinline__ T extrap_layer(T f0, T f1, int m) {
  T a = f1, b = f0;  // (layer m-2, layer m-1)
  for (int q = 0; q < m; ++q) {
    T c = T(2) * b - a;
    a = b;
    b = c;
  }
  return b;
}

template <class T>
struct ExtrapField {
  const T* f;
  Lay L;
  // value at (i, j, k) with i, j, k possibly in the ghost ring: extend x
  // first, then y, then z (dimension by dimension).
  __device__ T x_ext(int i, int j, int k) const {
    if (i < 0) return extrap_layer(f[L.at(0, j, k)], f[L.at(1, j, k)], -i);
    if (i >= L.nx) return extrap_layer(f[L.at(L.nx - 1, j, k)], f[L.at(L.nx - 2, j, k)], i - L.nx + 1);
    return f[L.at(i, j, k)];
  }
  __device__ T y_ext(int i, int j, int k) const {
    if (j < 0) return extrap_layer(x_ext(i, 0, k), x_ext(i, 1, k), -j);
    if (j >= L.ny) return extrap_layer(x_ext(i, L.ny - 1, k), x_ext(i, L.ny - 2, k), j - L.ny + 1);
    return x_ext(i, j, k);
  }
  __device__ T z_ext(int i, int j, int k) const {
    if (k < 0) return extrap_layer(y_ext(i, j, 0), y_ext(i, j, 1), -k);
    if (k >= L.nz) return extrap_layer(y_ext(i, j, L.nz - 1), y_ext(i, j, L.nz - 2), k - L.nz + 1);
    return y_ext(i, j, k);
  }
};

// Decode a flat index over the ghost shell: the z slabs (full padded x, y),
// then the y slabs (interior z, full padded x), then the x slabs (interior
// y, z).  Returns false past the end.
__device__ __forceinline__ bool shell_coord(const Lay& L, int64_t t, int& i, int& j, int& k) {
  const int px = L.nx + 2 * GH, py = L.py;  // logical extents: the alignment columns are not part of the shell
  const int64_t nzs = (int64_t)2 * GH * px * py;
  if (t < nzs) {
    const int64_t s = t / ((int64_t)px * py);
    const int64_t r = t % ((int64_t)px * py);
    k = s < GH ? (int)(s - GH) : (int)(L.nz + (s - GH));
    j = (int)(r / px) - GH;
    i = (int)(r % px) - GH;
    return true;
  }
  t -= nzs;
  const int64_t nys = (int64_t)2 * GH * px * L.nz;
  if (t < nys) {
    const int64_t s = t / ((int64_t)px * L.nz);
    const int64_t r = t % ((int64_t)px * L.nz);
    j = s < GH ? (int)(s - GH) : (int)(L.ny + (s - GH));
    k = (int)(r / px);
    i = (int)(r % px) - GH;
    return true;
  }
  t -= nys;
  const int64_t nxs = (int64_t)2 * GH * L.ny * L.nz;
  if (t < nxs) {
    const int64_t s = t / ((int64_t)L.ny * L.nz);
    const int64_t r = t % ((int64_t)L.ny * L.nz);
    i = s < GH ? (int)(s - GH) : (int)(L.nx + (s - GH));
    k = (int)(r / L.ny);
    j = (int)(r % L.ny);
    return true;
  }
  return false;
}

inline int64_t shell_count(const Lay& L) {
  const int64_t wx = L.nx + 2 * GH;
  return (int64_t)2 * GH * wx * L.py + (int64_t)2 * GH * wx * L.nz + (int64_t)2 * GH * L.ny * L.nz;
}

template <class T>
__global__ void k_fill_extrap(T* f, Lay L) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int i, j, k;
  if (!shell_coord(L, t, i, j, k)) return;
  ExtrapField<T> e{f, L};
  f[L.at(i, j, k)] = e.z_ext(i, j, k);
}

template <class T>
void fill_extrap(T* f, const Lay& L, cudaStream_t s) {
  const int64_t n = shell_count(L);
  k_fill_extrap<T><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(f, L);
}

// ---------------------------------------------------------------------------
// WENO5
// ---------------------------------------------------------------------------

__device__ __forceinline__ float reciprocal(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ double reciprocal(double x) { return 1.0 / x; }

// One side from its middle difference r3, its differences' differences e1 ..
// e4 (e_k = r_{k+1} - r_k) and the scaled squares T_k = eps + 13/12 (e_{k+1}
// - e_k)^2 of its three substencils.
template <class T>
__device__ __forceinline__ T weno_from(T r3, T e1, T e2, T e3, T e4, T T1, T T2, T T3) {
  const T g1 = T(3) * e2 - e1, g2 = e2 + e3, g3 = T(3) * e3 - e4;
  const T s1 = T1 + (T(0.25) * g1) * g1, s2 = T2 + (T(0.25) * g2) * g2, s3 = T3 + (T(0.25) * g3) * g3;
  const T q1 = s1 * s1, q2 = s2 * s2, q3 = s3 * s3;
  const T b1 = T(0.1) * (q2 * q3), b2 = T(0.6) * (q1 * q3), b3 = T(0.3) * (q1 * q2);
  // six times the substencil values less r3
  const T v1 = T(5) * e2 - T(2) * e1, v2 = T(2) * e3 + e2, v3 = T(4) * e3 - e4;
  const T num = (b1 * v1 + b2 * v2) + b3 * v3;
  return r3 + (num * T(1.0 / 6.0)) * reciprocal((b1 + b2) + b3);
}

// D- and D+ from the 7 samples v[0..6] = f[-3..3] along one axis.
template <class T>
__device__ __forceinline__ void weno_pair7(const T v[7], T inv_h, T eps, T& dm, T& dp) {
  const T d1 = inv_h * (v[1] - v[0]), d2 = inv_h * (v[2] - v[1]), d3 = inv_h * (v[3] - v[2]),
          d4 = inv_h * (v[4] - v[3]), d5 = inv_h * (v[5] - v[4]), d6 = inv_h * (v[6] - v[5]);
  const T e1 = d2 - d1, e2 = d3 - d2, e3 = d4 - d3, e4 = d5 - d4, e5 = d6 - d5;
  const T c1312 = T(13.0 / 12.0);
  const T t1 = e2 - e1, t2 = e3 - e2, t3 = e4 - e3, t4 = e5 - e4;
  const T T1 = eps + (c1312 * t1) * t1, T2 = eps + (c1312 * t2) * t2, T3 = eps + (c1312 * t3) * t3,
          T4 = eps + (c1312 * t4) * t4;
  dm = weno_from(d3, e1, e2, e3, e4, T1, T2, T3);
  dp = weno_from(d4, -e5, -e4, -e3, -e2, T4, T3, T2);
}

// The upwind one of the two: D- for a positive velocity, else D+, which is
// the same function of the differences in reverse order.
template <class T>
__device__ __forceinline__ T weno_upwind7(const T v[7], T inv_h, T eps, bool minus) {
  const T d1 = inv_h * (v[1] - v[0]), d2 = inv_h * (v[2] - v[1]), d3 = inv_h * (v[3] - v[2]),
          d4 = inv_h * (v[4] - v[3]), d5 = inv_h * (v[5] - v[4]), d6 = inv_h * (v[6] - v[5]);
  const T r1 = minus ? d1 : d6, r2 = minus ? d2 : d5, r3 = minus ? d3 : d4, r4 = minus ? d4 : d3,
          r5 = minus ? d5 : d2;
  const T e1 = r2 - r1, e2 = r3 - r2, e3 = r4 - r3, e4 = r5 - r4;
  const T c1312 = T(13.0 / 12.0);
  const T t1 = e2 - e1, t2 = e3 - e2, t3 = e4 - e3;
  return weno_from(r3, e1, e2, e3, e4, eps + (c1312 * t1) * t1, eps + (c1312 * t2) * t2, eps + (c1312 * t3) * t3);
}

// ---------------------------------------------------------------------------
// columns of the stencil kernels
// ---------------------------------------------------------------------------
constexpr int kTX = 32, kTY = 8, kColThreads = kTX * kTY;

// Thread -> column (i, j) of a layout: 32 x 8 tiles, or, where those would
// leave more than an eighth of their threads without a column (rows a little
// longer than a multiple of 32, small ragged boxes), 256 consecutive columns
// of the plane.  Tiles read fewer rows per block, so they are the rule.
struct ColumnGrid {
  dim3 grid;
  int kchunk, flat;
};
inline ColumnGrid column_grid(const Lay& L) {
  static int sms = 0;
  if (sms <= 0) {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sms = n;
  }
  const int tx = (L.nx + kTX - 1) / kTX, ty = (L.ny + kTY - 1) / kTY;
  const int64_t cols = (int64_t)L.nx * L.ny;
  ColumnGrid g;
  g.flat = (int64_t)tx * ty * kColThreads * 7 > cols * 8 ? 1 : 0;
  const int bx = g.flat ? (int)((cols + kColThreads - 1) / kColThreads) : tx, by = g.flat ? 1 : ty;
  // about 16 blocks per SM: several waves, so that the last one is short; a
  // chunk's start costs its six extra z samples only
  const int64_t want = (int64_t)16 * sms;
  const int chunks = (int)std::max<int64_t>(1, std::min<int64_t>(L.nz, (want + (int64_t)bx * by - 1) / ((int64_t)bx * by)));
  g.kchunk = (L.nz + chunks - 1) / chunks;
  g.grid = dim3(bx, by, (L.nz + g.kchunk - 1) / g.kchunk);
  return g;
}

__device__ __forceinline__ bool column_of(const Lay& L, int flat, int& i, int& j) {
  if (flat) {
    const unsigned t = blockIdx.x * (unsigned)kColThreads + threadIdx.x;  // at most 4097^2 columns
    j = (int)(t / (unsigned)L.nx);
    i = (int)(t - (unsigned)j * (unsigned)L.nx);
    return j < L.ny;
  }
  i = blockIdx.x * kTX + (threadIdx.x & (kTX - 1));
  j = blockIdx.y * kTY + threadIdx.x / kTX;
  return i < L.nx && j < L.ny;
}

// Samples outside [0, n) replaced by the recursion of extrap_layer.
template <class T>
__device__ __forceinline__ void extrapolate7(T v[7], int e, int n) {
#pragma unroll
  for (int m = 1; m <= 3; ++m) {
    if (e - m < 0) v[3 - m] = T(2) * v[4 - m] - v[5 - m];
    if (e + m >= n) v[3 + m] = T(2) * v[2 + m] - v[1 + m];
  }
}

// The seven samples around c along one axis (stride st, coordinate e of n).
template <class T>
__device__ __forceinline__ void samples7(T v[7], const T* __restrict__ f, int64_t c, int64_t st, T centre, int e, int n,
                                         bool extrapolate) {
#pragma unroll
  for (int m = 1; m <= 3; ++m) {
    v[3 - m] = f[c - m * st];
    v[3 + m] = f[c + m * st];
  }
  v[3] = centre;
  if (extrapolate && (e < 3 || e >= n - 3)) extrapolate7(v, e, n);
}

// The sliding window along z: advance to the next plane.  `next` is
// f[c + 4 slab] of the plane just done, loaded early; past the box it is
// extrapolated instead.
template <class T>
__device__ __forceinline__ void slide7(T v[7], T next, int k, int nz, bool extrapolate) {
  const T n = extrapolate && k + 4 >= nz ? T(2) * v[6] - v[5] : next;
#pragma unroll
  for (int m = 0; m < 6; ++m) v[m] = v[m + 1];
  v[6] = n;
}

// out = c0*base + c1*(src - dt*(u.grad src)), the level-set update at cell
// centres; u, v, w are the MAC faces (zero ghosts).  With c0 == 0 the
// combination is skipped and out is the forward-Euler value.
template <class T>
__global__ void __launch_bounds__(kColThreads) k_weno5_levelset(const T* __restrict__ src, const T* __restrict__ base,
                                                           T* __restrict__ out, const T* __restrict__ u,
                                                           const T* __restrict__ v, const T* __restrict__ w, Lay L,
                                                           Lay Lu, Lay Lv, Lay Lw, T inv_h, T eps, T dt, T c0, T c1,
                                                           int kchunk, int flat, PipeGeom pipe) {
  int i, j;
  if (!column_of(L, flat, i, j)) return;
  const int k0 = blockIdx.z * kchunk, k1 = min(L.nz, k0 + kchunk);
  const bool ex = !pipe.on;  // the pipe's ghosts are periodic, filled by the caller
  int64_t c = L.at(i, j, k0), cu = Lu.at(i, j, k0), cv = Lv.at(i, j, k0), cw = Lw.at(i, j, k0);
  T vx[7], vy[7], vz[7];
  samples7(vz, src, c, L.slab, src[c], k0, L.nz, ex);
  for (int k = k0; k < k1; ++k, c += L.slab, cu += Lu.slab, cv += Lv.slab, cw += Lw.slab) {
    const T next = k + 1 < k1 ? src[c + 4 * L.slab] : T(0);
    samples7(vx, src, c, 1, vz[3], i, L.nx, ex);
    samples7(vy, src, c, L.px, vz[3], j, L.ny, ex);
    const T uc = (u[cu + 1] + u[cu]) * T(0.5);
    const T vc = (v[cv + Lv.px] + v[cv]) * T(0.5);
    const T wc = (w[cw + Lw.slab] + w[cw]) * T(0.5);
    const T dx = weno_upwind7(vx, inv_h, eps, uc > T(0));
    const T dy = weno_upwind7(vy, inv_h, eps, vc > T(0));
    const T dz = weno_upwind7(vz, inv_h, eps, wc > T(0));
    T fe = vz[3] - dt * ((uc * dx + vc * dy) + wc * dz);
    // pipe mode: cells outside the pipe keep their value
    // (ADVECTION_METHOD_3D.h:293-296)
    if (pipe.on && pipe_wall_distance(pipe, 0, i, k) > 0.0) fe = vz[3];
    out[c] = c0 == T(0) ? fe : c0 * base[c] + c1 * fe;
    slide7(vz, next, k, L.nz, ex);
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

// ---------------------------------------------------------------------------
// ENO3 (ADVECTION_METHOD_3D.h:1639-1934)
// ---------------------------------------------------------------------------

// D- and D+ along a stride from the 7 samples f[-3..3]: divided differences
// d1 (scaled 1/dx), d2 (1/(2dx)), d3 ((1/dx)/3); each side takes the stencil
// with the smaller |d2|, then the smaller |d3|.
template <class T>
__device__ __forceinline__ void eno3_pair7(const T v[7], T h, T inv, T o2, T o3, T& dm, T& dp) {
  T d1[6], d2[5], d3[4];  // d1[q]: samples q+1 - q (s = q-3); d2[q] from d1[q+1], d1[q]; d3[q] from d2[q+1], d2[q]
#pragma unroll
  for (int q = 0; q < 6; ++q) d1[q] = inv * (v[q + 1] - v[q]);
#pragma unroll
  for (int q = 0; q < 5; ++q) d2[q] = o2 * (d1[q + 1] - d1[q]);
#pragma unroll
  for (int q = 0; q < 4; ++q) d3[q] = o3 * (d2[q + 1] - d2[q]);
  // in the reference's names: d1_n1 = d1[2], d1_0 = d1[3]; d2_n1 = d2[1],
  // d2_0 = d2[2], d2_p1 = d2[3]; d3_n2 = d3[0], d3_n1 = d3[1], d3_0 = d3[2], d3_p1 = d3[3]
  const T two = T(2);
  if (fabs(d2[1]) <= fabs(d2[2])) {
    dm = fabs(d3[0]) <= fabs(d3[1]) ? (d1[2] + d2[1] * h) + two * d3[0] * h * h : (d1[2] + d2[1] * h) + two * d3[1] * h * h;
  } else {
    dm = fabs(d3[1]) <= fabs(d3[2]) ? (d1[2] + d2[2] * h) - d3[1] * h * h : (d1[2] + d2[2] * h) - d3[2] * h * h;
  }
  if (fabs(d2[2]) <= fabs(d2[3])) {
    dp = fabs(d3[1]) <= fabs(d3[2]) ? (d1[3] - d2[2] * h) - d3[1] * h * h : (d1[3] - d2[2] * h) - d3[2] * h * h;
  } else {
    dp = fabs(d3[2]) <= fabs(d3[3]) ? (d1[3] - d2[3] * h) + two * d3[2] * h * h : (d1[3] - d2[3] * h) + two * d3[3] * h * h;
  }
}

// MAC self-advection of the three components, WENO5 or ENO3 (the reference's
// use_3rd_eno_v, ADVECTION_3D.h:323-325), on every face (wall faces included,
// as the reference's loop covers the whole face grid).  One launch for the
// three: blockIdx.z holds the component and the z chunk, so that a small box
// fills three times as many SMs (65 x 97 x 41 FP64 ENO3: 3 x 11.4 us -> 19.2 us).
// In a step the kernel also does what follows the advection there: add[a]
// (dt g_a) on the faces off the component's walls and, with zero_walls, no
// penetration on them (one pass per component each before).
template <class T>
struct MacFields {
  const T* in[3];
  T* out[3];
  Lay L[3];
  T add[3];
  int zero_walls, chunks;
};

template <class T, bool ENO, int axis>
__device__ __forceinline__ void mac_column(const MacFields<T>& A, int i, int j, int k0, int k1, T h, T inv_h, T eps,
                                           T dt) {
  const Lay& Lc = A.L[axis];
  const T* __restrict__ comp = A.in[axis];
  T* __restrict__ out = A.out[axis];
  const T add = A.add[axis];
  const T o2 = T(0.5) / h, o3 = inv_h * T(1) / T(3);
  int64_t c = Lc.at(i, j, k0);
  T vx[7], vy[7], vz[7];
  samples7(vz, comp, c, Lc.slab, comp[c], k0, Lc.nz, false);
  for (int k = k0; k < k1; ++k, c += Lc.slab) {
    const T next = k + 1 < k1 ? comp[c + 4 * Lc.slab] : T(0);
    T uvel, vvel, wvel;
    mac_velocity(A.in[0], A.in[1], A.in[2], A.L[0], A.L[1], A.L[2], axis, i, j, k, uvel, vvel, wvel);
    samples7(vx, comp, c, 1, vz[3], i, Lc.nx, false);
    samples7(vy, comp, c, Lc.px, vz[3], j, Lc.ny, false);
    T dx, dy, dz;
    if (ENO) {
      T dm, dp;
      eno3_pair7(vx, h, inv_h, o2, o3, dm, dp);
      dx = uvel > T(0) ? dm : dp;
      eno3_pair7(vy, h, inv_h, o2, o3, dm, dp);
      dy = vvel > T(0) ? dm : dp;
      eno3_pair7(vz, h, inv_h, o2, o3, dm, dp);
      dz = wvel > T(0) ? dm : dp;
    } else {
      dx = weno_upwind7(vx, inv_h, eps, uvel > T(0));
      dy = weno_upwind7(vy, inv_h, eps, vvel > T(0));
      dz = weno_upwind7(vz, inv_h, eps, wvel > T(0));
    }
    T r = vz[3] - dt * ((uvel * dx + vvel * dy) + wvel * dz);
    const int e = axis == 0 ? i : (axis == 1 ? j : k), n = axis == 0 ? Lc.nx : (axis == 1 ? Lc.ny : Lc.nz);
    if (e > 0 && e < n - 1) {
      if (add != T(0)) r += add;
    } else if (A.zero_walls) {
      r = T(0);
    }
    out[c] = r;
    slide7(vz, next, k, Lc.nz, false);
  }
}

template <class T, bool ENO>
__global__ void __launch_bounds__(kColThreads) k_mac(const __grid_constant__ MacFields<T> A, T h, T inv_h, T eps, T dt,
                                                     int kchunk, int flat) {
  const int axis = blockIdx.z / A.chunks;
  int i, j;
  if (!column_of(A.L[axis], flat, i, j)) return;
  const int k0 = (blockIdx.z - axis * A.chunks) * kchunk, k1 = min(A.L[axis].nz, k0 + kchunk);
  if (k0 >= k1) return;
  if (axis == 0) mac_column<T, ENO, 0>(A, i, j, k0, k1, h, inv_h, eps, dt);
  else if (axis == 1) mac_column<T, ENO, 1>(A, i, j, k0, k1, h, inv_h, eps, dt);
  else mac_column<T, ENO, 2>(A, i, j, k0, k1, h, inv_h, eps, dt);
}

// The vertical pipe's ENO3 self-advection of component `axis`
// (ADVECTION_METHOD_3D.h:1935-2240): faces inside the pipe and off the
// fixed centre line take the ENO3 upwind update in place, the x and z
// derivatives from the guarded copies gx, gz, the y derivative from the
// masked periodic copy gen, the advecting velocities from the masked
// periodic copies ug, vg, wg; the other faces keep their value.  One thread
// per face: the pipe grids are small and the three stencil sources differ.
template <class T>
__global__ void k_eno3_pipe(T* comp, const T* __restrict__ gen, const T* __restrict__ gx, const T* __restrict__ gz,
                            const T* __restrict__ ug, const T* __restrict__ vg, const T* __restrict__ wg, Lay Lf,
                            Lay Lu, Lay Lv, Lay Lw, int axis, PipeGeom G, T h, T dt, int fi0, int fi1, int fk0,
                            int fk1) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= Lf.nx || j >= Lf.ny || k >= Lf.nz) return;
  if ((i == fi0 || i == fi1) && (k == fk0 || k == fk1)) return;  // the fixed centre line
  if (!(pipe_wall_distance(G, 1 + axis, i, k) < 0.0)) return;
  const T inv = T(1) / h, o2 = T(0.5) / h, o3 = inv * T(1) / T(3);
  T vx[7], vy[7], vz[7];
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    vx[q] = gx[Lf.at(i + q - 3, j, k)];
    vy[q] = gen[Lf.at(i, j + q - 3, k)];
    vz[q] = gz[Lf.at(i, j, k + q - 3)];
  }
  T uvel, vvel, wvel;
  mac_velocity(ug, vg, wg, Lu, Lv, Lw, axis, i, j, k, uvel, vvel, wvel);
  T dxm, dxp, dym, dyp, dzm, dzp;
  eno3_pair7(vx, h, inv, o2, o3, dxm, dxp);
  eno3_pair7(vy, h, inv, o2, o3, dym, dyp);
  eno3_pair7(vz, h, inv, o2, o3, dzm, dzp);
  const int64_t f = Lf.at(i, j, k);
  comp[f] = comp[f] - dt * ((uvel * (uvel > T(0) ? dxm : dxp) + vvel * (vvel > T(0) ? dym : dyp)) +
                            wvel * (wvel > T(0) ? dzm : dzp));
}

// ---------------------------------------------------------------------------
// Sussman reinitialisation
// ---------------------------------------------------------------------------

template <class T>
__global__ void k_sign(const T* __restrict__ phi, T* __restrict__ s, Lay L, T dx) {
  FS_IJK(L);
  const int64_t c = L.at(i, j, k);
  const T p = phi[c];
  s[c] = p / sqrt(p * p + dx * dx);
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
// first: the block's first step, whose src is the field S comes from: S is
// formed here and stored in sgn for the steps that follow.
template <class T>
__global__ void __launch_bounds__(kColThreads) k_sussman(const T* __restrict__ src, T* __restrict__ sgn,
                                                    const T* __restrict__ base, T* __restrict__ out, Lay L, T dx,
                                                    T inv_h, T eps, T dtau, T c0, T c1, int typo, int first,
                                                    int extrapolate, int kchunk, int flat) {
  int i, j;
  if (!column_of(L, flat, i, j)) return;
  const int k0 = blockIdx.z * kchunk, k1 = min(L.nz, k0 + kchunk);
  const bool ex = extrapolate != 0;
  int64_t c = L.at(i, j, k0);
  T vx[7], vy[7], vz[7];
  samples7(vz, src, c, L.slab, src[c], k0, L.nz, ex);
  for (int k = k0; k < k1; ++k, c += L.slab) {
    const T next = k + 1 < k1 ? src[c + 4 * L.slab] : T(0);
    T s;
    if (first) {
      s = vz[3] / sqrt(vz[3] * vz[3] + dx * dx);
      sgn[c] = s;
    } else {
      s = sgn[c];
    }
    samples7(vx, src, c, 1, vz[3], i, L.nx, ex);
    samples7(vy, src, c, L.px, vz[3], j, L.ny, ex);
    T dxm, dxp, dym, dyp, dzm, dzp;
    weno_pair7(vx, inv_h, eps, dxm, dxp);
    weno_pair7(vy, inv_h, eps, dym, dyp);
    weno_pair7(vz, inv_h, eps, dzm, dzp);
    int cx, cy, cz;
    bool shx, shy, shz;
    const T gx = godunov(s, dxm, dxp, cx, shx);
    const T gy = godunov(s, dym, dyp, cy, shy);
    const T gz = godunov(s, dzm, dzp, cz, shz);
    T mag = sqrt((gx * gx + gy * gy) + gz * gz) - T(1);
    if (typo && shx && shy && cy == 1 && cz == 2) mag = (sqrt(gx * gx) + gy * gy) - T(1);
    T r = vz[3] - dtau * s * mag;
    if (s * r < T(0)) {
      if (s < T(0)) r = -eps;
      if (s > T(0)) r = eps;
    }
    out[c] = c0 == T(0) ? r : c0 * base[c] + c1 * r;
    slide7(vz, next, k, L.nz, ex);
  }
}

// ---------------------------------------------------------------------------
// elementwise helpers
// ---------------------------------------------------------------------------

// out = a*x + b*y over the interior of layout L.
template <class T>
__global__ void k_axpby(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ y, T a, T b, Lay L) {
  FS_IJK(L);
  const int64_t c = L.at(i, j, k);
  out[c] = a * x[c] + b * y[c];
}

// Add a constant (gravity*dt) to every interior face except the two wall
// planes normal to the component (which hold the no-penetration zero).
template <class T>
__global__ void k_add_const_interior_faces(T* __restrict__ f, Lay L, int axis, T value, int skip_walls) {
  FS_IJK(L);
  if (skip_walls) {
    const int e = axis == 0 ? i : (axis == 1 ? j : k);
    const int n = axis == 0 ? L.nx : (axis == 1 ? L.ny : L.nz);
    if (e == 0 || e == n - 1) return;
  }
  f[L.at(i, j, k)] += value;
}

// Zero the two wall planes normal to a face component.
template <class T>
__global__ void k_zero_walls(T* __restrict__ f, Lay L, int axis) {
  FS_IJK(L);
  const int e = axis == 0 ? i : (axis == 1 ? j : k);
  const int n = axis == 0 ? L.nx : (axis == 1 ? L.ny : L.nz);
  if (e == 0 || e == n - 1) f[L.at(i, j, k)] = T(0);
}

// ---------------------------------------------------------------------------
// host wrappers
// ---------------------------------------------------------------------------

template <class T>
void weno5_levelset(const T* src, const T* base, T* out, const T* u, const T* v, const T* w, const Lay& L,
                    const Lay& Lu, const Lay& Lv, const Lay& Lw, double dx, double eps, double dt, double c0, double c1,
                    cudaStream_t s, const PipeGeom* pipe) {
  const ColumnGrid g = column_grid(L);
  PipeGeom none{};
  k_weno5_levelset<T><<<g.grid, kColThreads, 0, s>>>(src, base, out, u, v, w, L, Lu, Lv, Lw, T(1.0 / dx), T(eps),
                                                     T(dt), T(c0), T(c1), g.kchunk, g.flat, pipe ? *pipe : none);
}

template <class T>
void mac_advect(const T* const in[3], T* const out[3], const Lay* const L[3], bool eno, double dx, double eps, double dt,
                const double add[3], int zero_walls, cudaStream_t s) {
  MacFields<T> A;
  ColumnGrid g = column_grid(*L[0]);
  unsigned gx = 0, gy = 0;
  int nz = 0;
  for (int a = 0; a < 3; ++a) {
    A.in[a] = in[a];
    A.out[a] = out[a];
    A.L[a] = *L[a];
    A.add[a] = T(add[a]);
    nz = std::max(nz, L[a]->nz);
    const int64_t cols = (int64_t)L[a]->nx * L[a]->ny;
    gx = std::max(gx, g.flat ? (unsigned)((cols + kColThreads - 1) / kColThreads) : (unsigned)((L[a]->nx + kTX - 1) / kTX));
    gy = std::max(gy, g.flat ? 1u : (unsigned)((L[a]->ny + kTY - 1) / kTY));
  }
  g.kchunk = std::min(nz, 3 * g.kchunk);  // three components share the GPU
  A.zero_walls = zero_walls;
  A.chunks = (nz + g.kchunk - 1) / g.kchunk;
  auto* kernel = eno ? k_mac<T, true> : k_mac<T, false>;
  kernel<<<dim3(gx, gy, 3 * A.chunks), kColThreads, 0, s>>>(A, T(dx), eno ? T(1) / T(dx) : T(1.0 / dx), T(eps), T(dt),
                                                            g.kchunk, g.flat);
}

template <class T>
void eno3_pipe(T* comp, const T* gen, const T* gx, const T* gz, const T* ug, const T* vg, const T* wg, const Lay& Lc,
               const Lay& Lu, const Lay& Lv, const Lay& Lw, int axis, const PipeGeom& G, double dx, double dt,
               cudaStream_t s) {
  const Lay& Lf = axis == 0 ? Lu : axis == 1 ? Lv : Lw;
  // the faces Solve_Velocity holds fixed (ADVECTION_3D.h:246-275): the
  // integer halves of the face grid's last indices
  int fi0, fi1, fk0, fk1;
  if (axis == 0) { fi0 = (Lf.nx - 1) / 2; fi1 = fi0 + 1; fk0 = fk1 = (Lc.nz - 1) / 2; }
  else if (axis == 1) { fi0 = fi1 = (Lc.nx - 1) / 2; fk0 = fk1 = (Lc.nz - 1) / 2; }
  else { fi0 = fi1 = (Lc.nx - 1) / 2; fk0 = (Lf.nz - 1) / 2; fk1 = fk0 + 1; }
  Launch3 g = launch3(Lf.nx, Lf.ny, Lf.nz);
  k_eno3_pipe<T><<<g.grid, g.block, 0, s>>>(comp, gen, gx, gz, ug, vg, wg, Lf, Lu, Lv, Lw, axis, G, T(dx), T(dt), fi0,
                                            fi1, fk0, fk1);
}

template <class T>
void sign_function(const T* phi, T* sgn, const Lay& L, double dx, cudaStream_t s) {
  Launch3 g = launch3(L.nx, L.ny, L.nz);
  k_sign<T><<<g.grid, g.block, 0, s>>>(phi, sgn, L, T(dx));
}

template <class T>
void sussman_step(const T* src, T* sgn, const T* base, T* out, const Lay& L, double dx, double eps, double dtau,
                  double c0, double c1, int typo, int first, int extrapolate, cudaStream_t s) {
  const ColumnGrid g = column_grid(L);
  k_sussman<T><<<g.grid, kColThreads, 0, s>>>(src, sgn, base, out, L, T(dx), T(1.0 / dx), T(eps), T(dtau), T(c0),
                                              T(c1), typo, first, extrapolate, g.kchunk, g.flat);
}

template <class T>
void axpby(T* out, const T* x, const T* y, double a, double b, const Lay& L, cudaStream_t s) {
  Launch3 g = launch3(L.nx, L.ny, L.nz);
  k_axpby<T><<<g.grid, g.block, 0, s>>>(out, x, y, T(a), T(b), L);
}

template <class T>
void add_const_faces(T* f, const Lay& L, int axis, double value, int skip_walls, cudaStream_t s) {
  Launch3 g = launch3(L.nx, L.ny, L.nz);
  k_add_const_interior_faces<T><<<g.grid, g.block, 0, s>>>(f, L, axis, T(value), skip_walls);
}

template <class T>
void zero_walls(T* f, const Lay& L, int axis, cudaStream_t s) {
  Launch3 g = launch3(L.nx, L.ny, L.nz);
  k_zero_walls<T><<<g.grid, g.block, 0, s>>>(f, L, axis);
}

#define FS_INST(T)                                                                                                    \
  template void fill_extrap<T>(T*, const Lay&, cudaStream_t);                                                         \
  template void weno5_levelset<T>(const T*, const T*, T*, const T*, const T*, const T*, const Lay&, const Lay&,       \
                                  const Lay&, const Lay&, double, double, double, double, double, cudaStream_t,       \
                                  const PipeGeom*);                                                                   \
  template void mac_advect<T>(const T* const[3], T* const[3], const Lay* const[3], bool, double, double, double,      \
                              const double[3], int, cudaStream_t);                                                    \
  template void eno3_pipe<T>(T*, const T*, const T*, const T*, const T*, const T*, const T*, const Lay&, const Lay&,  \
                             const Lay&, const Lay&, int, const PipeGeom&, double, double, cudaStream_t);             \
  template void sign_function<T>(const T*, T*, const Lay&, double, cudaStream_t);                                    \
  template void sussman_step<T>(const T*, T*, const T*, T*, const Lay&, double, double, double, double, double, int, \
                                int, int, cudaStream_t);                                                                   \
  template void axpby<T>(T*, const T*, const T*, double, double, const Lay&, cudaStream_t);                          \
  template void add_const_faces<T>(T*, const Lay&, int, double, int, cudaStream_t);                                  \
  template void zero_walls<T>(T*, const Lay&, int, cudaStream_t);

FS_INST(float)
FS_INST(double)

}  // namespace fsb
