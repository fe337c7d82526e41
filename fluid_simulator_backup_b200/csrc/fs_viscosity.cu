// Semi-implicit viscosity (VISCOSITY_3D.h:567-990 with the system of
// POISSON_SOLVER_3D.h:3359-3496), one velocity component at a time.
//
// The reference solves (1 + sum c/dx^2) u_f - sum c_arm/dx^2 u_nb = u* +
// dt/rho_f (transpose stress terms), with c = 2 dt mu/rho_f on the two normal
// arms and dt mu/rho_f on the four tangential arms.  Multiplying each row by
// the face density rho_f gives the symmetric positive definite form
//   (rho_f + sum k dt mu_arm/dx^2) u_f - sum k dt mu_arm/dx^2 u_nb = rho_f*rhs
// (k = 2 on the normal arms) with the same solution, which is what the
// conjugate-gradient engine here solves.  Each arm coupling is computed once
// per arm midpoint, so the matrix is exactly symmetric in floating point.
//
// Box boundary: the wall-normal faces of the component are Dirichlet zero
// (no penetration) and velocity ghosts beyond the walls are zero; both enter
// the diagonal through their arm couplings and drop out of the right-hand
// side.  Wall rows become identity rows with zero right-hand side.
#include <algorithm>

#include "fs_kernels.h"

namespace fsb {

__device__ __forceinline__ double heaviside_visc(double phi, double e) {
  // VISCOSITY_3D.h:1234-1253
  const double ooe = 1.0 / e, oop = 1.0 / 3.14159265358979323846;
  if (phi < -e) return 0.0;
  if (phi > e) return 1.0;
  return 0.5 * ((1.0 + phi * ooe) + oop * sin(3.14159265358979323846 * phi * ooe));
}

template <class T>
struct PhiX {  // phi with a one-layer linear extrapolation across the walls
  const T* phi;
  Lay L;
  __device__ double at(int i, int j, int k) const {
    // clamp-and-extrapolate dimension by dimension (one layer)
    int ii = min(max(i, 0), L.nx - 1), jj = min(max(j, 0), L.ny - 1), kk = min(max(k, 0), L.nz - 1);
    auto val = [&](int a, int b, int c) { return (double)phi[L.at(a, b, c)]; };
    auto ex = [&](int a, int b, int c) -> double {
      // extend in x
      if (i < 0) return 2.0 * val(0, b, c) - val(1, b, c);
      if (i >= L.nx) return 2.0 * val(L.nx - 1, b, c) - val(L.nx - 2, b, c);
      return val(a, b, c);
    };
    auto ey = [&](int a, int b, int c) -> double {
      if (j < 0) return 2.0 * ex(a, 0, c) - ex(a, 1, c);
      if (j >= L.ny) return 2.0 * ex(a, L.ny - 1, c) - ex(a, L.ny - 2, c);
      return ex(a, b, c);
    };
    if (k < 0) return 2.0 * ey(ii, jj, 0) - ey(ii, jj, 1);
    if (k >= L.nz) return 2.0 * ey(ii, jj, L.nz - 1) - ey(ii, jj, L.nz - 2);
    return ey(ii, jj, kk);
  }
};

// Face (i,j,k) of component `axis` sits between cell (i,j,k) and the cell
// one step back along the axis.  Its row needs phi at those two cells and at
// their four neighbours across the axis: two cell samples (normal arms), four
// edge averages (tangential arms) and the face average (density).
//
// Where the ten samples all lie beyond the smearing width on one side, every
// Heaviside is 0 or 1 and none is evaluated: the sines are left to the faces
// near the interface.  Samples inside the box are read at fixed offsets; only
// those beyond a wall (the first and last lane of a row, the outer rows and
// planes) go through the extrapolation.  The kernel is then bound by HBM and
// L1 (phi and the velocities read, five arrays written: 36 bytes per face in
// FP32) and instruction issue: inside the box the samples are compared in the
// storage type, so that only the faces near the interface convert them, and
// dt / rho of a phase comes from the host.  Measured, FP32, per component (x, y,
// z): with every sample through the extrapolating accessor and seven Heavisides
// per face 1580, 3045, 2883 us at 256^3, in this form 292, 319, 273 us (128^3:
// 228, 383, 361 and 53, 50, 52).
// The component's axis is a template parameter so that every per-direction
// array below is indexed by compile-time constants (registers, no stack).
template <class T>
__device__ __noinline__ double phi_beyond_wall(const T* phi, const Lay& Lc, int i, int j, int k) {
  return PhiX<T>{phi, Lc}.at(i, j, k);
}

// phi > smear_limit(e) in the storage type only where phi > e
template <class T> __device__ __forceinline__ T smear_limit(double e);
template <> __device__ __forceinline__ double smear_limit<double>(double e) { return e; }
template <> __device__ __forceinline__ float smear_limit<float>(double e) { return __double2float_ru(e); }

template <class T, class V>
struct ViscSystem {
  const T *phi, *u, *v, *w;
  Lay Lc, Lu, Lv, Lw, Lf;
  double inv_h, dt, rn, rp, mn, mp, coef_n, coef_p;
  V *ax, *ay, *az, *diag, *rhs;
};

template <class T, class V, int axis>
__device__ __forceinline__ void visc_face(const ViscSystem<T, V>& A, int i, int j, int k) {
  const Lay &Lc = A.Lc, &Lu = A.Lu, &Lv = A.Lv, &Lw = A.Lw, &Lf = A.Lf;
  const T *__restrict__ phi = A.phi, *__restrict__ u = A.u, *__restrict__ v = A.v, *__restrict__ w = A.w;
  V *__restrict__ ax = A.ax, *__restrict__ ay = A.ay, *__restrict__ az = A.az, *__restrict__ diag = A.diag,
    *__restrict__ rhs = A.rhs;
  const double inv_h = A.inv_h, dt = A.dt, rn = A.rn, rp = A.rp, mn = A.mn, mp = A.mp;
  constexpr int e0 = axis == 0, e1 = axis == 1, e2 = axis == 2;
  const int64_t f = Lf.at(i, j, k);
  const int e_ax = axis == 0 ? i : (axis == 1 ? j : k);
  const int n_ax = axis == 0 ? Lf.nx : (axis == 1 ? Lf.ny : Lf.nz);
  if (e_ax == 0 || e_ax == n_ax - 1) {  // wall rows: identity with zero right-hand side
    ax[f] = (V)0.0;
    ay[f] = (V)0.0;
    az[f] = (V)0.0;
    diag[f] = (V)1.0;
    rhs[f] = (V)0.0;
    return;
  }
  const double e = 1.5 / inv_h;
  const double inv2 = inv_h * inv_h;
  const int64_t c = Lc.at(i, j, k);
  const int sy = Lc.px;
  const int64_t sz = Lc.slab;
  auto at = [&](int di, int dj, int dk) -> double {
    const int a = i + di, b = j + dj, d = k + dk;
    if ((unsigned)a < (unsigned)Lc.nx && (unsigned)b < (unsigned)Lc.ny && (unsigned)d < (unsigned)Lc.nz)
      return (double)phi[c + di + dj * sy + dk * sz];
    return phi_beyond_wall(phi, Lc, a, b, d);
  };
  // the low and the high cell, and per tangential direction their two
  // neighbours (index: the direction; the axis' own entry is unused)
  double lo, hi, lm[3], lp[3], hm[3], hp[3];
  int phase = 0;  // 1: all below -e, 2: all above e, 0: neither (or a NaN)
  if (i > 0 && j > 0 && k > 0 && i < Lc.nx - 1 && j < Lc.ny - 1 && k < Lc.nz - 1) {
    // inside the box: compared in the storage type, converted near the interface only
    const int64_t back = e0 + e1 * sy + e2 * sz;
    T s[10];
    s[0] = phi[c - back];
    s[1] = phi[c];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int d = t ? (axis == 2 ? 1 : 2) : (axis == 0 ? 1 : 0);
      const int64_t step = d == 0 ? 1 : (d == 1 ? (int64_t)sy : sz);
      s[2 + 4 * t] = phi[c - back - step];
      s[3 + 4 * t] = phi[c - back + step];
      s[4 + 4 * t] = phi[c - step];
      s[5 + 4 * t] = phi[c + step];
    }
    const T te = smear_limit<T>(e);
    bool above = true, below = true;
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      above = above && s[q] > te;
      below = below && s[q] < -te;
    }
    phase = above ? 2 : (below ? 1 : 0);
    if (!phase) {
      lo = (double)s[0];
      hi = (double)s[1];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int d = t ? (axis == 2 ? 1 : 2) : (axis == 0 ? 1 : 0);
        lm[d] = (double)s[2 + 4 * t];
        lp[d] = (double)s[3 + 4 * t];
        hm[d] = (double)s[4 + 4 * t];
        hp[d] = (double)s[5 + 4 * t];
      }
    }
  } else {
    lo = at(-e0, -e1, -e2);
    hi = at(0, 0, 0);
    bool above = lo > e && hi > e, below = lo < -e && hi < -e;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (d == axis) continue;
      const int di = d == 0, dj = d == 1, dk = d == 2;
      lm[d] = at(-e0 - di, -e1 - dj, -e2 - dk);
      lp[d] = at(-e0 + di, -e1 + dj, -e2 + dk);
      hm[d] = at(-di, -dj, -dk);
      hp[d] = at(di, dj, dk);
      above = above && lm[d] > e && lp[d] > e && hm[d] > e && hp[d] > e;
      below = below && lm[d] < -e && lp[d] < -e && hm[d] < -e && hp[d] < -e;
    }
    phase = above ? 2 : (below ? 1 : 0);
  }
  // coupling on the low arm along direction d (between this face and the
  // face one step back along d): normal arm -> the low cell, tangential arm
  // -> the edge shared by the four cells {low, high} x {d-1, d}
  double mu_low[3], mu_high[3], low[3], high[3], rho_f;
  double coef;  // dt / rho_f
  if (phase) {
    const double mu = phase == 2 ? mn + (mp - mn) : mn;
    rho_f = phase == 2 ? rn + (rp - rn) : rn;
    coef = phase == 2 ? A.coef_p : A.coef_n;
#pragma unroll
    for (int d = 0; d < 3; ++d) mu_low[d] = mu_high[d] = mu;
  } else {
    auto mu_of = [&](double ph) { return mn + (mp - mn) * heaviside_visc(ph, e); };
    // density at the face from the face-averaged phi
    rho_f = rn + (rp - rn) * heaviside_visc(0.5 * (lo + hi), e);
    coef = dt / rho_f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (d == axis) {
        mu_low[d] = mu_of(lo);
        mu_high[d] = mu_of(hi);
      } else {
        // canonical order: (low cell, d-1), (low cell), (high cell, d-1), (high cell); the
        // edge one step up along d in the same order as the next face sees it
        mu_low[d] = mu_of(0.25 * (((lm[d] + lo) + hm[d]) + hi));
        mu_high[d] = mu_of(0.25 * (((lo + lp[d]) + hi) + hp[d]));
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double kk = d == axis ? 2.0 : 1.0;
    low[d] = kk * dt * mu_low[d] * inv2;
    high[d] = kk * dt * mu_high[d] * inv2;
  }
  // couplings stored at this face couple it with the face one step back;
  // couplings that touch a wall face are zeroed (Dirichlet neighbour)
  ax[f] = (V)(((axis == 0 && i == 1) || i == 0) ? 0.0 : low[0]);
  ay[f] = (V)(((axis == 1 && j == 1) || j == 0) ? 0.0 : low[1]);
  az[f] = (V)(((axis == 2 && k == 1) || k == 0) ? 0.0 : low[2]);
  diag[f] = (V)(rho_f + ((((low[0] + high[0]) + low[1]) + high[1]) + low[2]) + high[2]);
  // explicit transpose terms (VISCOSITY_3D.h:620-630): for each tangential
  // direction t, d/dt( mu_edge * d(vel_t)/d(axis) ) with zero ghosts
  const T* own = axis == 0 ? u : (axis == 1 ? v : w);
  double ex = (double)own[f];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    if (t == axis) continue;
    const T* vt = t == 0 ? u : (t == 1 ? v : w);
    const Lay& Lt = t == 0 ? Lu : (t == 1 ? Lv : Lw);
    const int64_t g = Lt.at(i, j, k);
    const int64_t up = t == 0 ? 1 : (t == 1 ? (int64_t)Lt.px : Lt.slab);
    const int64_t back = axis == 0 ? 1 : (axis == 1 ? (int64_t)Lt.px : Lt.slab);
    // vel_t at (face coords) + e_t and at the same place shifted back along axis
    const double hi_a = (double)vt[g + up], hi_b = (double)vt[g + up - back];
    const double lo_a = (double)vt[g], lo_b = (double)vt[g - back];
    ex = ex + coef * (inv_h * (mu_high[t] * inv_h * (hi_a - hi_b) - mu_low[t] * inv_h * (lo_a - lo_b)));
  }
  rhs[f] = (V)(rho_f * ex);
}

template <class T, class V, int axis>
__global__ void __launch_bounds__(256) k_visc_system(const __grid_constant__ ViscSystem<T, V> A, int chunk) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
  if (i >= A.Lf.nx || j >= A.Lf.ny) return;
  const int k0 = blockIdx.z * chunk, k1 = min(A.Lf.nz, k0 + chunk);
  for (int k = k0; k < k1; ++k) visc_face<T, V, axis>(A, i, j, k);
}

// ---------------------------------------------------------------------------
// The reference's air/water viscosity: the explicit variable-viscosity stress
// update of VISCOSITY_3D::ApplyViscosity (VISCOSITY_3D.h:452-563).  Per face
// of component a: the smeared density of the face-averaged phi, the smeared
// viscosity at the two cells across the face (normal stress, factor 2) and
// at the four edge averages (shear), each sample summed in the reference's
// operand order (VISCOSITY_3D.h:462-470, 502-510, 541-549).
//
// corrected (default): one explicit Euler step of the stress divergence from
// the input velocities into separate output arrays, every transposed-stress
// term on its own edge, wall-normal faces unchanged.  in_place
// (FS_FLAG_VISCOSITY_IN_PLACE): as the reference runs on one thread - x,
// then y, then z, each updated in place in (k, j, i) order, wall faces
// included, with the reference's velocity indices (its y update reads w one
// level low on both z edges, its z update reads u and v on the low edge's
// column/row for the high edge too).  The in-place order is reproduced by
// hyperplanes i + j + k = s: a face depends on its own component only through
// its x-1, y-1, z-1 neighbours (hyperplane s-1, already updated) and x+1,
// y+1, z+1 neighbours (s+1, not yet), so one launch per hyperplane reads
// exactly what the sequential loop reads.
// ---------------------------------------------------------------------------

struct ExplicitViscosity {
  Lay Lc, Lu, Lv, Lw;
  int axis;
  double inv_h, dt, rn, rp, mn, mp;
};

template <class T, bool IN_PLACE>
__device__ __forceinline__ double explicit_visc_face(const ExplicitViscosity& X, const PhiX<T>& P, const T* u,
                                                     const T* v, const T* w, int i, int j, int k) {
  const double e = 1.5 / X.inv_h, inv = X.inv_h;
  auto ph = [&](int di, int dj, int dk) { return P.at(i + di, j + dj, k + dk); };
  double half, hi, lo, e1, e2, e3, e4;
  if (X.axis == 0) {
    half = 0.5 * (ph(-1, 0, 0) + ph(0, 0, 0));
    hi = ph(0, 0, 0);
    lo = ph(-1, 0, 0);
    e1 = 0.25 * (((ph(-1, 0, 0) + ph(0, 0, 0)) + ph(-1, 1, 0)) + ph(0, 1, 0));
    e2 = 0.25 * (((ph(-1, 0, 0) + ph(0, 0, 0)) + ph(-1, -1, 0)) + ph(0, -1, 0));
    e3 = 0.25 * (((ph(-1, 0, 0) + ph(0, 0, 0)) + ph(-1, 0, 1)) + ph(0, 0, 1));
    e4 = 0.25 * (((ph(-1, 0, 0) + ph(0, 0, 0)) + ph(-1, 0, -1)) + ph(0, 0, -1));
  } else if (X.axis == 1) {
    half = 0.5 * (ph(0, -1, 0) + ph(0, 0, 0));
    hi = ph(0, 0, 0);
    lo = ph(0, -1, 0);
    e1 = 0.25 * (((ph(0, -1, 0) + ph(1, -1, 0)) + ph(0, 0, 0)) + ph(1, 0, 0));
    e2 = 0.25 * (((ph(-1, -1, 0) + ph(0, -1, 0)) + ph(-1, 0, 0)) + ph(0, 0, 0));
    e3 = 0.25 * (((ph(0, -1, 1) + ph(0, -1, 0)) + ph(0, 0, 1)) + ph(0, 0, 0));
    e4 = 0.25 * (((ph(0, -1, -1) + ph(0, -1, 0)) + ph(0, 0, -1)) + ph(0, 0, 0));
  } else {
    half = 0.5 * (ph(0, 0, -1) + ph(0, 0, 0));
    hi = ph(0, 0, 0);
    lo = ph(0, 0, -1);
    e1 = 0.25 * (((ph(0, 0, -1) + ph(1, 0, -1)) + ph(0, 0, 0)) + ph(1, 0, 0));
    e2 = 0.25 * (((ph(0, 0, -1) + ph(-1, 0, -1)) + ph(0, 0, 0)) + ph(-1, 0, 0));
    e3 = 0.25 * (((ph(0, 0, -1) + ph(0, 1, -1)) + ph(0, 0, 0)) + ph(0, 1, 0));
    e4 = 0.25 * (((ph(0, 0, -1) + ph(0, -1, -1)) + ph(0, 0, 0)) + ph(0, -1, 0));
  }
  auto mu = [&](double p) { return X.mn + (X.mp - X.mn) * heaviside_visc(p, e); };
  const double rho_h = X.rn + (X.rp - X.rn) * heaviside_visc(half, e);
  const double m0 = mu(hi), m1 = mu(lo), m2 = mu(e1), m3 = mu(e2), m4 = mu(e3), m5 = mu(e4);
  const T* comp[3] = {u, v, w};
  const Lay lay[3] = {X.Lu, X.Lv, X.Lw};
  auto at = [&](int c, int di, int dj, int dk) { return (double)comp[c][lay[c].at(i + di, j + dj, k + dk)]; };
  const double coef = X.dt * (1.0 / rho_h);
  if (X.axis == 0) {
    const double uc = at(0, 0, 0, 0);
    const double first = 2.0 * coef * inv * (m0 * inv * (at(0, 1, 0, 0) - uc) - m1 * inv * (uc - at(0, -1, 0, 0)));
    const double second = coef * inv * (m2 * (inv * (at(0, 0, 1, 0) - uc) + inv * (at(1, 0, 1, 0) - at(1, -1, 1, 0))) -
                                        m3 * (inv * (uc - at(0, 0, -1, 0)) + inv * (at(1, 0, 0, 0) - at(1, -1, 0, 0))));
    const double third = coef * inv * (m4 * (inv * (at(0, 0, 0, 1) - uc) + inv * (at(2, 0, 0, 1) - at(2, -1, 0, 1))) -
                                       m5 * (inv * (uc - at(0, 0, 0, -1)) + inv * (at(2, 0, 0, 0) - at(2, -1, 0, 0))));
    return uc + ((first + second) + third);
  }
  if (X.axis == 1) {
    const double vc = at(1, 0, 0, 0);
    const int zt = IN_PLACE ? 0 : 1;  // the w level of the z+ edge
    const double first = coef * inv * (m2 * (inv * (at(0, 1, 0, 0) - at(0, 1, -1, 0)) + inv * (at(1, 1, 0, 0) - vc)) -
                                       m3 * (inv * (at(0, 0, 0, 0) - at(0, 0, -1, 0)) + inv * (vc - at(1, -1, 0, 0))));
    const double second = 2.0 * coef * inv * (m0 * inv * (at(1, 0, 1, 0) - vc) - m1 * inv * (vc - at(1, 0, -1, 0)));
    const double third =
        coef * inv * (m4 * (inv * (at(1, 0, 0, 1) - vc) + inv * (at(2, 0, 0, zt) - at(2, 0, -1, zt))) -
                      m5 * (inv * (vc - at(1, 0, 0, -1)) + inv * (at(2, 0, 0, zt - 1) - at(2, 0, -1, zt - 1))));
    return vc + ((first + second) + third);
  }
  const double wc = at(2, 0, 0, 0);
  const int xt = IN_PLACE ? 0 : 1, yt = IN_PLACE ? 0 : 1;  // the u column / v row of the high edges
  const double first =
      coef * inv * (m2 * (inv * (at(0, xt, 0, 0) - at(0, xt, 0, -1)) + inv * (at(2, 1, 0, 0) - wc)) -
                    m3 * (inv * (at(0, xt - 1, 0, 0) - at(0, xt - 1, 0, -1)) + inv * (wc - at(2, -1, 0, 0))));
  const double second =
      coef * inv * (m4 * (inv * (at(1, 0, yt, 0) - at(1, 0, yt, -1)) + inv * (at(2, 0, 1, 0) - wc)) -
                    m5 * (inv * (at(1, 0, yt - 1, 0) - at(1, 0, yt - 1, -1)) + inv * (wc - at(2, 0, -1, 0))));
  const double third = 2.0 * coef * inv * (m0 * inv * (at(2, 0, 0, 1) - wc) - m1 * inv * (wc - at(2, 0, 0, -1)));
  return wc + ((first + second) + third);
}

// corrected: out = the updated component from the input velocities
template <class T>
__global__ void k_visc_explicit(ExplicitViscosity X, const T* __restrict__ phi, const T* __restrict__ u,
                                const T* __restrict__ v, const T* __restrict__ w, T* __restrict__ out) {
  const Lay& Lf = X.axis == 0 ? X.Lu : (X.axis == 1 ? X.Lv : X.Lw);
  FS_IJK(Lf);
  const int64_t f = Lf.at(i, j, k);
  const int e = X.axis == 0 ? i : (X.axis == 1 ? j : k);
  const int n = X.axis == 0 ? Lf.nx : (X.axis == 1 ? Lf.ny : Lf.nz);
  const T* comp = X.axis == 0 ? u : (X.axis == 1 ? v : w);
  if (e == 0 || e == n - 1) {
    out[f] = comp[f];
    return;
  }
  out[f] = (T)explicit_visc_face<T, false>(X, PhiX<T>{phi, X.Lc}, u, v, w, i, j, k);
}

// in place: the faces of hyperplane i + j + k = s of component X.axis
template <class T>
__global__ void k_visc_explicit_plane(ExplicitViscosity X, const T* __restrict__ phi, T* u, T* v, T* w, int s) {
  const Lay& Lf = X.axis == 0 ? X.Lu : (X.axis == 1 ? X.Lv : X.Lw);
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y * blockDim.y + threadIdx.y;
  const int i = s - j - k;
  if (j >= Lf.ny || k >= Lf.nz || i < 0 || i >= Lf.nx) return;
  T* comp = X.axis == 0 ? u : (X.axis == 1 ? v : w);
  comp[Lf.at(i, j, k)] = (T)explicit_visc_face<T, true>(X, PhiX<T>{phi, X.Lc}, u, v, w, i, j, k);
}

template <class T>
int viscosity_explicit(const T* phi, T* u, T* v, T* w, T* ua, T* va, T* wa, const Lay& Lc, const Lay& Lu,
                       const Lay& Lv, const Lay& Lw, double dx, double dt, double rho_neg, double rho_pos,
                       double mu_neg, double mu_pos, int in_place, cudaStream_t s) {
  ExplicitViscosity X{Lc, Lu, Lv, Lw, 0, 1.0 / dx, dt, rho_neg, rho_pos, mu_neg, mu_pos};
  int launches = 0;
  T* outs[3] = {ua, va, wa};
  const Lay* lays[3] = {&Lu, &Lv, &Lw};
  for (int a = 0; a < 3; ++a) {
    X.axis = a;
    const Lay& Lf = *lays[a];
    if (in_place) {
      const dim3 blk(32, 8, 1), grd((Lf.ny + 31) / 32, (Lf.nz + 7) / 8, 1);
      const int planes = Lf.nx + Lf.ny + Lf.nz - 2;
      for (int p = 0; p < planes; ++p) k_visc_explicit_plane<T><<<grd, blk, 0, s>>>(X, phi, u, v, w, p);
      launches += planes;
    } else {
      Launch3 g = launch3(Lf.nx, Lf.ny, Lf.nz);
      k_visc_explicit<T><<<g.grid, g.block, 0, s>>>(X, phi, u, v, w, outs[a]);
      launches += 1;
    }
  }
  return launches;
}

template int viscosity_explicit<float>(const float*, float*, float*, float*, float*, float*, float*, const Lay&,
                                       const Lay&, const Lay&, const Lay&, double, double, double, double, double,
                                       double, int, cudaStream_t);
template int viscosity_explicit<double>(const double*, double*, double*, double*, double*, double*, double*,
                                        const Lay&, const Lay&, const Lay&, const Lay&, double, double, double, double,
                                        double, double, int, cudaStream_t);

template <class T, class V>
void viscosity_system(const T* phi, const T* u, const T* v, const T* w, const Lay& Lc, const Lay& Lu, const Lay& Lv,
                      const Lay& Lw, int axis, double dx, double dt, double rho_neg, double rho_pos, double mu_neg,
                      double mu_pos, V* ax, V* ay, V* az, V* diag, V* rhs, cudaStream_t s) {
  const Lay& Lf = axis == 0 ? Lu : (axis == 1 ? Lv : Lw);
  const ViscSystem<T, V> A{phi,     u,       v,      w,      Lc,           Lu,
                           Lv,      Lw,      Lf,     1.0 / dx, dt,         rho_neg,
                           rho_pos, mu_neg,  mu_pos, dt / rho_neg, dt / (rho_neg + (rho_pos - rho_neg)),
                           ax,      ay,      az,     diag,   rhs};
  const unsigned bx = (Lf.nx + 31) / 32, by = (Lf.ny + 7) / 8;
  // up to 8 planes a thread where that still leaves some 30 blocks per SM: at 256^3 405 us with one
  // plane, 295 with 8 (block scheduling); at 128^3 52 us with one, 55 with 3
  const int chunk = std::max(1, std::min(8, (int)((int64_t)bx * by * Lf.nz / (148 * 32))));
  const dim3 grid(bx, by, (Lf.nz + chunk - 1) / chunk), block(32, 8, 1);
  if (axis == 0) k_visc_system<T, V, 0><<<grid, block, 0, s>>>(A, chunk);
  else if (axis == 1) k_visc_system<T, V, 1><<<grid, block, 0, s>>>(A, chunk);
  else k_visc_system<T, V, 2><<<grid, block, 0, s>>>(A, chunk);
}

#define FS_VISC_INST(T, V)                                                                                          \
  template void viscosity_system<T, V>(const T*, const T*, const T*, const T*, const Lay&, const Lay&, const Lay&, \
                                       const Lay&, int, double, double, double, double, double, double, V*, V*, V*, \
                                       V*, V*, cudaStream_t);
FS_VISC_INST(float, float)
FS_VISC_INST(double, double)
FS_VISC_INST(float, double)

}  // namespace fsb
