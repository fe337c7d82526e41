// Runs the library's resident solves with a limit of one poll per wait, so that
// waits run out, and then with the ordinary limit on the same buffers.
// Prints per solve: timed_out, then (second run) timed_out, status, iterations.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "fs_kernels.h"

using namespace fsb;

#define CK(x)                                                          \
  do {                                                                 \
    const cudaError_t e_ = (x);                                        \
    if (e_ != cudaSuccess) {                                           \
      std::printf("%s: %s\n", #x, cudaGetErrorString(e_));             \
      std::exit(1);                                                    \
    }                                                                  \
  } while (0)

template <class T>
T* device(const std::vector<T>& h) {
  T* d = nullptr;
  CK(cudaMalloc((void**)&d, h.size() * sizeof(T)));
  CK(cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
  return d;
}

double noise() { return std::rand() / (double)RAND_MAX - 0.5; }

// one phase: every face inside the box carries 1/dx^2
template <class T>
struct System {
  Lay L;
  std::vector<T> ax, ay, az, diag, phi;
  System(int n, double inv2) : L(make_lay(n, n, n)) {
    for (auto* v : {&ax, &ay, &az, &diag, &phi}) v->assign(L.total, T(0));
    for (int k = 0; k < n; ++k)
      for (int j = 0; j < n; ++j)
        for (int i = 0; i < n; ++i) {
          const int64_t c = L.at(i, j, k);
          ax[c] = T(i > 0 ? inv2 : 0.0);
          ay[c] = T(j > 0 ? inv2 : 0.0);
          az[c] = T(k > 0 ? inv2 : 0.0);
          diag[c] = T(inv2 * ((i > 0) + (i < n - 1) + (j > 0) + (j < n - 1) + (k > 0) + (k < n - 1)));
          phi[c] = T(-1);
        }
  }
};

PcgState* state_on_device(const PcgState& s) { return device(std::vector<PcgState>{s}); }
PcgState fetch(const PcgState* d) {
  PcgState s;
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(&s, d, sizeof s, cudaMemcpyDeviceToHost));
  return s;
}

int main() {
  const int n = 32, sms = 148;
  const double dx = 1.0 / n, inv2 = 1.0 / (dx * dx);
  void* slots = nullptr;
  CK(cudaMalloc(&slots, brick_slots_bytes()));
  {
    System<double> S(n, inv2);
    std::vector<double> b(S.L.total, 0.0), zero(S.L.total, 0.0), none(1, 0.0);
    double mean = 0.0;
    for (int pass = 0; pass < 2; ++pass)
      for (int k = 0; k < n; ++k)
        for (int j = 0; j < n; ++j)
          for (int i = 0; i < n; ++i) {
            double& v = b[S.L.at(i, j, k)];
            if (pass == 0) mean += (v = noise()) / ((double)n * n * n);
            else v -= mean;
          }
    Op7<double> A{device(S.ax), device(S.ay), device(S.az), device(S.diag), S.L, 1, device(none)};
    const double *phi = device(S.phi), *db = device(b);
    double *x = device(zero), *z = device(zero);
    BrickPlan P = brick_plan(S.L, sms);
    if (P.gx == 0) return 2;
    PcgState s{};
    s.tol = 1e-6;
    s.max_iter = 1000;
    for (const unsigned polls : {1u, P.polls}) {
      P.polls = polls;
      PcgState* d = state_on_device(s);
      CK(brick_solve(P, A, phi, db, x, z, slots, d, dx, 1.0, 1.0, 0));
      const PcgState r = fetch(d);
      std::printf("%d ", r.timed_out);
      if (polls != 1u) std::printf("%d %d\n", r.status, r.iter);
      CK(cudaMemcpy(x, zero.data(), zero.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
  }
  {
    System<float> S(n, inv2);
    const Lay H = make_half_lay(S.L);
    const float inv = 1.0f / (float)(6.0 * inv2);
    const unsigned short bf = (unsigned short)(reinterpret_cast<const unsigned&>(inv) >> 16);
    const unsigned rounded = (unsigned)bf << 16;
    const double dinv = reinterpret_cast<const float&>(rounded);
    std::vector<float> r(H.total, 0.0f), p(H.total, 0.0f), zero(H.total, 0.0f);
    std::vector<unsigned short> dv(H.total, bf);
    PcgState s{};
    for (int k = 0; k < n; ++k)
      for (int j = 0; j < n; ++j)
        for (int h = 0; h < H.nx; ++h) {
          const int64_t c = H.at(h, j, k);
          r[c] = (float)noise();
          p[c] = r[c] * (float)dinv;
          s.rr += (double)r[c] * r[c];
          s.rz += (double)r[c] * p[c];
        }
    s.best_rr = s.max_rr = s.bb = s.rr;
    s.rz_prev = s.rz;
    s.criterion = 2;
    s.max_iter = 20;
    s.x = device(std::vector<double>(H.total, 0.0));
    const RbOp A{device(S.ax), device(S.ay), device(S.az), S.L, H, device(std::vector<double>(1, 0.0))};
    const float* phi = device(S.phi);
    const unsigned short* ddv = device(dv);
    BrickPlan P = rb_brick_plan(S.L, H, sms);
    if (P.gx == 0) return 2;
    for (const unsigned polls : {1u, P.polls}) {
      P.polls = polls;
      PcgState* d = state_on_device(s);
      CK(rb_brick_iterate(P, A, phi, device(r), device(p), device(zero), ddv, slots, d, dx, 1.0, 1.0, 0));
      const PcgState e = fetch(d);
      std::printf("%d ", e.timed_out);
      if (polls != 1u) std::printf("%d %d\n", e.status, e.iter);
    }
  }
  return 0;
}
