// push.cuh -- per-particle arithmetic of the monomial pusher, shared by the
// forward stage kernels and their adjoints: relativistic velocity, Lagrange
// interpolation of nodal fields, Lorentz force and the fused low-storage RK
// stage update.
#pragma once

#include "common.cuh"
#include "handles.cuh"

// get_velocities arithmetic (particle_state.hpp:98-125), rounded as written.
__device__ __forceinline__ void velocity_exact(double p0, double p1, double p2, double m,
                                               double c, double &v0, double &v1,
                                               double &v2) {
  double pa = __dmul_rn(p0, p0);
  pa = __dadd_rn(pa, __dmul_rn(p1, p1));
  pa = __dadd_rn(pa, __dmul_rn(p2, p2));
  pa = __dsqrt_rn(pa);
  if (pa == 0) {
    v0 = v1 = v2 = 0;
    return;
  }
  double den = __dadd_rn(__dmul_rn(__dmul_rn(__dmul_rn(m, m), c), c), __dmul_rn(pa, pa));
  double vv = __ddiv_rn(__dmul_rn(c, pa), __dsqrt_rn(den));
  double s = __ddiv_rn(vv, pa);
  v0 = __dmul_rn(s, p0);
  v1 = __dmul_rn(s, p1);
  v2 = __dmul_rn(s, p2);
}

template <int ORDER>
struct Lagrange {
  static constexpr int NP = (ORDER + 1) * (ORDER + 2) * (ORDER + 3) / 6;
  // w[i*NP + j]: Lagrange value i = sum_j w[i][j] * monomial_j (canonical
  // monomial order: exponents (a, b, c), a fastest, a + b + c <= ORDER).
  double w[NP * NP];
};

struct Fields6 {
  const double *f[6];
};

// Interpolates the six field components at x inside element e: Lagrange
// values c = V^{-T} m(r) (push_monomial.hpp:155-210), then <c, F_k[e]>
// (push_monomial.hpp:99-111).
template <int ORDER>
__device__ __forceinline__ void interpolate_fields(const DevMesh &M,
                                                   const Lagrange<ORDER> &L,
                                                   const Fields6 &F, uint32_t e,
                                                   double x0, double x1, double x2,
                                                   double ef[6]) {
  constexpr int NP = Lagrange<ORDER>::NP;
  double r0, r1, r2;
  apply_map_exact(M.inv_maps + 12 * (size_t)e, x0, x1, x2, r0, r1, r2);
  double pw0[ORDER + 1], pw1[ORDER + 1], pw2[ORDER + 1];
  pw0[0] = pw1[0] = pw2[0] = 1.0;
#pragma unroll
  for (int k = 1; k <= ORDER; ++k) {
    pw0[k] = pw0[k - 1] * r0;
    pw1[k] = pw1[k - 1] * r1;
    pw2[k] = pw2[k - 1] * r2;
  }
  double mono[NP];
  {
    int idx = 0;
#pragma unroll
    for (int c = 0; c <= ORDER; ++c)
#pragma unroll
      for (int b = 0; b <= ORDER - c; ++b)
#pragma unroll
        for (int a = 0; a <= ORDER - b - c; ++a) mono[idx++] = pw0[a] * pw1[b] * pw2[c];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) ef[k] = 0;
  const size_t base = (size_t)e * NP;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    double ci = 0;
#pragma unroll
    for (int j = 0; j < NP; ++j) ci = fma(L.w[i * NP + j], mono[j], ci);
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (F.f[k]) ef[k] = fma(ci, __ldg(F.f[k] + base + i), ef[k]);
  }
}

template <int ORDER>
static Lagrange<ORDER> make_lagrange(const prt_pusher *P) {
  Lagrange<ORDER> L;
  for (int i = 0; i < Lagrange<ORDER>::NP * Lagrange<ORDER>::NP; ++i) L.w[i] = P->w[i];
  return L;
}

// The RK coefficients of a run of stages: stage t uses a[t % n], b[t % n].
constexpr int MAX_RK = 8;
struct RkTable {
  double a[MAX_RK], b[MAX_RK];
  int n;
};

// Powers of the reference coordinates.
template <int ORDER>
struct Powers {
  double p0[ORDER + 1], p1[ORDER + 1], p2[ORDER + 1];
  __device__ __forceinline__ explicit Powers(const double r[3]) {
    p0[0] = p1[0] = p2[0] = 1.0;
#pragma unroll
    for (int k = 1; k <= ORDER; ++k) {
      p0[k] = p0[k - 1] * r[0];
      p1[k] = p1[k - 1] * r[1];
      p2[k] = p2[k - 1] * r[2];
    }
  }
};

// Entries per field and element of FP64 monomial coefficients (Np rounded up
// to even), [E][6][ROW].
template <int ORDER>
constexpr int COEF_ROW = (Lagrange<ORDER>::NP + 1) / 2 * 2;

// RK update of one particle: k = a k + dt f, y += b k (rounded as written).
__device__ __forceinline__ void rk_update(double a, double b, double dt, double f, double &k,
                                          double &y) {
  k = __dadd_rn(__dmul_rn(a, k), __dmul_rn(dt, f));
  y = __dadd_rn(y, __dmul_rn(b, k));
}

// The same from a force f and velocity v, with the residuals kx, kp [3][n] at
// index i.
__device__ __forceinline__ void update_particle(const double f[3], const double v[3],
                                                double xx[3], double pp[3],
                                                double *__restrict__ kx,
                                                double *__restrict__ kp, long long n,
                                                long long i, double a, double b, double dt) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double kxd = kx[d * n + i], kpd = kp[d * n + i];
    rk_update(a, b, dt, v[d], kxd, xx[d]);
    rk_update(a, b, dt, f[d], kpd, pp[d]);
    kx[d * n + i] = kxd;
    kp[d * n + i] = kpd;
  }
}

// Lorentz force F = q E + v x (q B) in the reference's operation order
// (push_monomial.hpp:219-325).
__device__ __forceinline__ void lorentz_force(double charge, const double ef[6],
                                              const double v[3], double f[3]) {
  double elf[3], qb[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    elf[d] = __dmul_rn(charge, ef[d]);
    qb[d] = __dmul_rn(charge, ef[3 + d]);
  }
  f[0] = __dadd_rn(elf[0], __dsub_rn(__dmul_rn(v[1], qb[2]), __dmul_rn(v[2], qb[1])));
  f[1] = __dadd_rn(elf[1], __dsub_rn(__dmul_rn(v[2], qb[0]), __dmul_rn(v[0], qb[2])));
  f[2] = __dadd_rn(elf[2], __dsub_rn(__dmul_rn(v[0], qb[1]), __dmul_rn(v[1], qb[0])));
}

// The stage after the interpolation: Lorentz force from the fields ef at x
// and the RK update; the caller relocates (a warp at a time, common.cuh).
__device__ __forceinline__ void stage_from_fields(const double ef[6], double xx[3],
                                                  double pp[3], double charge, double mass,
                                                  double *__restrict__ kx,
                                                  double *__restrict__ kp, long long n,
                                                  long long i, double a, double b, double dt,
                                                  double c) {
  double v[3], f[3];
  velocity_exact(pp[0], pp[1], pp[2], mass, c, v[0], v[1], v[2]);
  lorentz_force(charge, ef, v, f);
  update_particle(f, v, xx, pp, kx, kp, n, i, a, b, dt);
}

// One low-storage RK stage of a warp's particles (live: this lane has one, in
// element e):
//   v = v(p), F = q E(x) + v x (q B(x)), k = a k + dt (v, F), (x, p) += b k,
// then relocation. Updates xx, pp in place and the residuals kx, kp [3][n]
// at index i (read and written before the relocation, which keeps them out
// of its live registers). Returns the new element (PRT_INVALID if the
// particle left the mesh); *err is set on a locate error.
template <int ORDER>
__device__ __forceinline__ uint32_t stage_particle(const DevMesh &M, const Lagrange<ORDER> &L,
                                                   const Fields6 &F, bool live, uint32_t e,
                                                   double xx[3], double pp[3],
                                                   const double *__restrict__ q,
                                                   const double *__restrict__ mass,
                                                   double *__restrict__ kx,
                                                   double *__restrict__ kp, long long n,
                                                   long long i, double a,
                                                   double b, double dt, double c,
                                                   unsigned ctr[4], int *err) {
  if (live) {
    double ef[6];
    interpolate_fields<ORDER>(M, L, F, e, xx[0], xx[1], xx[2], ef);
    stage_from_fields(ef, xx, pp, q[i], mass[i], kx, kp, n, i, a, b, dt, c);
  }
  double r[3];
  return relocate(M, live, xx, pp, e, ctr, err, r);
}
