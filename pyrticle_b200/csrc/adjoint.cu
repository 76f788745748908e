// adjoint.cu -- reverse-mode derivatives of the particle step.
//
// The reference has no derivatives; these kernels differentiate the forward
// kernels of this library (prt_lsrk_stage, prt_get_velocities,
// prt_deposit_shape in plain mode) exactly, treating the containing element
// of every stage as fixed (the element id is piecewise constant in x; the
// fields interpolated from continuous nodal data are continuous across
// faces, so the derivative is that of the smooth branch).
//
// Gather and scatter swap roles: the forward deposition gathers particles
// onto node positions, its adjoint gathers node adjoints onto particles
// (particles in registers, positions staged per block, tiles.cuh); the forward
// interpolation gathers nodal fields onto particles, its adjoint scatters particle
// adjoints onto the nodes (warp-segmented sums, then FP64 atomics, only when
// nodal field gradients are requested). Gradients along a few basis fields
// (field = sum_k theta_k basis_k + fixed) are reduced per block in a fixed
// order instead, which is deterministic.
//
// Stage adjoint, for the stage  kx' = a kx + dt v(p),  kp' = a kp + dt F(x, p),
// x' = x + b kx',  p' = p + b kp'  (F = q E(x) + q v x B(x)):
//   Lx = lkx' + b lx',  Lp = lkp' + b lp'
//   gE = dt q Lp,  gB = dt q (Lp x v)                  (dL/dE, dL/dB at x)
//   lx = lx' + grad_x [gE . E(x) + gB . B(x)]
//   lp = lp' + Jv^T (dt Lx + dt q (B(x) x Lp)),  Jv = (c/s)(I - p p^T / s^2),
//        s = sqrt(m^2 c^2 + |p|^2)
//   lkx = a Lx,  lkp = a Lp.

#include <cmath>

#include "push.cuh"
#include "tiles.cuh"

namespace {

struct FieldBasis {
  int count;
  const double *f[PRT_MAX_FIELD_BASIS][6];
};

struct GradFields {
  double *f[6];
};

constexpr int ADJ_BLOCK = 128;
// resident blocks per SM the stage adjoint is compiled for: the kernel is
// latency-bound, and 6 (80 registers at order 3, a few spilled) measured
// fastest on B200 (0.25 ms per 1M-particle stage against 0.27 at 5 and 0.37
// at 3); order 4 keeps 3 (35 monomials in registers)
#ifndef ADJ_MIN_BLOCKS
#define ADJ_MIN_BLOCKS 6
#endif

// Forward stage writing its output state to separate arrays (the recorded
// tape keeps the input). Same arithmetic as lsrk_stage_kernel.
template <int ORDER>
__global__ void __launch_bounds__(256, ORDER >= 4 ? 2 : 3)
    lsrk_stage_record_kernel(DevMesh M, const Lagrange<ORDER> L, Fields6 F, long long n,
                             const double *__restrict__ x_in, const double *__restrict__ p_in,
                             const uint32_t *__restrict__ el_in, double *__restrict__ x_out,
                             double *__restrict__ p_out, uint32_t *__restrict__ el_out,
                             const double *__restrict__ q, const double *__restrict__ mass,
                             double *__restrict__ kx, double *__restrict__ kp, double a,
                             double b, double dt, double c, DevStatus *st) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  unsigned ctr[4] = {0, 0, 0, 0};
  const uint32_t e = i < n ? el_in[i] : PRT_INVALID;
  double xx[3] = {0, 0, 0}, pp[3] = {0, 0, 0};
  if (i < n) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      xx[d] = x_in[d * n + i];
      pp[d] = p_in[d * n + i];
    }
  }
  int err = 0;
  const uint32_t ne = stage_particle<ORDER>(M, L, F, e != PRT_INVALID, e, xx, pp, q, mass, kx,
                                            kp, n, i, a, b, dt, c, ctr, &err);
  if (i < n) {
    if (err) record_error(st, err, i);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      x_out[d * n + i] = xx[d];
      p_out[d * n + i] = pp[d];
    }
    el_out[i] = err ? e : ne;
  }
  flush_counters(st, ctr);
}

// Per-element monomial coefficients of a nodal field:
// f(r) = sum_n F_n l_n(r) = sum_j (sum_n F_n W[n][j]) m_j(r).
template <int ORDER>
__global__ void to_monomial_kernel(const Lagrange<ORDER> L, long long E,
                                   const double *__restrict__ f, double *__restrict__ c) {
  constexpr int NP = Lagrange<ORDER>::NP;
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= E) return;
  double fv[NP];
#pragma unroll
  for (int nd = 0; nd < NP; ++nd) fv[nd] = f[e * NP + nd];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    double s = 0;
#pragma unroll
    for (int nd = 0; nd < NP; ++nd) s = fma(L.w[nd * NP + j], fv[nd], s);
    c[e * NP + j] = s;
  }
}

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double o[3]) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

// Adjoint of one stage (see the file comment). One thread per particle; dead
// particles (PRT_INVALID) pass their adjoints through unchanged, as the
// forward stage leaves them untouched. F and FB hold per-element monomial
// coefficients of the fields (to_monomial_kernel): the field and its
// gradient at x are then one pass over the monomials. NODAL: also scatter
// dL/dfield onto the nodes (per-warp shared staging of the Lagrange values
// and gE/gB, summed over runs of lanes in one element, then one atomic per
// run and node).
template <int ORDER, bool NODAL>
__global__ void __launch_bounds__(ADJ_BLOCK, ORDER >= 4 ? 3 : ADJ_MIN_BLOCKS)
    lsrk_stage_adjoint_kernel(DevMesh M, const Lagrange<ORDER> L, Fields6 F, FieldBasis FB,
                              GradFields GF, long long n, const double *__restrict__ x,
                              const double *__restrict__ p, const uint32_t *__restrict__ el,
                              const double *__restrict__ q, const double *__restrict__ mass,
                              double *__restrict__ lx, double *__restrict__ lp,
                              double *__restrict__ lkx, double *__restrict__ lkp, double a,
                              double b, double dt, double c,
                              double *__restrict__ theta_partials) {
  constexpr int NP = Lagrange<ORDER>::NP;
  extern __shared__ double sh_nodal[];  // NODAL: per warp [NP + 6][32] + el[32]
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double tb[PRT_MAX_FIELD_BASIS];
#pragma unroll
  for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k) tb[k] = 0;
  const uint32_t e = i < n ? el[i] : PRT_INVALID;
  double *wl = nullptr, *wg = nullptr;
  uint32_t *wel = nullptr;
  if (NODAL) {
    double *base = sh_nodal + (size_t)warp * ((NP + 6) * 32 + 16);
    wl = base;
    wg = base + NP * 32;
    wel = (uint32_t *)(base + (NP + 6) * 32);
    wel[lane] = e;
  }
  if (e != PRT_INVALID) {
    const double charge = q[i], m = mass[i];
    double LX[3], LP[3], pp[3], v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      LX[d] = fma(b, lx[d * n + i], lkx[d * n + i]);
      LP[d] = fma(b, lp[d * n + i], lkp[d * n + i]);
      pp[d] = p[d * n + i];
    }
    const double s2 = m * m * c * c + pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2];
    const double s = sqrt(s2);
    velocity_exact(pp[0], pp[1], pp[2], m, c, v[0], v[1], v[2]);
    double gE[3], gB[3];
    {
      double t[3];
      cross3(LP, v, t);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        gE[d] = dt * charge * LP[d];
        gB[d] = dt * charge * t[d];
      }
    }
    // powers of the reference coordinates
    const double *A = M.inv_maps + 12 * (size_t)e;
    double r0, r1, r2;
    apply_map_exact(A, x[i], x[n + i], x[2 * n + i], r0, r1, r2);
    double pw0[ORDER + 1], pw1[ORDER + 1], pw2[ORDER + 1];
    pw0[0] = pw1[0] = pw2[0] = 1.0;
#pragma unroll
    for (int k = 1; k <= ORDER; ++k) {
      pw0[k] = pw0[k - 1] * r0;
      pw1[k] = pw1[k - 1] * r1;
      pw2[k] = pw2[k - 1] * r2;
    }
    // one pass over the monomials (the fields come as per-element monomial
    // coefficients): B(x), grad of h = gE . E + gB . B, basis projections
    double mono[NP];
    double Bx[3] = {0, 0, 0}, gr[3] = {0, 0, 0};
    const size_t nb = (size_t)e * NP;
    {
      int idx = 0;
#pragma unroll
      for (int cc = 0; cc <= ORDER; ++cc)
#pragma unroll
        for (int bb = 0; bb <= ORDER - cc; ++bb)
#pragma unroll
          for (int aa = 0; aa <= ORDER - bb - cc; ++aa) {
            const double mj = pw0[aa] * pw1[bb] * pw2[cc];
            if (NODAL) mono[idx] = mj;
            double h = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const double ce = F.f[d] ? __ldg(F.f[d] + nb + idx) : 0.0;
              const double cb = F.f[3 + d] ? __ldg(F.f[3 + d] + nb + idx) : 0.0;
              Bx[d] = fma(cb, mj, Bx[d]);
              h = fma(gE[d], ce, h);
              h = fma(gB[d], cb, h);
            }
            if (aa > 0) gr[0] = fma(h, aa * pw0[aa - 1] * pw1[bb] * pw2[cc], gr[0]);
            if (bb > 0) gr[1] = fma(h, bb * pw0[aa] * pw1[bb - 1] * pw2[cc], gr[1]);
            if (cc > 0) gr[2] = fma(h, cc * pw0[aa] * pw1[bb] * pw2[cc - 1], gr[2]);
#pragma unroll
            for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k) {
              if (k >= FB.count) break;
              double hb = 0;
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                if (FB.f[k][d]) hb = fma(gE[d], __ldg(FB.f[k][d] + nb + idx), hb);
                if (FB.f[k][3 + d]) hb = fma(gB[d], __ldg(FB.f[k][3 + d] + nb + idx), hb);
              }
              tb[k] = fma(hb, mj, tb[k]);
            }
            ++idx;
          }
    }
    if (NODAL) {
      // Lagrange values for the nodal scatter
#pragma unroll
      for (int nd = 0; nd < NP; ++nd) {
        double ln = 0;
#pragma unroll
        for (int j = 0; j < NP; ++j) ln = fma(L.w[nd * NP + j], mono[j], ln);
        wl[nd * 32 + lane] = ln;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        wg[d * 32 + lane] = gE[d];
        wg[(3 + d) * 32 + lane] = gB[d];
      }
    }
    double w[3];
    {
      double t[3];
      cross3(Bx, LP, t);
#pragma unroll
      for (int d = 0; d < 3; ++d) w[d] = dt * (LX[d] + charge * t[d]);
    }
    const double pw_dot = pp[0] * w[0] + pp[1] * w[1] + pp[2] * w[2];
    const double cs = c / s;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      // r = A[0..8] x + A[9..11]: d r_k / d x_d = A[3k + d]
      const double gx = gr[0] * A[d] + gr[1] * A[3 + d] + gr[2] * A[6 + d];
      lx[d * n + i] += gx;
      lp[d * n + i] += cs * (w[d] - pp[d] * pw_dot / s2);
      lkx[d * n + i] = a * LX[d];
      lkp[d * n + i] = a * LP[d];
    }
  } else if (NODAL) {
#pragma unroll
    for (int k = 0; k < 6; ++k) wg[k * 32 + lane] = 0;
  }
  if (NODAL) {
    __syncwarp();
    // outputs (node, component) split over the lanes; each walks the 32
    // staged lanes in order and flushes one sum per run of equal elements
    for (int o = lane; o < NP * 6; o += 32) {
      const int nd = o / 6, k = o % 6;
      if (!GF.f[k]) continue;
      double acc = 0;
      for (int l = 0; l < 32; ++l) {
        const uint32_t el_l = wel[l];
        if (el_l != PRT_INVALID) acc = fma(wl[nd * 32 + l], wg[k * 32 + l], acc);
        if (l == 31 || wel[l + 1] != el_l) {
          if (el_l != PRT_INVALID && acc != 0)
            atomicAdd(GF.f[k] + (size_t)el_l * NP + nd, acc);
          acc = 0;
        }
      }
    }
  }
  if (FB.count > 0) {
    __shared__ double red[PRT_MAX_FIELD_BASIS][ADJ_BLOCK / 32];
#pragma unroll
    for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k) {
      double t = tb[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) red[k][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < FB.count) {
      double t = 0;
      for (int w2 = 0; w2 < ADJ_BLOCK / 32; ++w2) t += red[threadIdx.x][w2];
      theta_partials[(size_t)blockIdx.x * FB.count + threadIdx.x] = t;
    }
  }
}

// The non-zero components of the basis fields.
struct BasisList {
  int bases, count;
  const double *f[6 * PRT_MAX_FIELD_BASIS];
  int comp[6 * PRT_MAX_FIELD_BASIS], basis[6 * PRT_MAX_FIELD_BASIS];
};

// The adjoints of stages `stages` - 1 .. 0 of a tape, one thread per particle
// with its adjoints in registers: a stage reads 52 bytes of the tape (loaded a
// stage ahead) where a launch per stage moved 260, and the basis projections
// are reduced once. Field coefficients interleaved ([E][6][COEF_ROW]), the
// components of `mask`. The derivative of lsrk_stage_adjoint_kernel, equal to
// rounding (one reciprocal root in place of two roots and divisions, the basis
// projections summed over a field's value).
// 300,000 particles, order 3, two basis fields: 24 us a stage, with a launch per
// stage 100.
template <int ORDER>
__global__ void __launch_bounds__(ADJ_BLOCK, ORDER >= 4 ? 3 : 4)
    lsrk_steps_adjoint_kernel(DevMesh M, const double2 *__restrict__ coef, uint32_t mask,
                              const __grid_constant__ BasisList FB, long long n,
                              const double *__restrict__ tx, const double *__restrict__ tp,
                              const uint32_t *__restrict__ te, const double *__restrict__ q,
                              const double *__restrict__ mass, double *__restrict__ lx,
                              double *__restrict__ lp, double *__restrict__ lkx,
                              double *__restrict__ lkp, const __grid_constant__ RkTable rk,
                              int stages, double dt, double c,
                              double *__restrict__ theta_partials) {
  constexpr int NP = Lagrange<ORDER>::NP, ROW = COEF_ROW<ORDER>;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double tb[PRT_MAX_FIELD_BASIS];
#pragma unroll
  for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k) tb[k] = 0;
  if (i < n) {
    const double charge = q[i], m = mass[i], mc2 = m * m * c * c;
    double ax[3], ap[3], akx[3], akp[3], x[3], p[3];
    uint32_t e;
    auto load = [&](int t) {
      const double *sx = tx + (long long)t * 3 * n + i, *sp = tp + (long long)t * 3 * n + i;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        x[d] = __ldg(sx + d * n);
        p[d] = __ldg(sp + d * n);
      }
      e = __ldg(te + (long long)t * n + i);
    };
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      ax[d] = lx[d * n + i];
      ap[d] = lp[d * n + i];
      akx[d] = lkx[d * n + i];
      akp[d] = lkp[d * n + i];
    }
    load(stages - 1);
    int s = (stages - 1) % rk.n;
#pragma unroll 1
    for (int t = stages - 1; t >= 0; --t) {
      const double a = rk.a[s], b = rk.b[s];
      s = s == 0 ? rk.n - 1 : s - 1;
      const uint32_t el = e;
      double pp[3], r[3] = {0, 0, 0};
      if (el != PRT_INVALID) reference_coords(M, el, x[0], x[1], x[2], r);
#pragma unroll
      for (int d = 0; d < 3; ++d) pp[d] = p[d];
      if (t > 0) load(t - 1);
      if (el == PRT_INVALID) continue;  // passed through, as the stage left it untouched
      double LX[3], LP[3], v[3], gE[3], gB[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        LX[d] = fma(b, ax[d], akx[d]);
        LP[d] = fma(b, ap[d], akp[d]);
      }
      const double is = rsqrt(mc2 + pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2]);
      const double cs = c * is;
#pragma unroll
      for (int d = 0; d < 3; ++d) v[d] = cs * pp[d];
      {
        double w[3];
        cross3(LP, v, w);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          gE[d] = dt * charge * LP[d];
          gB[d] = dt * charge * w[d];
        }
      }
      const Powers<ORDER> pw(r);
      double Bx[3] = {0, 0, 0}, gr[3] = {0, 0, 0};
      const double2 *C = coef + (size_t)el * (6 * ROW / 2);
      const size_t nb = (size_t)el * NP;
      double2 u[6];
      int idx = 0;
#pragma unroll
      for (int cc = 0; cc <= ORDER; ++cc)
#pragma unroll
        for (int bb = 0; bb <= ORDER - cc; ++bb)
#pragma unroll
          for (int aa = 0; aa <= ORDER - bb - cc; ++aa) {
            const double mj = pw.p0[aa] * pw.p1[bb] * pw.p2[cc];
            double h = 0;
#pragma unroll
            for (int k = 0; k < 6; ++k)
              if (mask >> k & 1) {
                if (idx % 2 == 0) u[k] = __ldg(C + k * (ROW / 2) + idx / 2);
                const double ck = idx % 2 == 0 ? u[k].x : u[k].y;
                if (k >= 3) Bx[k - 3] = fma(ck, mj, Bx[k - 3]);
                h = fma(k < 3 ? gE[k] : gB[k - 3], ck, h);
              }
            if (aa > 0) gr[0] = fma(h, aa * pw.p0[aa - 1] * pw.p1[bb] * pw.p2[cc], gr[0]);
            if (bb > 0) gr[1] = fma(h, bb * pw.p0[aa] * pw.p1[bb - 1] * pw.p2[cc], gr[1]);
            if (cc > 0) gr[2] = fma(h, cc * pw.p0[aa] * pw.p1[bb] * pw.p2[cc - 1], gr[2]);
            ++idx;
          }
      // the basis fields' non-zero components, one after the other: the value
      // at x times its adjoint (unrolled over basis and component too, the
      // loop above outgrew the instruction cache)
#pragma unroll 1
      for (int o = 0; o < FB.count; ++o) {
        const double *f = FB.f[o] + nb;
        const int comp = FB.comp[o], base = FB.basis[o];
        double val = 0;
        int at = 0;
#pragma unroll
        for (int cc = 0; cc <= ORDER; ++cc)
#pragma unroll
          for (int bb = 0; bb <= ORDER - cc; ++bb) {
            const double t2 = pw.p1[bb] * pw.p2[cc];
#pragma unroll
            for (int aa = 0; aa <= ORDER - bb - cc; ++aa)
              val = fma(__ldg(f + at++), pw.p0[aa] * t2, val);
          }
        const double g = comp == 0   ? gE[0]
                         : comp == 1 ? gE[1]
                         : comp == 2 ? gE[2]
                         : comp == 3 ? gB[0]
                         : comp == 4 ? gB[1]
                                     : gB[2];
#pragma unroll
        for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k) {
          // (a zero times another field's infinity would not be nothing)
          if (k == base) tb[k] = fma(g, val, tb[k]);
        }
      }
      double w[3];
      {
        double z[3];
        cross3(Bx, LP, z);
#pragma unroll
        for (int d = 0; d < 3; ++d) w[d] = dt * (LX[d] + charge * z[d]);
      }
      const double pwd = (pp[0] * w[0] + pp[1] * w[1] + pp[2] * w[2]) * (is * is);
      const double *A = M.inv_maps + 12 * (size_t)el;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        // r = A[0..8] x + A[9..11]: d r_k / d x_d = A[3k + d]
        ax[d] += gr[0] * __ldg(A + d) + gr[1] * __ldg(A + 3 + d) + gr[2] * __ldg(A + 6 + d);
        ap[d] += cs * (w[d] - pp[d] * pwd);
        akx[d] = a * LX[d];
        akp[d] = a * LP[d];
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lx[d * n + i] = ax[d];
      lp[d * n + i] = ap[d];
      lkx[d * n + i] = akx[d];
      lkp[d * n + i] = akp[d];
    }
  }
  if (FB.bases > 0) {
    __shared__ double red[PRT_MAX_FIELD_BASIS][ADJ_BLOCK / 32];
#pragma unroll
    for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k) {
      double t = tb[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x < FB.bases) {
      double t = 0;
      for (int w2 = 0; w2 < ADJ_BLOCK / 32; ++w2) t += red[threadIdx.x][w2];
      theta_partials[(size_t)blockIdx.x * FB.bases + threadIdx.x] = t;
    }
  }
}

// grad_theta[k] += sum over blocks of the partials, in a fixed order.
__global__ void theta_reduce_kernel(long long blocks, int count,
                                    const double *__restrict__ partials,
                                    double *__restrict__ grad_theta) {
  __shared__ double sh[256];
  for (int k = 0; k < count; ++k) {
    double t = 0;
    for (long long bl = threadIdx.x; bl < blocks; bl += blockDim.x) t += partials[bl * count + k];
    sh[threadIdx.x] = t;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) grad_theta[k] += sh[0];
    __syncthreads();
  }
}

// lp += Jv^T lv, Jv = d v / d p = (c/s)(I - p p^T / s^2).
__global__ void velocities_adjoint_kernel(long long n, const double *__restrict__ p,
                                          const double *__restrict__ m, double c,
                                          const double *__restrict__ lv,
                                          double *__restrict__ lp) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double p0 = p[i], p1 = p[n + i], p2 = p[2 * n + i], mm = m[i];
  const double s2 = mm * mm * c * c + p0 * p0 + p1 * p1 + p2 * p2;
  const double cs = c / sqrt(s2);
  const double w0 = lv[i], w1 = lv[n + i], w2 = lv[2 * n + i];
  const double pw = (p0 * w0 + p1 * w1 + p2 * w2) / s2;
  lp[i] += cs * (w0 - p0 * pw);
  lp[n + i] += cs * (w1 - p1 * pw);
  lp[2 * n + i] += cs * (w2 - p2 * pw);
}

// Adjoint of the expansion from positions to nodes, per tile row: every
// position sums the node adjoints of its nodes (ascending node order). Records
// (x, y, z, G0 from dL/drho, G1..G3 from dL/dj).
__global__ void contract_kernel(prt_dep::TilesDev T, long long nn,
                                const uint32_t *__restrict__ run_starts,
                                const uint32_t *__restrict__ run_nodes,
                                const double *__restrict__ grho, const double *__restrict__ gj,
                                double2 *__restrict__ records) {
  const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= T.count) return;
  const uint32_t u = T.rows[r];
  double s[4] = {0, 0, 0, 0};
  for (uint32_t k = run_starts[u]; k < run_starts[u + 1]; ++k) {
    const uint32_t node = run_nodes[k];
    if (grho) s[0] += grho[node];
    if (gj) {
      s[1] += gj[node];
      s[2] += gj[nn + node];
      s[3] += gj[2 * nn + node];
    }
  }
  records[4 * r] = make_double2(T.pos[3 * r], T.pos[3 * r + 1]);
  records[4 * r + 1] = make_double2(T.pos[3 * r + 2], s[0]);
  records[4 * r + 2] = make_double2(s[1], s[2]);
  records[4 * r + 3] = make_double2(s[3], 0);
}

// Adjoint of the plain shape deposition. With weight w = q N and
// S = (a - r^2/a)^alpha:
//   dL/dx_p = w sum_u (G0_u + G_u . v_p) dS/dx_p,
//   dL/dv_p = w sum_u G_u S,   dS/dx_p = alpha (a - r^2/a)^(alpha-1) (2/a) (x_u - x_p),
// with the particles as targets, in bin order, and the positions as sources
// (tiles.cuh): 17 FP64 operations per evaluated pair.
constexpr int DEP_ADJ_PER = 4;
template <bool ALPHA2, bool SHARE>
__global__ void __launch_bounds__(32 * prt_dep::BW, 3)
    deposit_adjoint_kernel(DevMesh M, prt_dep::TilesDev T, prt_dep::TileBinsDev B,
                           const double2 *__restrict__ records, prt_dep::ShapeWeight S,
                           double normalizer, long long n, const uint32_t *__restrict__ perm,
                           const double *__restrict__ x, const double *__restrict__ q,
                           const double *__restrict__ v, const uint32_t *__restrict__ el,
                           double *__restrict__ lx, double *__restrict__ lv) {
  using namespace prt_dep;
  constexpr int PER = DEP_ADJ_PER, LANES = 32 / PER;
  __shared__ BlockStage<4, true> stage;
  __shared__ TileRows rows;
  __shared__ double boxes[BW][6];
  BlockBox X;
  ParticleTargets<PER> D;
  stage_begin(stage);
  const bool any = load_particles<PER, SHARE>(D, X, boxes, n, perm, x, el, S, B, M);
  double vv[3][PER], acc[6][PER];
#pragma unroll
  for (int h = 0; h < PER; ++h) {
#pragma unroll
    for (int d = 0; d < 3; ++d) vv[d][h] = v && D.live[h] ? v[d * n + D.id[h]] : 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k][h] = 0;
  }
  const double radius2 = S.radius * S.radius;
  if (any)
    evaluate_positions<PER, 4, SHARE>(
        stage, rows, T, B, records, M, X, S.radius, S.inv_radius,
        [&](double w0, double w1, double w2, const double *g) {
#pragma unroll
          for (int h = 0; h < PER; ++h) {
            const double d0 = w0 - D.p[0][h], d1 = w1 - D.p[1][h], d2 = w2 - D.p[2][h];
            const double t = inside(radius2, d0, d1, d2);
            // pm = t^(alpha - 1), sv = t^alpha for t > 0 (ALPHA2: by a and a^2 more)
            double pm, sv;
            if (ALPHA2) {
              pm = t > 0 ? t : 0.0;
              sv = pm * pm;
            } else {
              const double ta = t * S.inv_radius;
              pm = t > 0 ? pow(ta, S.alpha - 1.0) : 0.0;
              sv = pm * ta;
            }
            const double hd =
                pm * fma(g[2], vv[1][h], fma(g[1], vv[0][h], fma(g[3], vv[2][h], g[0])));
            acc[0][h] = fma(hd, d0, acc[0][h]);
            acc[1][h] = fma(hd, d1, acc[1][h]);
            acc[2][h] = fma(hd, d2, acc[2][h]);
            acc[3][h] = fma(g[1], sv, acc[3][h]);
            acc[4][h] = fma(g[2], sv, acc[4][h]);
            acc[5][h] = fma(g[3], sv, acc[5][h]);
          }
        });
  reduce_groups<PER, 6>(acc);
  if (SHARE) {
    share_sums<6, PER>(stage, acc);
    if (threadIdx.x >= 32) return;
  }
  const int grp = (threadIdx.x & 31) / LANES;
#pragma unroll
  for (int h = 0; h < PER; ++h) {
    if (h != grp || !D.live[h]) continue;
    const long long i = D.id[h];
    const double w = q[i] * normalizer, wv = w * direct_scale<ALPHA2>(S);
    const double wx = w * S.alpha * (2.0 * S.inv_radius) * (ALPHA2 ? S.inv_radius : 1.0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lx[d * n + i] += wx * acc[d][0];
      if (lv) lv[d * n + i] += wv * acc[3 + d][0];
    }
  }
}

template <int ORDER>
int launch_record(const prt_pusher *P, prt_workspace *ws, long long n, const double *x_in,
                  const double *p_in, const uint32_t *el_in, double *x_out, double *p_out,
                  uint32_t *el_out, const double *q, const double *m, double *kx, double *kp,
                  Fields6 F, double a, double b, double dt, double c, cudaStream_t s) {
  ScopedTimer timer(ws, PRT_TIME_LSRK_STAGE, s);
  lsrk_stage_record_kernel<ORDER><<<prt_grid_blocks(n, 256), 256, 0, s>>>(
      P->mesh->dev, make_lagrange<ORDER>(P), F, n, x_in, p_in, el_in, x_out, p_out, el_out, q,
      m, kx, kp, a, b, dt, c, ws->status);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}

template <int ORDER, bool NODAL>
int launch_adjoint(const prt_pusher *P, prt_workspace *ws, long long n, const double *x,
                   const double *p, const uint32_t *el, const double *q, const double *m,
                   double *lx, double *lp, double *lkx, double *lkp, Fields6 F,
                   const FieldBasis &FB, const GradFields &GF, double a, double b, double dt,
                   double c, double *grad_theta, cudaStream_t s) {
  constexpr int NP = Lagrange<ORDER>::NP;
  const long long blocks = prt_grid_blocks(n, ADJ_BLOCK);
  double *partials = nullptr;
  int rc = PRT_OK;
  if (FB.count > 0) {
    partials = (double *)ws_buffer(ws, PRT_WS_ADJ_PARTIALS,
                                   sizeof(double) * (size_t)blocks * FB.count, &rc);
    if (!partials) return rc;
  }
  const size_t shmem = NODAL ? sizeof(double) * (ADJ_BLOCK / 32) * ((NP + 6) * 32 + 16) : 0;
  auto kern = lsrk_stage_adjoint_kernel<ORDER, NODAL>;
  if (shmem > 48 * 1024)
    PRT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)shmem));
  {
    ScopedTimer timer(ws, PRT_TIME_STAGE_ADJOINT, s);
    kern<<<blocks, ADJ_BLOCK, shmem, s>>>(P->mesh->dev, make_lagrange<ORDER>(P), F, FB, GF, n,
                                          x, p, el, q, m, lx, lp, lkx, lkp, a, b, dt, c,
                                          partials);
    PRT_CHECK_CUDA(cudaGetLastError());
  }
  if (FB.count > 0) {
    theta_reduce_kernel<<<1, 256, 0, s>>>(blocks, FB.count, partials, grad_theta);
    PRT_CHECK_CUDA(cudaGetLastError());
  }
  return PRT_OK;
}

template <int ORDER>
int dispatch_adjoint(bool nodal, const prt_pusher *P, prt_workspace *ws, long long n,
                     const double *x, const double *p, const uint32_t *el, const double *q,
                     const double *m, double *lx, double *lp, double *lkx, double *lkp,
                     Fields6 F, const FieldBasis &FB, const GradFields &GF, double a, double b,
                     double dt, double c, double *grad_theta, cudaStream_t s) {
  if (nodal)
    return launch_adjoint<ORDER, true>(P, ws, n, x, p, el, q, m, lx, lp, lkx, lkp, F, FB, GF,
                                       a, b, dt, c, grad_theta, s);
  return launch_adjoint<ORDER, false>(P, ws, n, x, p, el, q, m, lx, lp, lkx, lkp, F, FB, GF, a,
                                      b, dt, c, grad_theta, s);
}

}  // namespace

extern "C" int prt_lsrk_stage_record(const prt_pusher *P, prt_workspace *ws, int64_t n,
                                     const double *x_in, const double *p_in,
                                     const uint32_t *el_in, double *x_out, double *p_out,
                                     uint32_t *el_out, const double *q, const double *m,
                                     double *kx, double *kp, const double *const fields[6],
                                     double a, double b, double dt, double c, void *stream) {
  if (!P || !ws || n < 0 || !fields) return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0) return PRT_OK;
  if (!x_in || !p_in || !el_in || !x_out || !p_out || !el_out || !q || !m || !kx || !kp)
    return PRT_ERR_INVALID_ARGUMENT;
  if (x_in == x_out || p_in == p_out || el_in == el_out) return PRT_ERR_INVALID_ARGUMENT;
  Fields6 F;
  for (int k = 0; k < 6; ++k) F.f[k] = fields[k];
  cudaStream_t s = (cudaStream_t)stream;
  switch (P->order) {
    case 1: return launch_record<1>(P, ws, n, x_in, p_in, el_in, x_out, p_out, el_out, q, m, kx, kp, F, a, b, dt, c, s);
    case 2: return launch_record<2>(P, ws, n, x_in, p_in, el_in, x_out, p_out, el_out, q, m, kx, kp, F, a, b, dt, c, s);
    case 3: return launch_record<3>(P, ws, n, x_in, p_in, el_in, x_out, p_out, el_out, q, m, kx, kp, F, a, b, dt, c, s);
    case 4: return launch_record<4>(P, ws, n, x_in, p_in, el_in, x_out, p_out, el_out, q, m, kx, kp, F, a, b, dt, c, s);
  }
  return PRT_ERR_INVALID_ARGUMENT;
}

extern "C" int prt_lsrk_stage_adjoint(const prt_pusher *P, prt_workspace *ws, int64_t n,
                                      const double *x, const double *p, const uint32_t *el,
                                      const double *q, const double *m, double *lam_x,
                                      double *lam_p, double *lam_kx, double *lam_kp,
                                      const double *const field_coefficients[6], double a,
                                      double b, double dt, double c,
                                      double *const grad_fields[6], int32_t nbasis,
                                      const double *const *basis, double *grad_theta,
                                      void *stream) {
  if (!P || !ws || n < 0 || !field_coefficients) return PRT_ERR_INVALID_ARGUMENT;
  if (nbasis < 0 || nbasis > PRT_MAX_FIELD_BASIS || (nbasis > 0 && (!basis || !grad_theta)))
    return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0) return PRT_OK;
  if (!x || !p || !el || !q || !m || !lam_x || !lam_p || !lam_kx || !lam_kp)
    return PRT_ERR_INVALID_ARGUMENT;
  Fields6 F;
  for (int k = 0; k < 6; ++k) F.f[k] = field_coefficients[k];
  FieldBasis FB;
  FB.count = nbasis;
  for (int k = 0; k < PRT_MAX_FIELD_BASIS; ++k)
    for (int d = 0; d < 6; ++d) FB.f[k][d] = k < nbasis ? basis[6 * k + d] : nullptr;
  GradFields GF;
  bool nodal = false;
  for (int d = 0; d < 6; ++d) {
    GF.f[d] = grad_fields ? grad_fields[d] : nullptr;
    nodal = nodal || GF.f[d];
  }
  cudaStream_t s = (cudaStream_t)stream;
  switch (P->order) {
    case 1: return dispatch_adjoint<1>(nodal, P, ws, n, x, p, el, q, m, lam_x, lam_p, lam_kx, lam_kp, F, FB, GF, a, b, dt, c, grad_theta, s);
    case 2: return dispatch_adjoint<2>(nodal, P, ws, n, x, p, el, q, m, lam_x, lam_p, lam_kx, lam_kp, F, FB, GF, a, b, dt, c, grad_theta, s);
    case 3: return dispatch_adjoint<3>(nodal, P, ws, n, x, p, el, q, m, lam_x, lam_p, lam_kx, lam_kp, F, FB, GF, a, b, dt, c, grad_theta, s);
    case 4: return dispatch_adjoint<4>(nodal, P, ws, n, x, p, el, q, m, lam_x, lam_p, lam_kx, lam_kp, F, FB, GF, a, b, dt, c, grad_theta, s);
  }
  return PRT_ERR_INVALID_ARGUMENT;
}

template <int ORDER>
static int launch_steps_adjoint(const prt_pusher *P, prt_workspace *ws, const double *coef,
                                uint32_t mask, const BasisList &FB, long long n,
                                const double *tx, const double *tp, const uint32_t *te,
                                const double *q, const double *m, double *lx, double *lp,
                                double *lkx, double *lkp, const RkTable &rk, int stages,
                                double dt, double c, double *grad_theta, cudaStream_t s) {
  const long long blocks = prt_grid_blocks(n, ADJ_BLOCK);
  double *partials = nullptr;
  int rc = PRT_OK;
  if (FB.bases > 0) {
    partials = (double *)ws_buffer(ws, PRT_WS_ADJ_PARTIALS,
                                   sizeof(double) * (size_t)blocks * FB.bases, &rc);
    if (!partials) return rc;
  }
  {
    ScopedTimer timer(ws, PRT_TIME_STAGE_ADJOINT, s);
    lsrk_steps_adjoint_kernel<ORDER><<<blocks, ADJ_BLOCK, 0, s>>>(
        P->mesh->dev, (const double2 *)coef, mask, FB, n, tx, tp, te, q, m, lx, lp, lkx, lkp, rk,
        stages, dt, c, partials);
    PRT_CHECK_CUDA(cudaGetLastError());
  }
  if (FB.bases > 0) {
    theta_reduce_kernel<<<1, 256, 0, s>>>(blocks, FB.bases, partials, grad_theta);
    PRT_CHECK_CUDA(cudaGetLastError());
  }
  return PRT_OK;
}

extern "C" int prt_lsrk_steps_adjoint(const prt_pusher *P, prt_workspace *ws, int64_t n,
                                      const double *tx, const double *tp, const uint32_t *te,
                                      const double *q, const double *m, double *lam_x,
                                      double *lam_p, double *lam_kx, double *lam_kp,
                                      const double *coef, uint32_t mask, const double *rk_a,
                                      const double *rk_b, int32_t rk_count, int32_t stages,
                                      double dt, double c, int32_t nbasis,
                                      const double *const *basis, double *grad_theta,
                                      void *stream) {
  if (!P || !ws || n < 0 || stages < 0 || !rk_a || !rk_b || rk_count < 1 || rk_count > MAX_RK)
    return PRT_ERR_INVALID_ARGUMENT;
  if (nbasis < 0 || nbasis > PRT_MAX_FIELD_BASIS || (nbasis > 0 && (!basis || !grad_theta)))
    return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0 || stages == 0) return PRT_OK;
  if (!tx || !tp || !te || !q || !m || !lam_x || !lam_p || !lam_kx || !lam_kp || !coef ||
      (uintptr_t)coef % 16)
    return PRT_ERR_INVALID_ARGUMENT;
  BasisList FB;
  FB.bases = nbasis;
  FB.count = 0;
  for (int k = 0; k < nbasis; ++k)
    for (int d = 0; d < 6; ++d)
      if (basis[6 * k + d]) {
        FB.f[FB.count] = basis[6 * k + d];
        FB.comp[FB.count] = d;
        FB.basis[FB.count++] = k;
      }
  RkTable rk;
  rk.n = rk_count;
  for (int k = 0; k < MAX_RK; ++k) {
    rk.a[k] = k < rk_count ? rk_a[k] : 0;
    rk.b[k] = k < rk_count ? rk_b[k] : 0;
  }
  cudaStream_t s = (cudaStream_t)stream;
  switch (P->order) {
    case 1: return launch_steps_adjoint<1>(P, ws, coef, mask, FB, n, tx, tp, te, q, m, lam_x, lam_p, lam_kx, lam_kp, rk, stages, dt, c, grad_theta, s);
    case 2: return launch_steps_adjoint<2>(P, ws, coef, mask, FB, n, tx, tp, te, q, m, lam_x, lam_p, lam_kx, lam_kp, rk, stages, dt, c, grad_theta, s);
    case 3: return launch_steps_adjoint<3>(P, ws, coef, mask, FB, n, tx, tp, te, q, m, lam_x, lam_p, lam_kx, lam_kp, rk, stages, dt, c, grad_theta, s);
    case 4: return launch_steps_adjoint<4>(P, ws, coef, mask, FB, n, tx, tp, te, q, m, lam_x, lam_p, lam_kx, lam_kp, rk, stages, dt, c, grad_theta, s);
  }
  return PRT_ERR_INVALID_ARGUMENT;
}

template <int ORDER>
static int launch_to_monomial(const prt_pusher *P, int32_t count, const double *const *fields,
                              double *const *coefficients, cudaStream_t s) {
  const long long E = P->mesh->dev.E;
  const Lagrange<ORDER> L = make_lagrange<ORDER>(P);
  for (int k = 0; k < count; ++k) {
    if (!fields[k] || !coefficients[k]) continue;
    to_monomial_kernel<ORDER><<<prt_grid_blocks(E, 128), 128, 0, s>>>(L, E, fields[k],
                                                                    coefficients[k]);
    PRT_CHECK_CUDA(cudaGetLastError());
  }
  return PRT_OK;
}

extern "C" int prt_fields_to_monomial(const prt_pusher *P, int32_t count,
                                      const double *const *fields, double *const *coefficients,
                                      void *stream) {
  if (!P || count < 0 || (count > 0 && (!fields || !coefficients)))
    return PRT_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  switch (P->order) {
    case 1: return launch_to_monomial<1>(P, count, fields, coefficients, s);
    case 2: return launch_to_monomial<2>(P, count, fields, coefficients, s);
    case 3: return launch_to_monomial<3>(P, count, fields, coefficients, s);
    case 4: return launch_to_monomial<4>(P, count, fields, coefficients, s);
  }
  return PRT_ERR_INVALID_ARGUMENT;
}

extern "C" int prt_velocities_adjoint(int64_t n, const double *p, const double *m, double c,
                                      const double *lam_v, double *lam_p, void *stream) {
  if (n < 0) return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0) return PRT_OK;
  if (!p || !m || !lam_v || !lam_p) return PRT_ERR_INVALID_ARGUMENT;
  velocities_adjoint_kernel<<<prt_grid_blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(
      n, p, m, c, lam_v, lam_p);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}

extern "C" int prt_deposit_shape_adjoint(const prt_mesh *mesh, prt_workspace *ws,
                                         prt_shape_function shape, int64_t n, const double *x,
                                         const double *q, const double *v, const uint32_t *el,
                                         const double *grad_rho, const double *grad_j,
                                         double *lam_x, double *lam_v, void *stream) {
  if (!mesh || !ws || n < 0 || n >= (1ll << 31) || !(shape.radius > 0))
    return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0 || (!grad_rho && !grad_j)) return PRT_OK;
  if (!x || !q || !lam_x || (grad_j && !v)) return PRT_ERR_INVALID_ARGUMENT;
  const PositionSet &PS = mesh->positions;
  const long long nn = mesh->dev.E * (long long)mesh->dev.Np;
  cudaStream_t s = (cudaStream_t)stream;
  ScopedTimer timer(ws, PRT_TIME_DEPOSIT_ADJOINT, s);
  int rc;
  double2 *records =
      (double2 *)ws_buffer(ws, PRT_WS_ADJ_POSITIONS, 4 * sizeof(double2) * PS.count, &rc);
  if (!records) return rc;
  const prt_dep::TilesDev T = prt_dep::tiles_dev(PS.tiles);
  contract_kernel<<<prt_grid_blocks(PS.count, 256), 256, 0, s>>>(
      T, nn, PS.run_starts, PS.run_nodes, grad_rho, grad_j, records);
  PRT_CHECK_CUDA(cudaGetLastError());
  const uint32_t *perm;
  if ((rc = prt_dep::order_particles(mesh, ws, shape.radius, n, x, el, &perm, s))) return rc;
  const double *vv = grad_j ? v : nullptr;
  double *lvv = grad_j ? lam_v : nullptr;
  const bool share = n < prt_dep::SHARE_PARTICLES;
  const long long per = share ? 32 : prt_dep::CHUNK_N;
  auto kern = shape.alpha == 2
                  ? (share ? deposit_adjoint_kernel<true, true> : deposit_adjoint_kernel<true, false>)
                  : (share ? deposit_adjoint_kernel<false, true>
                           : deposit_adjoint_kernel<false, false>);
  kern<<<(unsigned)((n + per - 1) / per), 32 * prt_dep::BW, 0, s>>>(
      mesh->dev, T, prt_dep::tile_bins_dev(PS.tiles), records,
      prt_dep::ShapeWeight{shape.radius, 1.0 / shape.radius, shape.alpha}, shape.normalizer, n,
      perm, x, q, vv, el, lam_x, lvv);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}
