// steps.cu -- whole low-storage RK steps of the monomial pusher in one launch.
//
// The stages of a step (cloud.py:172-186, 554-603; push_monomial.hpp:85-325)
// are independent per particle while the fields stand still, so one kernel
// takes a particle through all of them in registers: the state crosses HBM
// once per step (about 170 bytes a particle) instead of once per stage (five
// times 216), and a step is one launch.
//
// Fields: per-element monomial coefficients c_j = sum_i F_i W[i][j]
// (l_i = sum_j W[i][j] m_j, the Lagrange polynomials), made once per call for
// all its steps. The value at a particle is then sum_j c_j m_j(r): 6 Np
// multiply-adds from 48 Np bytes, where the nodal form first contracts the
// Np x Np matrix for every particle (Np^2 + 6 Np). With FP64 coefficients this
// is the plain form (forces of a linear field to 2e-16 at orders 1-3, 3.5e-16
// at order 4; the nodal form 2e-16 to 1e-14); the chosen form keeps FP32
// coefficients (rounded from FP64 ones) and sums in FP32, and does everything
// else in FP64: momentum changes within 1.5e-8 to 3.6e-8 of FP64 for fields that
// the elements resolve, orders 1-4 (the tensor-core stage of prt_lsrk_stage:
// 1.9e-8 to 4.2e-8 at orders 1 and 2, 8e-7 and 4.4e-6 at 3 and 4). For fields
// that vary by themselves within an element the monomials' coefficients cancel:
// 3.3e-8, 7.9e-8, 3.0e-7 and 2.7e-6 at orders 1-4 (3.4e-8, 5.0e-8, 7.7e-7 and
// 4.5e-6). Callers with far fewer particles than elements take the nodal form
// of the same kernel.
//
// The reference coordinates that the location test computes for the element
// a particle is found in are the ones the next stage's interpolation needs,
// so each stage applies one inverse map.
//
// What bounds it: every lane receives its element's coefficients through L1
// (960 bytes a stage at order 3, L1 at 88-92% of its throughput), then the
// latency of the location searches at 20 warps an SM. 4M particles, order 3,
// per step of five stages: 0.86 ms (FP64) and 0.80 ms (FP32 coefficients);
// five launches of the nodal stage took 2.5 ms. 5 blocks of 128 threads an SM
// (96 registers) measured best of 3-6.
//
// A tape (optional) receives the state after every stage.

#include "push.cuh"

namespace {

constexpr int ST_BLOCK = 128;
// The state after every stage; in_place: the store is updated too.
struct Tape {
  double *__restrict__ x, *__restrict__ p;  // [stages + 1][3][n], slots 1.. written
  uint32_t *__restrict__ el;                // [stages + 1][n]
  bool in_place;
};

// The monomials of a point in pairs or quadruples, in the canonical order:
// V(k, m) is called with the first index and the values of each group (zeros
// past the last).
template <int ORDER, int G, class T, class V>
__device__ __forceinline__ void monomial_groups(const double r[3], V &&visit) {
  const Powers<ORDER> pw(r);
  T m[G];
  int idx = 0;
#pragma unroll
  for (int cc = 0; cc <= ORDER; ++cc)
#pragma unroll
    for (int bb = 0; bb <= ORDER - cc; ++bb) {
      const double t = pw.p1[bb] * pw.p2[cc];
#pragma unroll
      for (int aa = 0; aa <= ORDER - bb - cc; ++aa) {
        m[idx % G] = (T)(pw.p0[aa] * t);
        if (++idx % G == 0) visit(idx / G - 1, m);
      }
    }
  if (idx % G) {
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (k >= idx % G) m[k] = 0;
    visit(idx / G, m);
  }
}

// FP64 coefficients [E][6][ROW], ROW = NP rounded up to even: 16-byte loads
// of two monomials' coefficients of one field.
template <int ORDER>
struct Coefficients64 {
  static constexpr int ROW = COEF_ROW<ORDER>;
  const double2 *__restrict__ c;
  __device__ __forceinline__ void fields(const DevMesh &, uint32_t e, const double r[3],
                                         const double *, double ef[6]) const {
    const double2 *C = c + (size_t)e * (6 * ROW / 2);
#pragma unroll
    for (int k = 0; k < 6; ++k) ef[k] = 0;
    monomial_groups<ORDER, 2, double>(r, [&](int g, const double *m) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double2 u = __ldg(C + k * (ROW / 2) + g);
        ef[k] = fma(u.y, m[1], fma(u.x, m[0], ef[k]));
      }
    });
  }
};

// FP32 coefficients [E][6][ROW], ROW = NP rounded up to a multiple of four:
// 16-byte loads of four. The monomials are FP64 products rounded once.
template <int ORDER>
struct Coefficients32 {
  static constexpr int ROW = (Lagrange<ORDER>::NP + 3) / 4 * 4;
  const float4 *__restrict__ c;
  __device__ __forceinline__ void fields(const DevMesh &, uint32_t e, const double r[3],
                                         const double *, double ef[6]) const {
    const float4 *C = c + (size_t)e * (6 * ROW / 4);
    float f[6] = {0, 0, 0, 0, 0, 0};
    // the constant's group last: the sums reach the fields' magnitude in their
    // last additions only
    float first[4];
    monomial_groups<ORDER, 4, float>(r, [&](int g, const float *m) {
      if (g == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) first[i] = m[i];
        return;
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const float4 u = __ldg(C + k * (ROW / 4) + g);
        f[k] = fmaf(u.x, m[0], fmaf(u.y, m[1], fmaf(u.z, m[2], fmaf(u.w, m[3], f[k]))));
      }
    });
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float4 u = __ldg(C + k * (ROW / 4));
      ef[k] = (double)fmaf(u.x, first[0], fmaf(u.y, first[1],
                                               fmaf(u.z, first[2], fmaf(u.w, first[3], f[k]))));
    }
  }
};

// The nodal form (interpolate_fields).
template <int ORDER>
struct Nodal {
  Lagrange<ORDER> L;
  Fields6 F;
  __device__ __forceinline__ void fields(const DevMesh &M, uint32_t e, const double r[3],
                                         const double x[3], double ef[6]) const {
    interpolate_fields<ORDER>(M, L, F, e, x[0], x[1], x[2], ef);
  }
};

// v = c p / sqrt(m^2 c^2 + p^2) with one reciprocal root: the reference's
// order (velocity_exact) chains two roots and two divisions, most of a
// stage's latency; this has fewer roundings.
__device__ __forceinline__ void velocity(const double p[3], double m, double c, double v[3]) {
  const double p2 = fma(p[0], p[0], fma(p[1], p[1], p[2] * p[2]));
  const double mc = m * c;
  const double s = p2 == 0 ? 0.0 : c * rsqrt(fma(mc, mc, p2));
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = s * p[d];
}

template <int ORDER, class Source, int MIN_BLOCKS>
__global__ void __launch_bounds__(ST_BLOCK, MIN_BLOCKS)
    lsrk_steps_kernel(DevMesh M, const __grid_constant__ Source S, long long n,
                      double *__restrict__ x, double *__restrict__ p,
                      const double *__restrict__ q, const double *__restrict__ mass,
                      uint32_t *__restrict__ el, double *__restrict__ kx,
                      double *__restrict__ kp, const __grid_constant__ RkTable rk, int stages,
                      double dt, double c, Tape tape, DevStatus *st) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  unsigned ctr[4] = {0, 0, 0, 0};
  uint32_t e = i < n ? el[i] : PRT_INVALID;
  const bool mine = e != PRT_INVALID;
  double xx[3] = {0, 0, 0}, pp[3] = {0, 0, 0}, kxx[3] = {0, 0, 0}, kpp[3] = {0, 0, 0};
  double r[3] = {0, 0, 0}, charge = 0, m = 0;
  if (i < n && (mine || tape.x)) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      xx[d] = x[d * n + i];
      pp[d] = p[d * n + i];
    }
  }
  if (mine) {
    charge = q[i];
    m = mass[i];
    // a first stage with a = 0 drops the old residuals
    if (rk.a[0] != 0) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        kxx[d] = kx[d * n + i];
        kpp[d] = kp[d * n + i];
      }
    }
    reference_coords(M, e, xx[0], xx[1], xx[2], r);
  }
  for (int t = 0, s = 0; t < stages; ++t, s = s + 1 == rk.n ? 0 : s + 1) {
    const bool live = e != PRT_INVALID;
    if (live) {
      const double a = rk.a[s], b = rk.b[s];
      double ef[6], v[3], f[3];
      S.fields(M, e, r, xx, ef);
      velocity(pp, m, c, v);
      lorentz_force(charge, ef, v, f);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        rk_update(a, b, dt, v[d], kxx[d], xx[d]);
        rk_update(a, b, dt, f[d], kpp[d], pp[d]);
      }
    }
    int err = 0;
    const uint32_t ne = relocate(M, live, xx, pp, e, ctr, &err, r);
    if (live) {
      if (err) {
        // the particle keeps its element
        record_error(st, err, i);
        reference_coords(M, e, xx[0], xx[1], xx[2], r);
      } else {
        e = ne;
      }
    }
    if (tape.x && i < n) {
      const long long row = (t + 1) * 3LL * n + i;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        tape.x[row + d * n] = xx[d];
        tape.p[row + d * n] = pp[d];
      }
      tape.el[(t + 1LL) * n + i] = e;
    }
  }
  if (mine && stages > 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      kx[d * n + i] = kxx[d];
      kp[d * n + i] = kpp[d];
      if (tape.in_place) {
        x[d * n + i] = xx[d];
        p[d * n + i] = pp[d];
      }
    }
    if (tape.in_place) el[i] = e;
  }
  flush_counters(st, ctr);
}

// Per-element monomial coefficients of six nodal fields (NULL: zero), out
// [E][6][ROW], entries past NP zero. A block takes 32 elements: their nodal
// values and then their coefficients pass through shared memory, so that
// global memory sees whole rows; a thread contracts one element and field
// with W at uniform addresses. FP64 mma.sync (8 x 8 x 4, W in
// registers) ran the contraction at a quarter of the FMA units' rate: 306 us at
// order 4 and 165,888 elements against 198, with its traffic at 100.
constexpr int FC_ELEMENTS = 32;

template <int ORDER, class T>
struct CoefficientShape {
  static constexpr int NP = Lagrange<ORDER>::NP;
  static constexpr int ROW =
      sizeof(T) == 4 ? Coefficients32<ORDER>::ROW : Coefficients64<ORDER>::ROW;
  // odd strides between lanes: different banks
  static constexpr int STRIDE = NP | 1, OSTRIDE = 6 * ROW + 1;
  static constexpr int IN = 6 * FC_ELEMENTS * STRIDE * 8, 
                       OUT = FC_ELEMENTS * (6 * ROW + 1) * (int)sizeof(T);
  static constexpr int SMEM = IN > OUT ? IN : OUT;
};

template <int ORDER, class T>
__global__ void __launch_bounds__(6 * FC_ELEMENTS)
    field_coefficients_kernel(const __grid_constant__ Lagrange<ORDER> Lt, long long E, Fields6 F,
                              T *__restrict__ out) {
  using SH = CoefficientShape<ORDER, T>;
  constexpr int NP = SH::NP, ROW = SH::ROW;
  extern __shared__ __align__(16) unsigned char fc_smem[];
  double *in = reinterpret_cast<double *>(fc_smem);
  T *rows = reinterpret_cast<T *>(fc_smem);
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;  // a warp per field
  const long long e0 = blockIdx.x * (long long)FC_ELEMENTS;
  const int ne = (int)(E - e0 < FC_ELEMENTS ? E - e0 : FC_ELEMENTS);
  const double *f = nullptr;
#pragma unroll
  for (int c = 0; c < 6; ++c)
    if (k == c) f = F.f[c];
  double *fin = in + k * (FC_ELEMENTS * SH::STRIDE);
  if (f)
    for (int i = lane; i < ne * NP; i += 32)
      fin[(i / NP) * SH::STRIDE + i % NP] = __ldg(f + e0 * NP + i);
  __syncwarp();
  double fv[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) fv[i] = f && lane < ne ? fin[lane * SH::STRIDE + i] : 0.0;
  // relative to the first node's value, which the constant gets back: the
  // contraction's rounding errors scale with the field's variation in the
  // element, not with the field
  const double f0 = fv[0];
#pragma unroll
  for (int i = 0; i < NP; ++i) fv[i] -= f0;
  __syncthreads();  // the rows overwrite the nodal values
  T *o = rows + lane * SH::OSTRIDE + k * ROW;
  // unrolled up to order 3 (42 us at 98,304 elements); at order 4 (1225
  // multiply-adds, 9.8 KB of constants) an output at a time: 198 us at 165,888
  // elements against 256 with five and 418 with all at once
  constexpr int JB = NP <= 20 ? NP : 1;
#pragma unroll 1
  for (int j0 = 0; j0 < NP; j0 += JB) {
    double s[JB];
#pragma unroll
    for (int j = 0; j < JB; ++j) s[j] = j0 + j == 0 ? f0 : 0.0;
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
      for (int j = 0; j < JB; ++j)
        if (NP % JB == 0 || j0 + j < NP) s[j] = fma(Lt.w[(j0 + j) * NP + i], fv[i], s[j]);
#pragma unroll
    for (int j = 0; j < JB; ++j)
      if (NP % JB == 0 || j0 + j < NP) o[j0 + j] = (T)s[j];
  }
#pragma unroll
  for (int j = NP; j < ROW; ++j) o[j] = 0;
  __syncthreads();
  T *dst = out + e0 * 6 * ROW;
  for (int i = threadIdx.x; i < ne * 6 * ROW; i += 6 * FC_ELEMENTS)
    dst[i] = rows[i + i / (6 * ROW)];
}

template <int ORDER, class T>
int launch_coefficients(const prt_pusher *P, Fields6 F, void *out, cudaStream_t s) {
  const long long E = P->mesh->dev.E;
  constexpr int smem = CoefficientShape<ORDER, T>::SMEM;
  auto kern = field_coefficients_kernel<ORDER, T>;
  if (smem > 48 * 1024)
    PRT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  Lagrange<ORDER> Lt;  // transposed: an output's entries lie together
  constexpr int NP = Lagrange<ORDER>::NP;
  for (int i = 0; i < NP; ++i)
    for (int j = 0; j < NP; ++j) Lt.w[j * NP + i] = P->w[(size_t)i * NP + j];
  kern<<<prt_grid_blocks(E, FC_ELEMENTS), 6 * FC_ELEMENTS, smem, s>>>(Lt, E, F, (T *)out);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}

template <int ORDER>
int coefficients(const prt_pusher *P, Fields6 F, int32_t precision, void *out, cudaStream_t s) {
  return precision == PRT_PRECISION_MIXED ? launch_coefficients<ORDER, float>(P, F, out, s)
                                          : launch_coefficients<ORDER, double>(P, F, out, s);
}

struct StepArgs {
  long long n;
  double *x, *p;
  const double *q, *m;
  uint32_t *el;
  double *kx, *kp;
  RkTable rk;
  int stages;
  double dt, c;
  Tape tape;
};

template <int ORDER, int MIN_BLOCKS, class Source>
int launch_steps(const prt_pusher *P, prt_workspace *ws, const Source &S, const StepArgs &A,
                 cudaStream_t s) {
  ScopedTimer timer(ws, PRT_TIME_LSRK_STAGE, s);
  // few particles: one warp per block, so that they spread over all SMs
  const int block = A.n <= 148 * ST_BLOCK ? 32 : ST_BLOCK;
  lsrk_steps_kernel<ORDER, Source, MIN_BLOCKS><<<prt_grid_blocks(A.n, block), block, 0, s>>>(
      P->mesh->dev, S, A.n, A.x, A.p, A.q, A.m, A.el, A.kx, A.kp, A.rk, A.stages, A.dt, A.c,
      A.tape, ws->status);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}

template <int ORDER>
int steps(const prt_pusher *P, prt_workspace *ws, const void *coef, Fields6 F,
          int32_t precision, const StepArgs &A, cudaStream_t s) {
  if (!coef) {
    Nodal<ORDER> S;
    S.L = make_lagrange<ORDER>(P);
    S.F = F;
    return launch_steps<ORDER, 4>(P, ws, S, A, s);
  }
  if (precision == PRT_PRECISION_MIXED) {
    Coefficients32<ORDER> S;
    S.c = (const float4 *)coef;
    return launch_steps<ORDER, 5>(P, ws, S, A, s);
  }
  Coefficients64<ORDER> S;
  S.c = (const double2 *)coef;
  return launch_steps<ORDER, 5>(P, ws, S, A, s);
}

}  // namespace

extern "C" int prt_field_coefficients_bytes(const prt_pusher *P, int32_t precision,
                                            int64_t *bytes) {
  if (!P || !bytes) return PRT_ERR_INVALID_ARGUMENT;
  if (precision != PRT_PRECISION_FP64 && precision != PRT_PRECISION_MIXED)
    return PRT_ERR_INVALID_ARGUMENT;
  const long long rows =
      precision == PRT_PRECISION_MIXED ? (P->np + 3) / 4 * 4 : (P->np + 1) / 2 * 2;
  *bytes = P->mesh->dev.E * rows * 6 * (precision == PRT_PRECISION_MIXED ? 4 : 8);
  return PRT_OK;
}

extern "C" int prt_field_coefficients(const prt_pusher *P, const double *const fields[6],
                                      int32_t precision, void *coefficients_out, void *stream) {
  if (!P || !fields || !coefficients_out) return PRT_ERR_INVALID_ARGUMENT;
  if (precision != PRT_PRECISION_FP64 && precision != PRT_PRECISION_MIXED)
    return PRT_ERR_INVALID_ARGUMENT;
  if ((uintptr_t)coefficients_out % 16) return PRT_ERR_INVALID_ARGUMENT;
  Fields6 F;
  for (int k = 0; k < 6; ++k) F.f[k] = fields[k];
  cudaStream_t s = (cudaStream_t)stream;
  switch (P->order) {
    case 1: return coefficients<1>(P, F, precision, coefficients_out, s);
    case 2: return coefficients<2>(P, F, precision, coefficients_out, s);
    case 3: return coefficients<3>(P, F, precision, coefficients_out, s);
    case 4: return coefficients<4>(P, F, precision, coefficients_out, s);
  }
  return PRT_ERR_INVALID_ARGUMENT;
}

extern "C" int prt_lsrk_steps(const prt_pusher *P, prt_workspace *ws, int64_t n, double *x,
                              double *p, const double *q, const double *m, uint32_t *el,
                              double *kx, double *kp, const void *coef,
                              const double *const fields[6], int32_t precision,
                              const double *rk_a, const double *rk_b, int32_t rk_count,
                              int32_t stages, double dt, double c, double *tape_x,
                              double *tape_p, uint32_t *tape_el, void *stream) {
  if (!P || !ws || n < 0 || stages < 0 || !rk_a || !rk_b || rk_count < 1 || rk_count > MAX_RK)
    return PRT_ERR_INVALID_ARGUMENT;
  if (precision != PRT_PRECISION_FP64 && precision != PRT_PRECISION_MIXED)
    return PRT_ERR_INVALID_ARGUMENT;
  if (!coef && !fields) return PRT_ERR_INVALID_ARGUMENT;
  if ((uintptr_t)coef % 16) return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0 || stages == 0) return PRT_OK;
  if (!x || !p || !q || !m || !el || !kx || !kp) return PRT_ERR_INVALID_ARGUMENT;
  if ((tape_x || tape_p || tape_el) && (!tape_x || !tape_p || !tape_el))
    return PRT_ERR_INVALID_ARGUMENT;
  // a store that is the tape's slot 0 is that in all three arrays
  if ((x == tape_x) != (p == tape_p) || (x == tape_x) != (el == tape_el))
    return PRT_ERR_INVALID_ARGUMENT;
  Fields6 F;
  for (int k = 0; k < 6; ++k) F.f[k] = fields ? fields[k] : nullptr;
  StepArgs A;
  A.n = n;
  A.x = x;
  A.p = p;
  A.q = q;
  A.m = m;
  A.el = el;
  A.kx = kx;
  A.kp = kp;
  A.rk.n = rk_count;
  for (int k = 0; k < MAX_RK; ++k) {
    A.rk.a[k] = k < rk_count ? rk_a[k] : 0;
    A.rk.b[k] = k < rk_count ? rk_b[k] : 0;
  }
  A.stages = stages;
  A.dt = dt;
  A.c = c;
  A.tape.x = tape_x;
  A.tape.p = tape_p;
  A.tape.el = tape_el;
  A.tape.in_place = x != tape_x;
  cudaStream_t s = (cudaStream_t)stream;
  switch (P->order) {
    case 1: return steps<1>(P, ws, coef, F, precision, A, s);
    case 2: return steps<2>(P, ws, coef, F, precision, A, s);
    case 3: return steps<3>(P, ws, coef, F, precision, A, s);
    case 4: return steps<4>(P, ws, coef, F, precision, A, s);
  }
  return PRT_ERR_INVALID_ARGUMENT;
}
