// common.cuh -- device-side mesh view, status word and exact-arithmetic
// helpers shared by the libprt kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/prt.h"

#define PRT_INVALID PRT_INVALID_ELEMENT

// Launch-status check: returns PRT_ERR_CUDA from the enclosing C-ABI call.
#define PRT_CHECK_CUDA(expr)                         \
  do {                                               \
    cudaError_t prt_e_ = (expr);                     \
    if (prt_e_ != cudaSuccess) {                     \
      prt_note_cuda_error(prt_e_, #expr, __LINE__);  \
      return PRT_ERR_CUDA;                           \
    }                                                \
  } while (0)

void prt_note_cuda_error(cudaError_t e, const char *what, int line);

// Device-resident status word of a workspace: first error (code, particle),
// first warning, and the four find-path counters.
struct DevStatus {
  int error;
  int warning;
  long long error_index;
  long long warning_index;
  unsigned long long counters[4];  // same, neighbor, vertex, global
};

enum { CTR_SAME = 0, CTR_NEIGHBOR = 1, CTR_VERTEX = 2, CTR_GLOBAL = 3 };

// Device copy of mesh_data (meshdata.hpp:53-124), passed to kernels by value.
struct DevMesh {
  long long E, V;
  int Np;
  const double *__restrict__ inv_maps;     // [E][12]
  const double *__restrict__ jacobians;    // [E]
  const double *__restrict__ normals;      // [E][4][3]
  const double *__restrict__ plane_rhs;    // [E][4]
  const uint32_t *__restrict__ neighbors;  // [E][4]
  const uint32_t *__restrict__ axes;       // [E][4]
  const uint32_t *__restrict__ el_verts;   // [E][4]
  const double *__restrict__ verts;        // [V][3]
  const uint32_t *__restrict__ vadj_starts;
  const uint32_t *__restrict__ vadj;
  double pmin[3], pmax[3];
  const double *__restrict__ nodes;        // [E*Np][3]
  double bin_origin[3], bin_inv[3];
  int bin_dims[3];
  const uint32_t *__restrict__ bin_starts;
  const uint32_t *__restrict__ bin_elements;
};

// Records the first device error (lowest particle index wins among equal
// codes raised in one launch) without trapping.
__device__ __forceinline__ void record_error(DevStatus *st, int code, long long idx) {
  if (atomicCAS(&st->error, 0, code) == 0) {
    atomicExch((unsigned long long *)&st->error_index, (unsigned long long)idx);
  } else if (st->error == code) {
    atomicMin(&st->error_index, idx);
  }
}

__device__ __forceinline__ void record_warning(DevStatus *st, int code, long long idx) {
  if (atomicCAS(&st->warning, 0, code) == 0) {
    atomicExch((unsigned long long *)&st->warning_index, (unsigned long long)idx);
  } else if (st->warning == code) {
    atomicMin(&st->warning_index, idx);
  }
}

// ---- exact restatements (round-to-nearest, no contraction) ---------------

// hedge affine_map::operator(): y_i = ((A_i0 x0 + A_i1 x1) + A_i2 x2) + b_i
__device__ __forceinline__ void apply_map_exact(const double *__restrict__ m, double x0,
                                                double x1, double x2, double &y0,
                                                double &y1, double &y2) {
  double t;
  t = __dmul_rn(m[0], x0);
  t = __dadd_rn(t, __dmul_rn(m[1], x1));
  t = __dadd_rn(t, __dmul_rn(m[2], x2));
  y0 = __dadd_rn(t, m[9]);
  t = __dmul_rn(m[3], x0);
  t = __dadd_rn(t, __dmul_rn(m[4], x1));
  t = __dadd_rn(t, __dmul_rn(m[5], x2));
  y1 = __dadd_rn(t, m[10]);
  t = __dmul_rn(m[6], x0);
  t = __dadd_rn(t, __dmul_rn(m[7], x1));
  t = __dadd_rn(t, __dmul_rn(m[8], x2));
  y2 = __dadd_rn(t, m[11]);
}

// is_in_unit_simplex (meshdata.hpp:38-48), tolerance 1e-10.
__device__ __forceinline__ bool in_unit_simplex(double r0, double r1, double r2) {
  const double lo = -1.0 - 1e-10;
  if (r0 < lo) return false;
  if (r1 < lo) return false;
  if (r2 < lo) return false;
  double s = __dadd_rn(__dadd_rn(r0, r1), r2);
  return s <= -1.0 + 1e-10;
}

// Reference coordinates of x in element e (the map's 96 bytes as six 16-byte
// loads; same arithmetic as apply_map_exact).
__device__ __forceinline__ void reference_coords(const DevMesh &M, uint32_t e, double x0,
                                                 double x1, double x2, double r[3]) {
  const double2 *m2 = reinterpret_cast<const double2 *>(M.inv_maps + 12 * (size_t)e);
  double m[12];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double2 v = __ldg(m2 + k);
    m[2 * k] = v.x;
    m[2 * k + 1] = v.y;
  }
  apply_map_exact(m, x0, x1, x2, r[0], r[1], r[2]);
}

__device__ __forceinline__ bool in_element(const DevMesh &M, uint32_t e, double x0,
                                           double x1, double x2, double r[3]) {
  reference_coords(M, e, x0, x1, x2, r);
  return in_unit_simplex(r[0], r[1], r[2]);
}

__device__ __forceinline__ double inner3_exact(const double *__restrict__ a, double b0,
                                               double b1, double b2) {
  double t = __dmul_rn(a[0], b0);
  t = __dadd_rn(t, __dmul_rn(a[1], b1));
  return __dadd_rn(t, __dmul_rn(a[2], b2));
}

__device__ __forceinline__ double dist_exact(const double *__restrict__ a, double b0,
                                             double b1, double b2) {
  double d0 = __dsub_rn(a[0], b0), d1 = __dsub_rn(a[1], b1), d2 = __dsub_rn(a[2], b2);
  double t = __dmul_rn(d0, d0);
  t = __dadd_rn(t, __dmul_rn(d1, d1));
  t = __dadd_rn(t, __dmul_rn(d2, d2));
  return __dsqrt_rn(t);
}

// ---- location, a warp at a time ------------------------------------------
//
// All 32 lanes call the functions below; lanes without a particle pass
// active = false. The reference's sequence (same element, the neighbour across
// the face whose normal has the largest product with p, the nearest vertex's
// elements in CSR order, everything) is kept with its arithmetic, so ids and
// counters are the reference's. The two lists are searched by the whole warp
// for one particle after the other, 32 candidates at once, the first hit by
// ballot: a lane walking its list alone is a chain of about a dozen dependent
// inverse-map loads while the other lanes wait (a stage of 10,000 particles
// took 24 us, most of it in that chain).

// The element bin of a point.
__device__ __forceinline__ uint32_t element_bin(const DevMesh &M, const double xs[3]) {
  int b[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double u = (xs[d] - M.bin_origin[d]) * M.bin_inv[d];
    int bi;
    if (!(u >= 0.0))
      bi = 0;
    else if (u >= (double)M.bin_dims[d])
      bi = M.bin_dims[d] - 1;
    else
      bi = min((int)u, M.bin_dims[d] - 1);
    b[d] = bi;
  }
  return (uint32_t)(b[0] + (size_t)M.bin_dims[0] * (b[1] + (size_t)M.bin_dims[1] * b[2]));
}

// For each lane with `need`: the first element of list[starts[row] ..
// starts[row + 1]) that contains x (PRT_INVALID if none, and for the others).
// Two particles are searched at a time, so that one's loads cover the other's.
__device__ __forceinline__ uint32_t search_lists(const DevMesh &M, bool need, uint32_t row,
                                                 const uint32_t *__restrict__ starts,
                                                 const uint32_t *__restrict__ list,
                                                 const double x[3]) {
  const int lane = threadIdx.x & 31;
  uint32_t found = PRT_INVALID, s = 0, t = 0;
  if (need) {
    s = __ldg(starts + row);
    t = __ldg(starts + row + 1);
  }
  unsigned mask = __ballot_sync(0xffffffffu, need);
  while (mask) {
    const int p0 = __ffs(mask) - 1;
    mask &= mask - 1;
    const int p1 = mask ? __ffs(mask) - 1 : p0;
    mask &= mask - 1;  // 0 stays 0
    uint32_t b0 = __shfl_sync(0xffffffffu, s, p0), b1 = __shfl_sync(0xffffffffu, s, p1);
    const uint32_t t0 = __shfl_sync(0xffffffffu, t, p0), t1 = __shfl_sync(0xffffffffu, t, p1);
    double y0[3], y1[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      y0[d] = __shfl_sync(0xffffffffu, x[d], p0);
      y1[d] = __shfl_sync(0xffffffffu, x[d], p1);
    }
    uint32_t f0 = PRT_INVALID, f1 = PRT_INVALID;
    while (b0 < t0 || b1 < t1) {
      const uint32_t e0 = b0 + lane < t0 ? __ldg(list + b0 + lane) : PRT_INVALID;
      const uint32_t e1 = b1 + lane < t1 ? __ldg(list + b1 + lane) : PRT_INVALID;
      double r0[3], r1[3];
      bool in0 = false, in1 = false;
      if (e0 != PRT_INVALID) in0 = in_element(M, e0, y0[0], y0[1], y0[2], r0);
      if (e1 != PRT_INVALID) in1 = in_element(M, e1, y1[0], y1[1], y1[2], r1);
      const unsigned h0 = __ballot_sync(0xffffffffu, in0);
      const unsigned h1 = __ballot_sync(0xffffffffu, in1);
      if (h0) {
        f0 = __shfl_sync(0xffffffffu, e0, __ffs(h0) - 1);
        b0 = t0;
      }
      if (h1) {
        f1 = __shfl_sync(0xffffffffu, e1, __ffs(h1) - 1);
        b1 = t1;
      }
      if (b0 < t0) b0 = min(t0, b0 + 32);
      if (b1 < t1) b1 = min(t1, b1 + 32);
    }
    if (lane == p1) found = f1;
    if (lane == p0) found = f0;
  }
  return found;
}

// Global search (meshdata.hpp:208-215) through the element bins: the lowest
// id among the bin's elements that contain the point.
__device__ __forceinline__ uint32_t find_global(const DevMesh &M, bool active,
                                                const double x[3]) {
  return search_lists(M, active, active ? element_bin(M, x) : 0, M.bin_starts,
                      M.bin_elements, x);
}

// find_new_containing_element (particle_state.hpp:130-261), same decision
// sequence and arithmetic. ctr[] counts locally; *err receives
// PRT_ERR_NO_BEST_NORMAL when no face normal has a positive product with p.
// r receives the reference coordinates of x in the element found.
__device__ __forceinline__ uint32_t find_new_containing(const DevMesh &M, bool active,
                                                        const double x[3], const double p[3],
                                                        uint32_t prev, unsigned ctr[4],
                                                        int *err, double r[3]) {
  uint32_t ne = PRT_INVALID;
  bool open = false;  // still to be found
  if (active) {
    open = !in_element(M, prev, x[0], x[1], x[2], r);
    if (!open) {
      ++ctr[CTR_SAME];
      ne = prev;
    }
  }
  if (!__any_sync(0xffffffffu, open)) return ne;
  uint32_t cv = PRT_INVALID;
  if (open) {
    int best = -1;
    double max_ip = 0;
    const double *nrm = M.normals + 12 * (size_t)prev;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      double ip = inner3_exact(nrm + 3 * f, p[0], p[1], p[2]);
      if (ip > max_ip) {
        best = f;
        max_ip = ip;
      }
    }
    if (best < 0) {
      *err = PRT_ERR_NO_BEST_NORMAL;
      open = false;
    } else {
      const uint32_t nb = M.neighbors[4 * (size_t)prev + best];
      if (nb != PRT_INVALID && in_element(M, nb, x[0], x[1], x[2], r)) {
        ++ctr[CTR_NEIGHBOR];
        ne = nb;
        open = false;
      }
    }
    if (open) {
      double min_dist = __longlong_as_double(0x7ff0000000000000ll);  // +inf
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint32_t vi = M.el_verts[4 * (size_t)prev + v];
        double d = dist_exact(M.verts + 3 * (size_t)vi, x[0], x[1], x[2]);
        if (d < min_dist) {
          cv = vi;
          min_dist = d;
        }
      }
    }
  }
  const uint32_t ve = search_lists(M, open && cv != PRT_INVALID, cv, M.vadj_starts, M.vadj, x);
  if (ve != PRT_INVALID) {
    ++ctr[CTR_VERTEX];
    ne = ve;
    open = false;
  }
  if (__any_sync(0xffffffffu, open)) {
    const uint32_t ge = find_global(M, open, x);
    if (open) {
      ++ctr[CTR_GLOBAL];
      ne = ge;
    }
  }
  if (ne != PRT_INVALID && (ne == ve || open)) reference_coords(M, ne, x[0], x[1], x[2], r);
  return ne;
}

// update of one particle's element (particle_state.hpp:266-357): locate,
// else periodic wrap (positions written back) and locate again, else mark
// dead (PRT_INVALID). A successful wrap costs the extra find_same the
// reference's loop spends re-visiting the particle.
__device__ __forceinline__ uint32_t relocate(const DevMesh &M, bool active, double x[3],
                                             const double p[3], uint32_t prev,
                                             unsigned ctr[4], int *err, double r[3],
                                             bool *wrapped = nullptr) {
  uint32_t ne = PRT_INVALID;
  bool act = active, trip = false;
#pragma unroll 1
  for (int pass = 0;; ++pass) {
    const uint32_t f = find_new_containing(M, act, x, p, prev, ctr, err, r);
    if (act) ne = f;
    if (pass) {
      if (act && ne != PRT_INVALID) ++ctr[CTR_SAME];
      break;
    }
    if (active && ne == PRT_INVALID && !*err) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double mn = M.pmin[a], mx = M.pmax[a];
        if (mn != mx) {
          if (x[a] < mn) {
            x[a] = __dadd_rn(x[a], __dsub_rn(mx, mn));
            trip = true;
          } else if (x[a] > mx) {
            x[a] = __dsub_rn(x[a], __dsub_rn(mx, mn));
            trip = true;
          }
        }
      }
    }
    if (!__any_sync(0xffffffffu, trip)) break;
    act = trip;
  }
  if (wrapped) *wrapped = trip;
  return ne;
}

// Warp-reduce the four counters and add them to the status word.
__device__ __forceinline__ void flush_counters(DevStatus *st, unsigned ctr[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    unsigned v = ctr[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&st->counters[k], (unsigned long long)v);
  }
}

inline int prt_grid_blocks(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  return (int)(b < 1 ? 1 : b);
}
