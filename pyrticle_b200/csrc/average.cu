// average.cu -- the averaging pusher (push_average.hpp:26-420): forces from
// the shape-weighted averages of the fields over the nodes within the
// depositor's radius, and the RK update from given forces.
//
// The reference deposits each particle's shape onto the elements its walk
// reaches and accumulates, per element and node, |J_e| w_i rho_i F_i and
// |J_e| w_i rho_i (rho_i = q S(x_i - x_p), w = M 1 the integration weights);
// the force is q <E> + v x (q <B>) with <F> = sum |J| w S F / sum |J| w S
// (the charge cancels). The same sums regroup by node position:
//   <F> = sum_u S(x_u - x_p) WF_u / sum_u S(x_u - x_p) W_u,
// W_u = sum over the nodes at u of |J| w, WF_u = sum |J| w F. A per-position
// pass builds records of W, WE, WB (and, for the verbose standard deviations,
// the weighted squares); the particles gather them as targets of the FP64 pair
// sums (tiles.cuh). No atomics; deterministic.

#include <cmath>

#include "push.cuh"
#include "tiles.cuh"

namespace {

using namespace prt_dep;

// values per position: W, WE[3], WB[3] and, with squares, W|E|^2, W|B|^2
template <bool SQUARES>
constexpr int AVG_NV = SQUARES ? 9 : 7;

// Per tile row the record (x, y, z, values); RUN_LANES lanes share a row.
template <bool SQUARES>
__global__ void average_records_kernel(TilesDev T, int np, const uint32_t *__restrict__ run_starts,
                                       const uint32_t *__restrict__ run_nodes,
                                       const __grid_constant__ NodeWeights N,
                                       const double *__restrict__ jac, Fields6 F,
                                       double2 *__restrict__ records) {
  constexpr int NV = AVG_NV<SQUARES>, RAW = BlockStage<NV, true>::RAW;
  __shared__ double shared[PRT_NODE_WEIGHTS];
  const double *iw = stage_node_weights(N, np, shared);
  const long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / RUN_LANES;
  const int part = threadIdx.x % RUN_LANES;
  double s[2 * RAW];
#pragma unroll
  for (int k = 0; k < 2 * RAW; ++k) s[k] = 0;
  if (r < T.count) {
    const uint32_t u = T.rows[r];
    for (uint32_t k = run_starts[u] + part; k < run_starts[u + 1]; k += RUN_LANES) {
      const uint32_t node = run_nodes[k];
      const double w = iw[node % np] * jac[node / np];
      double f[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) f[c] = F.f[c] ? F.f[c][node] : 0.0;
      s[3] += w;
#pragma unroll
      for (int c = 0; c < 6; ++c) s[4 + c] += w * f[c];
      if (SQUARES) {
        s[10] += w * (f[0] * f[0] + f[1] * f[1] + f[2] * f[2]);
        s[11] += w * (f[3] * f[3] + f[4] * f[4] + f[5] * f[5]);
      }
    }
  }
#pragma unroll
  for (int k = 3; k < 3 + NV; ++k) s[k] = sum_run(s[k]);
  if (r >= T.count || part != 0) return;
#pragma unroll
  for (int k = 0; k < 3; ++k) s[k] = T.pos[3 * r + k];
#pragma unroll
  for (int k = 0; k < RAW; ++k) records[RAW * r + k] = make_double2(s[2 * k], s[2 * k + 1]);
}

template <bool SQUARES>
struct AverageShared {
  BlockStage<AVG_NV<SQUARES>, true> stage;
  TileRows rows;
  double boxes[BW][6];
};

// vis rows [14][n]: pt_e (3), pt_b (3), pt_e_stddev, pt_b_stddev, el_force
// (3), mag_force (3) (push_average.hpp:388-421), written where SQUARES
constexpr int AVG_PER = 4;
template <bool ALPHA2, bool SQUARES, bool SHARE>
__global__ void __launch_bounds__(32 * BW, 3)
    average_forces_kernel(DevMesh M, TilesDev T, TileBinsDev B,
                          const double2 *__restrict__ records, ShapeWeight S, double normalizer,
                          long long n, const uint32_t *__restrict__ perm,
                          const double *__restrict__ x, const double *__restrict__ q,
                          const double *__restrict__ v, const uint32_t *__restrict__ el,
                          double *__restrict__ forces, double *__restrict__ vis,
                          double *__restrict__ scales, DevStatus *st) {
  constexpr int PER = AVG_PER, LANES = 32 / PER, NV = AVG_NV<SQUARES>;
  extern __shared__ __align__(16) unsigned char avg_smem[];
  AverageShared<SQUARES> &A = *reinterpret_cast<AverageShared<SQUARES> *>(avg_smem);
  BlockBox X;
  ParticleTargets<PER> D;
  stage_begin(A.stage);
  const bool any = load_particles<PER, SHARE>(D, X, A.boxes, n, perm, x, el, S, B, M);
  double sum[NV][PER];
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int h = 0; h < PER; ++h) sum[k][h] = 0;
  const double radius2 = S.radius * S.radius;
  if (any)
    evaluate_positions<PER, NV, SHARE>(
        A.stage, A.rows, T, B, records, M, X, S.radius, S.inv_radius,
        [&](double w0, double w1, double w2, const double *g) {
#pragma unroll
          for (int h = 0; h < PER; ++h) {
            const double sw = direct_power<ALPHA2>(
                inside(radius2, w0 - D.p[0][h], w1 - D.p[1][h], w2 - D.p[2][h]), S);
#pragma unroll
            for (int k = 0; k < NV; ++k) sum[k][h] = fma(sw, g[k], sum[k][h]);
          }
        });
  reduce_groups<PER, NV>(sum);
  if (SHARE) {
    share_sums<NV, PER>(A.stage, sum);
    if (threadIdx.x >= 32) return;
  }
  // this lane's particle
  const int grp = (threadIdx.x & 31) / LANES;
  long long i = -1;
#pragma unroll
  for (int h = 0; h < PER; ++h)
    if (h == grp && D.live[h]) i = D.id[h];
  if (i < 0) return;
  double acc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = normalizer * direct_scale<ALPHA2>(S) * sum[k][0];
  const double charge = q[i];
  double f[3] = {0, 0, 0}, ef[6] = {0, 0, 0, 0, 0, 0}, sde = 0, sdb = 0;
  const double den = charge * acc[0];  // the reconstructed charge
  double el_f[3] = {0, 0, 0}, mag_f[3] = {0, 0, 0};
  if (den == 0) {
    record_warning(st, PRT_WARN_ZERO_AVERAGE, i);
  } else {
#pragma unroll
    for (int c = 0; c < 6; ++c) ef[c] = acc[1 + c] / acc[0];
    const double vv[3] = {v[i], v[n + i], v[2 * n + i]};
    double qb[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      el_f[d] = charge * ef[d];
      qb[d] = charge * ef[3 + d];
    }
    mag_f[0] = vv[1] * qb[2] - vv[2] * qb[1];
    mag_f[1] = vv[2] * qb[0] - vv[0] * qb[2];
    mag_f[2] = vv[0] * qb[1] - vv[1] * qb[0];
#pragma unroll
    for (int d = 0; d < 3; ++d) f[d] = el_f[d] + mag_f[d];
    if (SQUARES) {
      const double ve = acc[NV - 2] / acc[0] - (ef[0] * ef[0] + ef[1] * ef[1] + ef[2] * ef[2]);
      const double vb = acc[NV - 1] / acc[0] - (ef[3] * ef[3] + ef[4] * ef[4] + ef[5] * ef[5]);
      sde = ve < 0 ? 0.0 : sqrt(ve);
      sdb = vb < 0 ? 0.0 : sqrt(vb);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) forces[d * n + i] = f[d];
  if (scales) scales[i] = den == 0 ? 0.0 : charge / den;
  if (SQUARES) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      vis[d * n + i] = ef[d];
      vis[(3 + d) * n + i] = ef[3 + d];
      vis[(8 + d) * n + i] = el_f[d];
      vis[(11 + d) * n + i] = mag_f[d];
    }
    vis[6 * n + i] = sde;
    vis[7 * n + i] = sdb;
  }
}

// RK update and relocation from given forces (the stage of a pusher whose
// forces come from a separate pass).
__global__ void __launch_bounds__(256)
    lsrk_update_kernel(DevMesh M, long long n, double *__restrict__ x, double *__restrict__ p,
                       const double *__restrict__ mass, uint32_t *__restrict__ el,
                       double *__restrict__ kx, double *__restrict__ kp,
                       const double *__restrict__ forces, double a, double b, double dt,
                       double c, DevStatus *st) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  unsigned ctr[4] = {0, 0, 0, 0};
  const uint32_t e = i < n ? el[i] : PRT_INVALID;
  const bool live = e != PRT_INVALID;
  double xx[3] = {0, 0, 0}, pp[3] = {0, 0, 0}, r[3];
  if (live) {
    double v[3], f[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      xx[d] = x[d * n + i];
      pp[d] = p[d * n + i];
      f[d] = forces[d * n + i];
    }
    velocity_exact(pp[0], pp[1], pp[2], mass[i], c, v[0], v[1], v[2]);
    update_particle(f, v, xx, pp, kx, kp, n, i, a, b, dt);
  }
  int err = 0;
  const uint32_t ne = relocate(M, live, xx, pp, e, ctr, &err, r);
  if (live) {
    if (err) record_error(st, err, i);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      x[d * n + i] = xx[d];
      p[d * n + i] = pp[d];
    }
    if (!err) el[i] = ne;
  }
  flush_counters(st, ctr);
}

}  // namespace

namespace {

template <bool SQUARES>
int average_forces(const prt_mesh *mesh, prt_workspace *ws, const prt_shape_function &shape,
                   const double *integral_weights, long long n, const double *positions,
                   const double *charges, const double *velocities, const uint32_t *elements,
                   const Fields6 &F, const uint32_t *perm, double *forces, double *vis,
                   double *scales, cudaStream_t s) {
  constexpr int NV = AVG_NV<SQUARES>;
  const PositionSet &PS = mesh->positions;
  const int np = mesh->dev.Np;
  int rc;
  const size_t rec = BlockStage<NV, true>::RAW * (size_t)PS.count;
  double2 *records =
      (double2 *)ws_buffer(ws, PRT_WS_AVERAGE, sizeof(double2) * rec + sizeof(double) * np, &rc);
  if (!records) return rc;
  NodeWeights N;
  if ((rc = prt_node_weights(integral_weights, np, (double *)(records + rec), &N, s))) return rc;
  const TilesDev T = tiles_dev(PS.tiles);
  average_records_kernel<SQUARES><<<prt_grid_blocks(RUN_LANES * PS.count, 128), 128, 0, s>>>(
      T, np, PS.run_starts, PS.run_nodes, N, mesh->dev.jacobians, F, records);
  PRT_CHECK_CUDA(cudaGetLastError());
  const bool share = n < SHARE_PARTICLES;
  const long long per = share ? 32 : CHUNK_N;
  auto kern = shape.alpha == 2 ? (share ? average_forces_kernel<true, SQUARES, true>
                                        : average_forces_kernel<true, SQUARES, false>)
                               : (share ? average_forces_kernel<false, SQUARES, true>
                                        : average_forces_kernel<false, SQUARES, false>);
  constexpr int smem = (int)sizeof(AverageShared<SQUARES>);
  PRT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kern<<<(unsigned)((n + per - 1) / per), 32 * BW, smem, s>>>(
      mesh->dev, T, tile_bins_dev(PS.tiles), records,
      ShapeWeight{shape.radius, 1.0 / shape.radius, shape.alpha}, shape.normalizer, n, perm,
      positions, charges, velocities, elements, forces, vis, scales, ws->status);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}

}  // namespace

extern "C" int prt_average_forces_ordered(const prt_mesh *mesh, prt_workspace *ws,
                                          prt_shape_function shape,
                                          const double *integral_weights, int64_t n,
                                          const double *positions, const double *charges,
                                          const double *velocities, const uint32_t *elements,
                                          const double *const fields[6], double *forces,
                                          double *vis, double *scales, int32_t ordered,
                                          void *stream) {
  if (!mesh || !ws || n < 0 || !(shape.radius > 0) || !integral_weights || !fields)
    return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0) return PRT_OK;
  if (!positions || !charges || !velocities || !forces || n >= (1ll << 31))
    return PRT_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  int rc;
  // A warp evaluates every position near the box of its 32 particles, so these
  // have to lie together; the bins' order sees to it whatever the store's.
  // 100,000 particles, five passes a step: 0.93 ms in the middle of a periodic
  // beam line and 1.09 with the beam across its ends; in the order of a store
  // sorted before the step 0.72, but 1.29 as soon as particles wrap.
  const uint32_t *perm = nullptr;
  if (!ordered && (rc = order_particles(mesh, ws, shape.radius, n, positions, elements, &perm, s)))
    return rc;
  Fields6 F;
  for (int k = 0; k < 6; ++k) F.f[k] = fields[k];
  return vis ? average_forces<true>(mesh, ws, shape, integral_weights, n, positions, charges,
                                    velocities, elements, F, perm, forces, vis, scales, s)
             : average_forces<false>(mesh, ws, shape, integral_weights, n, positions, charges,
                                     velocities, elements, F, perm, forces, vis, scales, s);
}

extern "C" int prt_average_forces(const prt_mesh *mesh, prt_workspace *ws,
                                  prt_shape_function shape, const double *integral_weights,
                                  int64_t n, const double *positions, const double *charges,
                                  const double *velocities, const uint32_t *elements,
                                  const double *const fields[6], double *forces, double *vis,
                                  double *scales, void *stream) {
  return prt_average_forces_ordered(mesh, ws, shape, integral_weights, n, positions, charges,
                                    velocities, elements, fields, forces, vis, scales, 0, stream);
}

extern "C" int prt_lsrk_update(const prt_mesh *mesh, prt_workspace *ws, int64_t n,
                               double *positions, double *momenta, const double *masses,
                               uint32_t *elements, double *kx, double *kp,
                               const double *forces, double rk_a, double rk_b, double dt,
                               double vacuum_c, void *stream) {
  if (!mesh || !ws || n < 0) return PRT_ERR_INVALID_ARGUMENT;
  if (n == 0) return PRT_OK;
  if (!positions || !momenta || !masses || !elements || !kx || !kp || !forces)
    return PRT_ERR_INVALID_ARGUMENT;
  ScopedTimer timer(ws, PRT_TIME_LSRK_STAGE, (cudaStream_t)stream);
  lsrk_update_kernel<<<prt_grid_blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(
      mesh->dev, n, positions, momenta, masses, elements, kx, kp, forces, rk_a, rk_b, dt,
      vacuum_c, ws->status);
  PRT_CHECK_CUDA(cudaGetLastError());
  return PRT_OK;
}
