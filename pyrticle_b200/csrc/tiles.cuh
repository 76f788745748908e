// tiles.cuh -- FP64 sums over (target, source) pairs within the shape radius,
// a warp per tile of 32 targets held in registers.
//
// The FP64 depositions, the normalising integral, the averaging pusher and
// the deposition adjoint are all sums over the pairs (point, particle) closer
// than the shape radius a of the shape weight (a - r^2/a)^alpha times a few
// values of the source. They run here in one form. A block takes four tiles
// (128 targets, compact) and stages the sources near their common box in
// shared memory, 128 at a time (a chunk): every thread copies one record
// (cp.async, two chunks ahead) and moves it into the block's frame. Each warp
// then picks the chunk's entries near its own tile (a ballot per 32, an index
// list) and evaluates those.
//
// Positions as targets (the depositions): with u the target and w the source
// relative to the block's centre,
//   a - r^2/a = (a - |u|^2/a) - |w|^2/a + (2/a) u.w = B + e + V.w,
// three multiply-adds and an add per pair. Its rounding error grows with the
// square of the block's half extent H, about (H/a)^2 2^-53 a; a mesh's tiles
// are compact. Particles as targets (DIRECT) may lie far apart in a block (few
// particles in a long beam line), so these sums take the differences,
//   a^2 - r^2 = a^2 - |w - u|^2,
// three subtractions and three multiply-adds, and the powers of 1/a at the end:
// the error is a few 2^-53 a^2 whatever the block. (By the expansion, 3,000
// particles 30 radii apart on average had a deposition adjoint with a median
// relative error of 3.5e-12, by differences 1.2e-13.)
//
// Lane layout: PER targets per lane, so 32/PER lanes cover the tile and PER
// groups of lanes take different sources at the same time. One source per
// warp (every lane reads the same entry) made shared memory the bound: an
// entry of 64 bytes costs 16 cycles of its bandwidth for 32 x 9 FP64
// operations worth 4.5 cycles; here it is read for PER targets per lane. The
// groups' sums are added at the end by a halving exchange that leaves every
// lane with one target. All orders are fixed: results repeat bitwise.
//
// Measured, deposition of 4M particles on 3.6M positions (7.6e9 pairs within
// the radius): 17.3 ms, FP64 pipe about half busy (the pairs evaluated, 2.2 per
// pair within the radius, would take 8.1 ms on it); the rest are shared-memory
// latencies at 12 warps an SM and the choice of the entries. Before: a warp per
// 64 positions, two per lane, 21.8 ms. A dense bunch (1M particles, order 4)
// 10.1 -> 4.6 ms. Tried: warps that each stream the sources of their own tile
// without barriers (20.7 ms and more: as much time for streaming as for the
// pairs); chunks of consecutive sources (19.3 ms); 8 targets per lane (18.6 ms,
// spills at three blocks an SM); 4 or 5 blocks an SM with 4 per lane (17.6 ms,
// spills with the counters).
#pragma once

#include "binning.cuh"

namespace prt_dep {

// Lanes that share a position's nodes (a vertex has up to a few dozen, an
// interior node one): a lane's loads wait for one another. With one lane a
// position the averaging pass's records of 18,900 positions took 20 us; four,
// and the weights as an argument instead of copied, made a step with five such
// passes 717 -> 678 us (100k particles) and a normalised step of 10k in the
// chosen form 423 -> 413.
constexpr int RUN_LANES = 4;

__device__ __forceinline__ double sum_run(double s) {
#pragma unroll
  for (int o = 1; o < RUN_LANES; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The node weights for a block's threads (every thread calls it)
__device__ __forceinline__ const double *stage_node_weights(const NodeWeights &N, int np,
                                                            double *shared) {
  if (N.more) return N.more;
  for (int k = threadIdx.x; k < np; k += blockDim.x) shared[k] = N.w[k];
  __syncthreads();
  return shared;
}


constexpr int TILE = 32;

// max(t, 0) of an FP64 as one integer maximum on its high word (a negative
// value keeps its low word: a denormal whose square is zero), off the FP64
// pipe.
__device__ __forceinline__ double relu(double t) {
  return __hiloint2double(max(__double2hiint(t), 0), __double2loint(t));
}

struct ShapeWeight {
  double radius, inv_radius, alpha;
};

struct TilesDev {
  long long tiles, count;
  const uint32_t *__restrict__ rows;   // [count] the target of each row
  const double *__restrict__ pos;      // [count][3], row order
  const double *__restrict__ boxes;    // [tiles][6]: centre, half extents
};

inline TilesDev tiles_dev(const TileSet &T) { return {T.tiles, T.count, T.rows, T.pos, T.boxes}; }

// The sums of a plain deposition onto a tile set's targets, FP64: out[d] (or
// NULL) receives, per target, rho (d = 0) and the three j. `run_starts` (or
// NULL) gives the nodes per target for the counters (or NULL): pairs within
// the radius, (particle, node) pairs, evaluated pairs. With a workspace the
// blocks are launched heaviest first.
int launch_deposit_tiles(prt_workspace *ws, const TileSet &T, const uint32_t *run_starts,
                         const BinGrid &G, const DepParticles &P, const ShapeParams &S,
                         double *const out[4], unsigned long long *counters, cudaStream_t s);

// a^2 - |d|^2.
__device__ __forceinline__ double inside(double radius2, double d0, double d1, double d2) {
  return fma(-d0, d0, fma(-d1, d1, fma(-d2, d2, radius2)));
}

__device__ __forceinline__ bool not_finite(double v) {
  return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
}

// The weight (t)^alpha for t > 0, else 0.
template <bool ALPHA2>
__device__ __forceinline__ double shape_power(double t, double alpha) {
  if (ALPHA2) {
    const double r = relu(t);
    return r * r;
  }
  return t > 0 ? pow(t, alpha) : 0.0;
}

// The same from t = a^2 - r^2, up to a factor direct_scale: (t / a)^alpha.
template <bool ALPHA2>
__device__ __forceinline__ double direct_power(double t, const ShapeWeight &S) {
  if (ALPHA2) return shape_power<true>(t, 2);
  return t > 0 ? pow(t * S.inv_radius, S.alpha) : 0.0;
}
template <bool ALPHA2>
__device__ __forceinline__ double direct_scale(const ShapeWeight &S) {
  return ALPHA2 ? S.inv_radius * S.inv_radius : 1.0;
}

// Adds the lanes' partial sums of the groups: v[N][PER] per lane (PER targets,
// N sums) -> v[.][0]: lane (l % (32/PER), l / (32/PER)) ends with the sums of
// target PER (l % (32/PER)) + l / (32/PER).
template <int PER, int N>
__device__ __forceinline__ void reduce_groups(double (&v)[N][PER]) {
  const int grp = (threadIdx.x & 31) / (32 / PER);
#pragma unroll
  for (int half = PER / 2; half > 0; half >>= 1) {
    const bool up = grp & half;
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int h = 0; h < half; ++h) {
        const double give = up ? v[k][h] : v[k][h + half];
        const double keep = up ? v[k][h + half] : v[k][h];
        v[k][h] = keep + __shfl_xor_sync(0xffffffffu, give, half * (32 / PER));
      }
  }
}

// The choice of entries near a warp's box runs in FP32 on coordinates relative
// to the block's centre in units of the radius; it only decides what is
// evaluated. NEAR_LIMIT is (2 radius)^2 with a margin for the rounding of what
// is of the order of the radius. The rounding of the entry, of the box's
// centre and half extent and of their differences grows with the block's half
// extent H instead: at most 2^-24 (5 H + 2) together, which near_half adds to
// the box. (Without the second part, pairs close to the radius were left out
// from some 150 radii on.)
constexpr float NEAR_LIMIT = 4.0f * (1 + 1e-5f) * (1 + 1e-5f);
__device__ __forceinline__ float near_half(double half, double block_half, double inv_radius) {
  return (float)((half + 4e-7 * block_half) * inv_radius + 1e-5);
}

// ------------------------------------------------ four tiles per block

constexpr int BW = 4;          // warps, tiles per block
constexpr int CHUNK_N = 32 * BW;

// Staging of one block: three chunks of entries, W 16-byte words each
// ((w0, w1), (w2, e), values), word by word; entry CHUNK_N lies beyond every
// radius. A record (x, y, z, values) is copied to the same place and moved
// into the block's frame there by the thread that copied it. DIRECT: the
// entries are the records, moved by a whole period at most.
template <int NV, bool DIRECT>
struct BlockStage {
  static constexpr int RAW = (3 + NV + 1) / 2, W = DIRECT ? RAW : 2 + (NV + 1) / 2, STAGES = 3;
  double2 e[STAGES][W][CHUNK_N + 1];
  float4 w[STAGES][CHUNK_N];  // the entries' positions over the radius, for the choice
  uint32_t cum[CHUNK_N + 1];  // sources before the segment
  uint32_t start[CHUNK_N];    // its first record
  double shift[DIRECT ? 1 : CHUNK_N][3];  // from a record's position to the block's frame
  uint32_t wsum[BW];
  uint8_t list[BW][CHUNK_N + 32];
};

// Exclusive scan over the block's threads; `total` receives the sum. The
// threads must be past any use of S.wsum; two barriers.
template <class Stage>
__device__ __forceinline__ uint32_t block_scan(Stage &S, uint32_t v, uint32_t &total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) S.wsum[wid] = x;
  __syncthreads();
  uint32_t before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < BW; ++w) {
    if (w < wid) before += S.wsum[w];
    total += S.wsum[w];
  }
  __syncthreads();
  return before + x - v;
}

__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// A coordinate beyond every radius of what is in the mesh, whose square and
// whose distance's square from its opposite are finite.
constexpr double FAR = 1e150;

template <int NV, bool DIRECT>
__device__ __forceinline__ void stage_begin(BlockStage<NV, DIRECT> &S) {
  using ST = BlockStage<NV, DIRECT>;
  if (threadIdx.x < ST::STAGES * ST::W) {
    const int st = threadIdx.x / ST::W, w = threadIdx.x % ST::W;
    S.e[st][w][CHUNK_N] = DIRECT ? make_double2(w < 2 ? FAR : 0, w < 1 ? FAR : 0)
                                 : make_double2(0, w == 1 ? -1e300 : 0);
  }
}

// The boxes of a block's tiles: the block's centre c and half extents, and
// this warp's tile box in the block's frame over the radius (mid, hf with the
// FP32 margin, near_half); a warp without a tile has hf < 0 with a magnitude
// that keeps everything out.
struct BlockBox {
  double c[3], h[3];
  float mid[3], hf[3];
};

// Evaluates the `total` sources of the present segments (S.cum, S.start and
// the shifts to the block's frame S.shift, or DIRECT `shift` for all; written
// before a barrier) against the block's tiles: op(w0, w1, w2, e, v), DIRECT
// op(x, y, z, v), on every lane with its group's entry.
// SHARE: the warps have the same tile and take 32 of a chunk's entries each.
// A chunk with an entry whose values are not all finite goes through op.within
// (not DIRECT), which adds nothing where the weight is zero: a weight of zero
// times infinity would spoil targets beyond the radius.
// Returns the entries evaluated (per warp). Ends with a barrier.
template <int PER, int NV, bool SHARE, bool DIRECT, class Op>
__device__ __forceinline__ uint32_t evaluate_segments(BlockStage<NV, DIRECT> &S,
                                                      const double2 *__restrict__ records,
                                                      uint32_t total, const BlockBox &X,
                                                      const double *shift, double inv_radius,
                                                      Op &&op) {
  using ST = BlockStage<NV, DIRECT>;
  constexpr int LANES = 32 / PER;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, grp = lane / LANES;
  uint8_t *list = S.list[wid];
  uint32_t evaluated = 0;
  // Thread t takes the sources t chunks .. t chunks + chunks - 1, one per
  // chunk: a chunk is a sample of the whole neighbourhood, so that every warp
  // finds its share in it. (128 consecutive sources lie together: near one
  // tile and far from the others, whose warps then wait at the barrier.)
  const uint32_t chunks = (total + CHUNK_N - 1) / CHUNK_N;
  const uint32_t first = tid * chunks;
  const uint32_t mine = first < total ? min(chunks, total - first) : 0;
  int seg = 0;
  if (mine) {
#pragma unroll
    for (int step = CHUNK_N / 2; step > 0; step >>= 1)
      if (S.cum[seg + step] <= first) seg += step;
  }
  // two chunks are in flight: the segments of this thread's records in them
  int seg0 = 0, seg1 = 0;
  auto copy = [&](uint32_t chunk) {
    if (chunk < mine) {
      const uint32_t f = first + chunk;
      while (f >= S.cum[seg + 1]) ++seg;
      const double2 *src = records + (size_t)ST::RAW * (S.start[seg] + (f - S.cum[seg]));
#pragma unroll
      for (int w = 0; w < ST::RAW; ++w) copy16_async(&S.e[chunk % ST::STAGES][w][tid], src + w);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy(0);
  seg0 = seg;
  copy(1);
  seg1 = seg;
  for (uint32_t k = 0; k < chunks; ++k) {
    const int st = k % ST::STAGES;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (k < mine) {
      if constexpr (DIRECT) {
        const double2 t0 = S.e[st][0][tid], t1 = S.e[st][1][tid];
        const double w0 = t0.x + shift[0], w1 = t0.y + shift[1], w2 = t1.x + shift[2];
        S.w[st][tid] = make_float4((float)((w0 - X.c[0]) * inv_radius),
                                   (float)((w1 - X.c[1]) * inv_radius),
                                   (float)((w2 - X.c[2]) * inv_radius), 0);
        S.e[st][0][tid] = make_double2(w0, w1);
        S.e[st][1][tid] = make_double2(w2, t1.y);
      } else {
        double v[2 * ST::RAW];
#pragma unroll
        for (int w = 0; w < ST::RAW; ++w) {
          const double2 t = S.e[st][w][tid];
          v[2 * w] = t.x;
          v[2 * w + 1] = t.y;
        }
        const double w0 = v[0] + S.shift[seg0][0], w1 = v[1] + S.shift[seg0][1],
                     w2 = v[2] + S.shift[seg0][2];
        bool odd = false;
#pragma unroll
        for (int k = 3; k < 3 + NV; ++k) odd = odd || not_finite(v[k]);
        S.w[st][tid] = make_float4((float)(w0 * inv_radius), (float)(w1 * inv_radius),
                                   (float)(w2 * inv_radius), odd ? 1.0f : 0.0f);
        S.e[st][0][tid] = make_double2(w0, w1);
        S.e[st][1][tid] = make_double2(w2, -(w0 * w0 + w1 * w1 + w2 * w2) * inv_radius);
#pragma unroll
        for (int w = 2; w < ST::W; ++w)
          S.e[st][w][tid] =
              make_double2(v[2 * w - 1], 2 * w < 3 + NV ? v[2 * w < 2 * ST::RAW ? 2 * w : 0] : 0.0);
      }
    } else {
      S.w[st][tid] = make_float4(1e30f, 0, 0, 0);
    }
    // chunk k is in place, chunk k - 1 done with: its stage takes chunk k + 2
    __syncthreads();
    copy(k + 2);
    seg0 = seg1;
    seg1 = seg;
    int n = 0;
    bool odd = false;
#pragma unroll
    for (int q = 0; q < BW; ++q) {
      if (SHARE && q != wid) continue;
      const float4 w = S.w[st][32 * q + lane];
      const float d0 = fabsf(w.x - X.mid[0]) - X.hf[0], d1 = fabsf(w.y - X.mid[1]) - X.hf[1],
                  d2 = fabsf(w.z - X.mid[2]) - X.hf[2];
      const float e0 = d0 + fabsf(d0), e1 = d1 + fabsf(d1), e2 = d2 + fabsf(d2);
      const bool in = e0 * e0 + e1 * e1 + e2 * e2 <= NEAR_LIMIT;
      const unsigned bal = __ballot_sync(0xffffffffu, in);
      if (in) list[n + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)(32 * q + lane);
      n += __popc(bal);
      if (!DIRECT) odd = odd || (in && w.w != 0);
    }
    // up to a whole turn with entries beyond every radius
    if (lane < PER) list[n + lane] = CHUNK_N;
    __syncwarp();
    evaluated += n;
    if constexpr (!DIRECT) {
      if (__any_sync(0xffffffffu, odd)) {
#pragma unroll 1
        for (int i = 0; i < n; i += PER) {
          double v[2 * ST::W];
#pragma unroll
          for (int w = 0; w < ST::W; ++w) {
            const double2 t = S.e[st][w][list[i + grp]];
            v[2 * w] = t.x;
            v[2 * w + 1] = t.y;
          }
          op.within(v[0], v[1], v[2], v[3], v + 4);
        }
        n = 0;
      }
    }
    int id = list[grp];
#pragma unroll 2
    for (int i = 0; i < n; i += PER) {
      const int cur = id;
      id = list[i + PER + grp];
      double v[2 * ST::W];
#pragma unroll
      for (int w = 0; w < ST::W; ++w) {
        const double2 t = S.e[st][w][cur];
        v[2 * w] = t.x;
        v[2 * w + 1] = t.y;
      }
      if constexpr (DIRECT)
        op(v[0], v[1], v[2], v + 3);
      else
        op(v[0], v[1], v[2], v[3], v + 4);
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  return evaluated;
}

// All particles of the bin rows near the block's box, evaluated against its
// tiles (evaluate_segments).
template <int PER, int NV, bool SHARE, class Op>
__device__ __forceinline__ uint32_t evaluate_particles(BlockStage<NV, false> &S, const BinGrid &G,
                                                       const DepParticles &P, const BlockBox &X,
                                                       double radius, double inv_radius,
                                                       Op &&op) {
  const int tid = threadIdx.x;
  const double rr = radius * (1 + 1e-5), rr2 = rr * rr;
  int ulo[3], uhi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    ulo[d] = bin_floor(G, d, X.c[d] - X.h[d] - rr);
    uhi[d] = bin_floor(G, d, X.c[d] + X.h[d] + rr);
    if (G.periodic[d]) {
      ulo[d] -= 1;
      uhi[d] += 1;
    } else {
      ulo[d] = max(ulo[d], 0);
      uhi[d] = min(uhi[d], G.dims[d] - 1);
    }
  }
  auto slab_gap = [&](int d, double blo) {
    const double e = fmax(0.0, fmax(blo - (X.c[d] + X.h[d]), (X.c[d] - X.h[d]) - (blo + G.w[d]))) -
                     G.slack[d];
    return e > 0 ? e * e : 0.0;
  };
  const int ny = max(0, uhi[1] - ulo[1] + 1), nz = max(0, uhi[2] - ulo[2] + 1);
  const long long nrows = (long long)ny * nz;
  // along a periodic x a row is in as many pieces as the block's reach has
  // periods in it (the points of a brick may be any number of periods apart)
  const int pieces =
      G.periodic[0] ? floor_div(uhi[0], G.dims[0]) - floor_div(ulo[0], G.dims[0]) + 1 : 1;
  uint32_t evaluated = 0;
  for (long long i0 = 0; i0 < nrows * pieces; i0 += CHUNK_N) {
    const long long r = (i0 + tid) / pieces;
    const int piece = (int)(i0 + tid - r * pieces);
    uint32_t start = 0, len = 0;
    double sh[3] = {0, 0, 0};
    if (r < nrows) {
      const int bz = ulo[2] + (int)(r / ny), by = ulo[1] + (int)(r % ny);
      int wz = bz, wy = by, qz = 0, qy = 0;
      if (G.periodic[2]) {
        qz = floor_div(bz, G.dims[2]);
        wz = bz - qz * G.dims[2];
      }
      if (G.periodic[1]) {
        qy = floor_div(by, G.dims[1]);
        wy = by - qy * G.dims[1];
      }
      const double dyz2 =
          slab_gap(2, G.origin[2] + bz * G.w[2]) + slab_gap(1, G.origin[1] + by * G.w[1]);
      if (dyz2 <= rr2) {
        const double rem = sqrt(rr2 - dyz2);
        int bx0 = bin_floor(G, 0, X.c[0] - X.h[0] - rem);
        int bx1 = bin_floor(G, 0, X.c[0] + X.h[0] + rem);
        int qx = 0;
        if (G.periodic[0]) {
          bx0 = max(bx0 - 1, ulo[0]);
          bx1 = min(bx1 + 1, uhi[0]);
          qx = floor_div(bx0, G.dims[0]) + piece;
          bx0 = max(bx0, qx * G.dims[0]);
          bx1 = min(bx1, qx * G.dims[0] + G.dims[0] - 1);
        } else {
          bx0 = max(bx0, ulo[0]);
          bx1 = min(bx1, uhi[0]);
        }
        if (bx0 <= bx1) {
          const long long row = (long long)G.dims[0] * (wy + (long long)G.dims[1] * wz);
          const int wx = bx0 - qx * G.dims[0];
          start = P.starts[row + wx];
          len = P.starts[row + wx + (bx1 - bx0) + 1] - start;
          sh[0] = qx * G.period[0] - X.c[0];
          sh[1] = qy * G.period[1] - X.c[1];
          sh[2] = qz * G.period[2] - X.c[2];
        }
      }
    }
    uint32_t total;
    const uint32_t before = block_scan(S, len, total);
    if (total == 0) continue;
    // (empty segments stay: the walk steps over them)
    S.cum[tid] = before;
    S.start[tid] = start;
#pragma unroll
    for (int d = 0; d < 3; ++d) S.shift[tid][d] = sh[d];
    if (tid == 0) S.cum[CHUNK_N] = total;
    __syncthreads();
    evaluated += evaluate_segments<PER, NV, SHARE, false>(
        S, reinterpret_cast<const double2 *>(P.payload), total, X, nullptr, inv_radius, op);
  }
  return evaluated;
}

// ------------------------------------------- particles as the targets

struct TileBinsDev {
  double origin[3], extent[3], inv_w[3], max_half[3];
  int dims[3];
  const uint32_t *__restrict__ starts, *__restrict__ tiles;
};

inline TileBinsDev tile_bins_dev(const TileSet &T) {
  TileBinsDev B;
  for (int d = 0; d < 3; ++d) {
    B.origin[d] = T.bins.origin[d];
    B.extent[d] = T.bins.extent[d];
    B.inv_w[d] = T.bins.inv_w[d];
    B.max_half[d] = T.bins.max_half[d];
    B.dims[d] = T.bins.dims[d];
  }
  B.starts = T.bins.starts;
  B.tiles = T.bins.tiles;
  return B;
}

// The rows of tile bins of one turn of the search.
struct TileRows {
  uint32_t cum[CHUNK_N + 1], first[CHUNK_N];
};

// All positions of the tiles near the block's box (periodic images included),
// evaluated against its targets: `records` in the tiles' row order.
template <int PER, int NV, bool SHARE, class Op>
__device__ __forceinline__ void evaluate_positions(BlockStage<NV, true> &S, TileRows &Q,
                                                   const TilesDev &T, const TileBinsDev &B,
                                                   const double2 *__restrict__ records,
                                                   const DevMesh &M, const BlockBox &X,
                                                   double radius, double inv_radius, Op &&op) {
  const int tid = threadIdx.x;
  const double rr = radius * (1 + 1e-5), rr2 = rr * rr;
  int lo_img[3], hi_img[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo_img[d] = hi_img[d] = 0;
    if (M.pmin[d] != M.pmax[d]) {
      if (X.c[d] - X.h[d] - rr < M.pmin[d]) hi_img[d] = 1;
      if (X.c[d] + X.h[d] + rr > M.pmax[d]) lo_img[d] = -1;
    }
  }
  for (int iz = lo_img[2]; iz <= hi_img[2]; ++iz)
    for (int iy = lo_img[1]; iy <= hi_img[1]; ++iy)
      for (int ix = lo_img[0]; ix <= hi_img[0]; ++ix) {
        // the box moved by whole periods, or the positions by their opposite
        const double shift[3] = {-ix * (M.pmax[0] - M.pmin[0]), -iy * (M.pmax[1] - M.pmin[1]),
                                 -iz * (M.pmax[2] - M.pmin[2])};
        const double c[3] = {X.c[0] - shift[0], X.c[1] - shift[1], X.c[2] - shift[2]};
        int b0[3], b1[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double reach = X.h[d] + rr + B.max_half[d];
          const double l = floor((c[d] - reach - B.origin[d]) * B.inv_w[d]);
          const double h = floor((c[d] + reach - B.origin[d]) * B.inv_w[d]);
          b0[d] = (int)fmax(0.0, fmin(l, B.dims[d] - 1.0));
          b1[d] = (int)fmax(0.0, fmin(h, B.dims[d] - 1.0));
        }
        const int ny = b1[1] - b0[1] + 1;
        const int nrows = ny * (b1[2] - b0[2] + 1);
        for (int r0 = 0; r0 < nrows; r0 += CHUNK_N) {
          const int r = r0 + tid;
          uint32_t first = 0, len = 0;
          if (r < nrows) {
            const long long row =
                (long long)B.dims[0] * (b0[1] + r % ny + (long long)B.dims[1] * (b0[2] + r / ny));
            first = B.starts[row + b0[0]];
            len = B.starts[row + b1[0] + 1] - first;
          }
          uint32_t tiles;
          const uint32_t before = block_scan(S, len, tiles);
          if (tiles == 0) continue;
          Q.cum[tid] = before;
          Q.first[tid] = first;
          if (tid == 0) Q.cum[CHUNK_N] = tiles;
          __syncthreads();
          for (uint32_t t0 = 0; t0 < tiles; t0 += CHUNK_N) {
            const uint32_t j = t0 + tid;
            uint32_t tile = 0, n = 0;
            if (j < tiles) {
              int at = 0;
#pragma unroll
              for (int step = CHUNK_N / 2; step > 0; step >>= 1)
                if (Q.cum[at + step] <= j) at += step;
              tile = B.tiles[Q.first[at] + (j - Q.cum[at])];
              double d2 = 0;
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                const double e = fmax(0.0, fabs(T.boxes[6 * (size_t)tile + d] - c[d]) -
                                               T.boxes[6 * (size_t)tile + 3 + d] - X.h[d]);
                d2 = fma(e, e, d2);
              }
              if (d2 <= rr2) n = (uint32_t)min((long long)TILE, T.count - (long long)TILE * tile);
            }
            uint32_t total;
            const uint32_t at = block_scan(S, n, total);
            if (total == 0) continue;
            S.cum[tid] = at;
            S.start[tid] = TILE * tile;
            if (tid == 0) S.cum[CHUNK_N] = total;
            __syncthreads();
            evaluate_segments<PER, NV, SHARE, true>(S, records, total, X, shift, inv_radius, op);
          }
          __syncthreads();
        }
      }
}

// The particles of a warp's lanes as targets: lane (tg, .) holds PER of the 32
// from k0 (bin order with `perm`, else store order), and the block's and the
// warp's boxes around those within reach of a position. Particles that are not
// (removed, or outside the mesh by more than the radius and a period, or at no
// finite place) have zero sums and no part in the boxes: one at infinity would
// take its whole block's frame there. SHARE: all warps have the same 32.
// Returns whether the block has a particle within reach at all.
template <int PER>
struct ParticleTargets {
  long long id[PER];  // store index, -1 for none
  bool live[PER];
  double p[3][PER];  // out of reach: beyond every radius
};

template <int PER, bool SHARE>
__device__ __forceinline__ bool load_particles(ParticleTargets<PER> &D, BlockBox &X,
                                               double (*boxes)[6], long long n,
                                               const uint32_t *__restrict__ perm,
                                               const double *__restrict__ x,
                                               const uint32_t *__restrict__ el,
                                               const ShapeWeight &S, const TileBinsDev &B,
                                               const DevMesh &M) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int tg = lane % (32 / PER);
  const long long k0 = 32 * (SHARE ? (long long)blockIdx.x : BW * (long long)blockIdx.x + wid);
  double lo[3] = {INFINITY, INFINITY, INFINITY},
         hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int h = 0; h < PER; ++h) {
    const long long k = k0 + PER * tg + h;
    D.id[h] = k < n ? (perm ? (long long)perm[k] : k) : -1;
    D.live[h] = D.id[h] >= 0 && !(el && el[D.id[h]] == PRT_INVALID);
    bool near = D.live[h];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      D.p[d][h] = D.live[h] ? x[d * n + D.id[h]] : 0;
      const double reach = B.max_half[d] + S.radius * (1 + 1e-5) + (M.pmax[d] - M.pmin[d]);
      const double from = D.p[d][h] - B.origin[d];
      near = near && from >= -reach && from <= B.extent[d] + reach;  // (false for a NaN)
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (near) {
        lo[d] = fmin(lo[d], D.p[d][h]);
        hi[d] = fmax(hi[d], D.p[d][h]);
      } else {
        D.p[d][h] = -FAR;
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int o = 16 / PER; o > 0; o >>= 1) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      boxes[wid][d] = lo[d];
      boxes[wid][3 + d] = hi[d];
    }
  }
  __syncthreads();
  bool any = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double bl = INFINITY, bh = -INFINITY;
#pragma unroll
    for (int w = 0; w < BW; ++w) {
      bl = fmin(bl, boxes[w][d]);
      bh = fmax(bh, boxes[w][3 + d]);
    }
    any = bl <= bh;
    X.c[d] = any ? 0.5 * (bl + bh) : 0;
    X.h[d] = any ? 0.5 * (bh - bl) + 1e-5 * S.radius : 0;
    const bool have = lo[d] <= hi[d];
    X.mid[d] = have ? (float)((0.5 * (lo[d] + hi[d]) - X.c[d]) * S.inv_radius) : 0;
    X.hf[d] = have ? near_half(0.5 * (hi[d] - lo[d]), X.h[d], S.inv_radius) : -1e30f;
  }
  return any;
}

// Adds up the sums of the warps that shared a tile (after evaluate_...):
// v[k][0] of every lane; the first warp's lanes get the totals.
template <int N, int PER, class Stage>
__device__ __forceinline__ void share_sums(Stage &S, double (&v)[N][PER]) {
  double *part = reinterpret_cast<double *>(&S.e[0][0][0]);
  const int tid = threadIdx.x;
  static_assert(sizeof(S.e) >= N * CHUNK_N * sizeof(double), "partial sums fit the staging");
#pragma unroll
  for (int k = 0; k < N; ++k) part[k * CHUNK_N + tid] = v[k][0];
  __syncthreads();
  if (tid < 32) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int w = 1; w < BW; ++w) v[k][0] += part[k * CHUNK_N + 32 * w + tid];
  }
}

// particles below which a block takes 32 (its warps share them) instead of 128:
// with 128 the blocks would leave SMs empty
constexpr long long SHARE_PARTICLES = 148 * CHUNK_N;

}  // namespace prt_dep
