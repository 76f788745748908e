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
// With u the target and w the source relative to the block's centre,
//   a - r^2/a = (a - |u|^2/a) - |w|^2/a + (2/a) u.w = B + e + V.w,
// three multiply-adds and an add per pair.
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

// The weight (t)^alpha for t > 0, else 0.
template <bool ALPHA2>
__device__ __forceinline__ double shape_power(double t, double alpha) {
  if (ALPHA2) {
    const double r = relu(t);
    return r * r;
  }
  return t > 0 ? pow(t, alpha) : 0.0;
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

// Candidate segments of one warp: runs of consecutive particles in bin order.
// At most SEGS per turn of 32 bin rows: a row falls into at most four pieces
// along a periodic x (a tile no wider than the period, a radius below half).
struct Segments {
  static constexpr int PIECES = 4, SEGS = 32 * PIECES;
  uint32_t cum[SEGS + 1];  // candidates before the segment
  uint32_t start[SEGS];    // its first bin-order particle
  double shift[SEGS][3];   // from a particle's position to the tile's frame
};

// Walks the particles of the bin rows within `radius` of the box c +- hf, 32
// at a time: visit(valid, k, w0, w1, w2, q) on all lanes, with w relative to c
// (periodic image included). Warps part of `parts` takes every parts-th batch.
// The rows are laid out 32 at a time, one per lane, and their particles
// numbered through, so that short rows fill the lanes together; the next
// batch's particles are loaded before the present one is visited (`q` is the
// payload's charge).
template <class Visit>
__device__ __forceinline__ void stream_particles(const BinGrid &G, const DepParticles &P,
                                                 const double c[3], const double hf[3],
                                                 double radius, Segments &S, int part,
                                                 int parts, Visit &&visit) {
  const int lane = threadIdx.x & 31;
  const double rr = radius * (1 + 1e-5), rr2 = rr * rr;
  int ulo[3], uhi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    ulo[d] = bin_floor(G, d, c[d] - hf[d] - rr);
    uhi[d] = bin_floor(G, d, c[d] + hf[d] + rr);
    if (G.periodic[d]) {
      ulo[d] -= 1;
      uhi[d] += 1;
    } else {
      ulo[d] = max(ulo[d], 0);
      uhi[d] = min(uhi[d], G.dims[d] - 1);
    }
  }
  const double2 *__restrict__ pay = reinterpret_cast<const double2 *>(P.payload);
  auto slab_gap = [&](int d, double blo) {
    const double e =
        fmax(0.0, fmax(blo - (c[d] + hf[d]), (c[d] - hf[d]) - (blo + G.w[d]))) - G.slack[d];
    return e > 0 ? e * e : 0.0;
  };
  const int ny = max(0, uhi[1] - ulo[1] + 1), nz = max(0, uhi[2] - ulo[2] + 1);
  const long long nrows = (long long)ny * nz;
  for (long long r0 = 0; r0 < nrows; r0 += 32) {
    const long long r = r0 + lane;
    uint32_t s_start[Segments::PIECES], s_len[Segments::PIECES];
    int s_q[Segments::PIECES];
    int cnt = 0;
    uint32_t mine = 0;
    int qz = 0, qy = 0;
    if (r < nrows) {
      const int bz = ulo[2] + (int)(r / ny), by = ulo[1] + (int)(r % ny);
      int wz = bz, wy = by;
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
        int bx0 = bin_floor(G, 0, c[0] - hf[0] - rem);
        int bx1 = bin_floor(G, 0, c[0] + hf[0] + rem);
        if (G.periodic[0]) {
          bx0 -= 1;
          bx1 += 1;
        }
        bx0 = max(bx0, ulo[0]);
        bx1 = min(bx1, uhi[0]);
        const long long row = (long long)G.dims[0] * (wy + (long long)G.dims[1] * wz);
        int bx = bx0;
#pragma unroll
        for (int i = 0; i < Segments::PIECES; ++i) {
          if (bx <= bx1) {
            int wx = bx, q = 0, end = bx1;
            if (G.periodic[0]) {
              q = floor_div(bx, G.dims[0]);
              wx = bx - q * G.dims[0];
              end = min(bx1, (q + 1) * G.dims[0] - 1);
            }
            s_start[i] = P.starts[row + wx];
            s_len[i] = P.starts[row + wx + (end - bx) + 1] - s_start[i];
            s_q[i] = q;
            mine += s_len[i];
            cnt = i + 1;
            bx = end + 1;
          }
        }
      }
    }
    // place the segments: exclusive scans of their number and candidates
    int ns = cnt;
    uint32_t nc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ns, o);
      const uint32_t b = __shfl_up_sync(0xffffffffu, nc, o);
      if (lane >= o) {
        ns += a;
        nc += b;
      }
    }
    const int segs = __shfl_sync(0xffffffffu, ns, 31);
    const uint32_t total = __shfl_sync(0xffffffffu, nc, 31);
    if (total == 0) continue;
    __syncwarp();
    {
      int at = ns - cnt;
      uint32_t before = nc - mine;
#pragma unroll
      for (int i = 0; i < Segments::PIECES; ++i)
        if (i < cnt) {
          S.cum[at] = before;
          S.start[at] = s_start[i];
          S.shift[at][0] = s_q[i] * G.period[0] - c[0];
          S.shift[at][1] = qy * G.period[1] - c[1];
          S.shift[at][2] = qz * G.period[2] - c[2];
          before += s_len[i];
          ++at;
        }
      if (lane == 31) S.cum[segs] = total;
    }
    __syncwarp();
    int sg = 0;
    uint32_t k = 0;
    double2 xy = make_double2(0, 0), zq = make_double2(0, 0);
    int seg = 0;
    auto load = [&](uint32_t f) {
      if (f < total) {
        while (f >= S.cum[sg + 1]) ++sg;
        seg = sg;
        k = S.start[sg] + (f - S.cum[sg]);
        xy = pay[4 * (size_t)k];
        zq = pay[4 * (size_t)k + 1];
      }
    };
    uint32_t b = 32u * part;
    load(b + lane);
    for (; b < total; b += 32u * parts) {
      const bool valid = b + lane < total;
      const uint32_t k0 = k;
      const double w0 = xy.x + S.shift[seg][0], w1 = xy.y + S.shift[seg][1],
                   w2 = zq.x + S.shift[seg][2], q = zq.y;
      load(b + 32u * parts + lane);
      visit(valid, k0, w0, w1, w2, q);
    }
    __syncwarp();
  }
}

// Whether a source at w (relative to the centre of a box with half extents hf,
// grown by 1e-5 radii) may lie within the radius of the box; rc4 = 4 radius^2,
// grown likewise. Per axis 2 max(|w| - hf, 0) = d + |d|. It only chooses what
// is evaluated: FP32 on the FP64 offsets, with the margin above its rounding.
__device__ __forceinline__ bool near_box(double w0, double w1, double w2, const float hf[3],
                                         float rc4) {
  const float d0 = fabsf((float)w0) - hf[0], d1 = fabsf((float)w1) - hf[1],
              d2 = fabsf((float)w2) - hf[2];
  const float e0 = d0 + fabsf(d0), e1 = d1 + fabsf(d1), e2 = d2 + fabsf(d2);
  return e0 * e0 + e1 * e1 + e2 * e2 <= rc4;
}

__device__ __forceinline__ float near_limit(double radius) {
  const float r = (float)(radius * (1 + 1e-5));
  return 4.0f * r * r;
}

// ------------------------------------------------ four tiles per block

constexpr int BW = 4;          // warps, tiles per block
constexpr int CHUNK_N = 32 * BW;

// Staging of one block: three chunks of entries, W 16-byte words each
// ((w0, w1), (w2, e), values), word by word; entry CHUNK_N lies beyond every
// radius. A record (x, y, z, values) is copied to the same place and moved
// into the block's frame there by the thread that copied it.
template <int NV>
struct BlockStage {
  static constexpr int W = 2 + (NV + 1) / 2, RAW = (3 + NV + 1) / 2, STAGES = 3;
  double2 e[STAGES][W][CHUNK_N + 1];
  float4 w[STAGES][CHUNK_N];  // the entries' positions, for the choice
  uint32_t cum[CHUNK_N + 1];  // sources before the segment
  uint32_t start[CHUNK_N];    // its first record
  double shift[CHUNK_N][3];   // from a record's position to the block's frame
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

template <int NV>
__device__ __forceinline__ void stage_begin(BlockStage<NV> &S) {
  using ST = BlockStage<NV>;
  if (threadIdx.x < ST::STAGES * ST::W) {
    const int st = threadIdx.x / ST::W, w = threadIdx.x % ST::W;
    S.e[st][w][CHUNK_N] = make_double2(0, w == 1 ? -1e300 : 0);
  }
}

// Evaluates the `total` sources of the present segments (S.cum, S.start,
// S.shift; written before a barrier) against the block's tiles:
// op(w0, w1, w2, e, v) on every lane with its group's entry. mid, hf: this
// warp's tile box in the block's frame, grown as near_box wants it; a warp
// without a tile passes hf < 0 with a magnitude that keeps everything out.
// Returns the entries evaluated (per warp). Ends with a barrier.
template <int PER, int NV, class Op>
__device__ __forceinline__ uint32_t evaluate_segments(BlockStage<NV> &S,
                                                      const double2 *__restrict__ records,
                                                      uint32_t total, const float mid[3],
                                                      const float hf[3], float rc4,
                                                      double inv_radius, Op &&op) {
  using ST = BlockStage<NV>;
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
      double v[2 * ST::RAW];
#pragma unroll
      for (int w = 0; w < ST::RAW; ++w) {
        const double2 t = S.e[st][w][tid];
        v[2 * w] = t.x;
        v[2 * w + 1] = t.y;
      }
      const double w0 = v[0] + S.shift[seg0][0], w1 = v[1] + S.shift[seg0][1],
                   w2 = v[2] + S.shift[seg0][2];
      S.w[st][tid] = make_float4((float)w0, (float)w1, (float)w2, 0);
      S.e[st][0][tid] = make_double2(w0, w1);
      S.e[st][1][tid] = make_double2(w2, -(w0 * w0 + w1 * w1 + w2 * w2) * inv_radius);
#pragma unroll
      for (int w = 2; w < ST::W; ++w)
        S.e[st][w][tid] =
            make_double2(v[2 * w - 1], 2 * w < 3 + NV ? v[2 * w < 2 * ST::RAW ? 2 * w : 0] : 0.0);
    } else {
      S.w[st][tid] = make_float4(1e30f, 0, 0, 0);
    }
    // chunk k is in place, chunk k - 1 done with: its stage takes chunk k + 2
    __syncthreads();
    copy(k + 2);
    seg0 = seg1;
    seg1 = seg;
    int n = 0;
#pragma unroll
    for (int q = 0; q < BW; ++q) {
      const float4 w = S.w[st][32 * q + lane];
      const float d0 = fabsf(w.x - mid[0]) - hf[0], d1 = fabsf(w.y - mid[1]) - hf[1],
                  d2 = fabsf(w.z - mid[2]) - hf[2];
      const float e0 = d0 + fabsf(d0), e1 = d1 + fabsf(d1), e2 = d2 + fabsf(d2);
      const bool in = e0 * e0 + e1 * e1 + e2 * e2 <= rc4;
      const unsigned bal = __ballot_sync(0xffffffffu, in);
      if (in) list[n + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)(32 * q + lane);
      n += __popc(bal);
    }
    // up to a whole turn with entries beyond every radius
    if (lane < PER) list[n + lane] = CHUNK_N;
    __syncwarp();
    evaluated += n;
    int id = list[grp];
#pragma unroll 2
    for (int i = 0; i < n; i += PER) {
      const int cur = id;
      id = list[i + PER + grp];
      const double2 w01 = S.e[st][0][cur], w2e = S.e[st][1][cur];
      double v[2 * (ST::W - 2)];
#pragma unroll
      for (int w = 2; w < ST::W; ++w) {
        const double2 t = S.e[st][w][cur];
        v[2 * w - 4] = t.x;
        v[2 * w - 3] = t.y;
      }
      op(w01.x, w01.y, w2e.x, w2e.y, v);
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  return evaluated;
}

// The boxes of a block's tiles: the block's centre c and half extents, and
// this warp's tile box in the block's frame (mid, hf with the FP32 margin).
struct BlockBox {
  double c[3], h[3];
  float mid[3], hf[3];
};

// All particles of the bin rows near the block's box, evaluated against its
// tiles (evaluate_segments).
template <int PER, int NV, class Op>
__device__ __forceinline__ uint32_t evaluate_particles(BlockStage<NV> &S, const BinGrid &G,
                                                       const DepParticles &P, const BlockBox &X,
                                                       double radius, double inv_radius,
                                                       Op &&op) {
  const int tid = threadIdx.x;
  const double rr = radius * (1 + 1e-5), rr2 = rr * rr;
  const float rc4 = near_limit(radius);
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
  // a row falls into at most four pieces along a periodic x (a block no wider
  // than the period, a radius below half), else it is one
  const int pieces = G.periodic[0] ? 4 : 1;
  const int turn = CHUNK_N / pieces;
  uint32_t evaluated = 0;
  for (long long r0 = 0; r0 < nrows; r0 += turn) {
    const int slot = tid / pieces, piece = tid % pieces;
    const long long r = r0 + slot;
    uint32_t start = 0, len = 0;
    double sh[3] = {0, 0, 0};
    if (slot < turn && r < nrows) {
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
    evaluated += evaluate_segments<PER, NV>(S, reinterpret_cast<const double2 *>(P.payload), total,
                                            X.mid, X.hf, rc4, inv_radius, op);
  }
  return evaluated;
}

}  // namespace prt_dep
