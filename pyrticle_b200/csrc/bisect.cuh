// bisect.cuh -- recursive bisection of points into compact tiles (host).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <exception>
#include <mutex>
#include <numeric>
#include <thread>
#include <vector>

namespace prt_dep {

// Splits the points idx[b, e) along the longest axis of their box, at a
// multiple of g rows (so that all parts but the last of a branch hold exactly
// g), unless they are a final part: at most g points and, when wmax > 0, at
// most wmax wide along every axis. Returns the left part's size, or 0.
inline uint32_t bisect_once(const double *P, std::vector<uint32_t> &idx, uint32_t b, uint32_t e,
                            uint32_t g, double wmax) {
  const uint32_t n = e - b;
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t i = b; i < e; ++i)
    for (int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], P[3 * (size_t)idx[i] + a]);
      hi[a] = std::max(hi[a], P[3 * (size_t)idx[i] + a]);
    }
  int ax = 0;
  for (int a = 1; a < 3; ++a)
    if (hi[a] - lo[a] > hi[ax] - lo[ax]) ax = a;
  const bool wide = wmax > 0 && hi[ax] - lo[ax] > wmax;
  if (n <= 1 || (n <= g && !wide)) return 0;
  uint32_t nl;
  if (n > g) {
    nl = g * std::max<uint32_t>(1, (uint32_t)std::lround((double)n / (2.0 * g)));
    if (nl >= n) nl = g * ((n - 1) / g);
  } else {
    nl = n / 2;
  }
  std::nth_element(idx.begin() + b, idx.begin() + b + nl, idx.begin() + e,
                   [&](uint32_t x, uint32_t y) {
                     const double px = P[3 * (size_t)x + ax], py = P[3 * (size_t)y + ax];
                     return px != py ? px < py : x < y;
                   });
  return nl;
}

// Recursive bisection of idx[b, e) into final parts (bisect_once); their
// starts are appended to `cuts` when given, depth first: neighbouring parts
// are neighbours in space.
inline void bisect(const double *P, std::vector<uint32_t> &idx, uint32_t b, uint32_t e,
                   uint32_t g, double wmax, std::vector<uint32_t> *cuts) {
  struct Part {
    uint32_t b, e;
  };
  std::vector<Part> stack{{b, e}};
  while (!stack.empty()) {
    const Part t = stack.back();
    stack.pop_back();
    const uint32_t nl = bisect_once(P, idx, t.b, t.e, g, wmax);
    if (!nl) {
      if (cuts) cuts->push_back(t.b);
      continue;
    }
    stack.push_back({t.b + nl, t.e});
    stack.push_back({t.b, t.b + nl});
  }
}

// f(w) for w = 0 .. n - 1 on host threads; those that cannot be started run
// here. The first exception of an f is thrown here once all have ended.
template <class F>
inline void on_threads(unsigned n, F &&f) {
  std::exception_ptr failed;
  std::mutex mutex;
  auto run = [&](unsigned w) {
    try {
      f(w);
    } catch (...) {
      std::lock_guard<std::mutex> lock(mutex);
      if (!failed) failed = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(n);
  unsigned w = 0;
  try {
    for (; w + 1 < n; ++w) pool.emplace_back(run, w);
  } catch (...) {  // no (more) threads
  }
  for (; w < n; ++w) run(w);
  for (std::thread &t : pool) t.join();
  if (failed) std::rethrow_exception(failed);
}

inline unsigned host_threads() {
  return std::min(16u, std::max(1u, std::thread::hardware_concurrency()));
}

// The same without a width limit, on the host's cores: the parts are split,
// all of a level at a time, until there are some for every thread, then each is
// bisected by one (the cuts depend only on the points).
inline void bisect_parallel(const double *P, std::vector<uint32_t> &idx, uint32_t g) {
  struct Part {
    uint32_t b, e;
  };
  const unsigned threads = host_threads();
  std::vector<Part> parts{{0u, (uint32_t)idx.size()}};
  while (parts.size() < 4 * threads) {
    std::vector<uint32_t> left(parts.size());
    const unsigned n = (unsigned)std::min<size_t>(threads, parts.size());
    on_threads(n, [&](unsigned w) {
      for (size_t i = w; i < parts.size(); i += n)
        left[i] = parts[i].e - parts[i].b > 4096
                      ? bisect_once(P, idx, parts[i].b, parts[i].e, g, 0.0)
                      : 0;
    });
    std::vector<Part> next;
    for (size_t i = 0; i < parts.size(); ++i) {
      const Part t = parts[i];
      if (left[i]) next.push_back({t.b, t.b + left[i]});
      next.push_back({t.b + left[i], t.e});
    }
    if (next.size() == parts.size()) break;
    parts.swap(next);
  }
  const unsigned n = (unsigned)std::min<size_t>(threads, parts.size());
  on_threads(n, [&](unsigned w) {
    for (size_t i = w; i < parts.size(); i += n)
      bisect(P, idx, parts[i].b, parts[i].e, g, 0.0, nullptr);
  });
}

// The host points [count][3] cut into tiles of exactly `tile` (the last one
// partial), in blocks of `block` points (a multiple of it) first, so that a
// block's tiles lie together: the point of each row, the rows' points, and per
// tile centre and half extents of its box.
inline void cut_tiles(const double *points, size_t count, uint32_t tile, uint32_t block,
                      std::vector<uint32_t> &rows, std::vector<double> &pos,
                      std::vector<double> &boxes) {
  const size_t tiles = (count + tile - 1) / tile, blocks = (count + block - 1) / block;
  rows.resize(count);
  pos.resize(3 * count);
  boxes.resize(6 * tiles);
  std::iota(rows.begin(), rows.end(), 0u);
  bisect_parallel(points, rows, block);
  const unsigned n = (unsigned)std::min<size_t>(host_threads(), blocks / 64 + 1);
  on_threads(n, [&](unsigned w) {
    for (size_t b = blocks * w / n; b < blocks * (w + 1) / n; ++b) {
      const size_t r1 = std::min(count, (b + 1) * block);
      bisect(points, rows, (uint32_t)(b * block), (uint32_t)r1, tile, 0.0, nullptr);
      for (size_t r0 = b * block; r0 < r1; r0 += tile) {
        double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (size_t r = r0; r < std::min(r1, r0 + tile); ++r)
          for (int a = 0; a < 3; ++a) {
            const double x = points[3 * (size_t)rows[r] + a];
            pos[3 * r + a] = x;
            lo[a] = std::min(lo[a], x);
            hi[a] = std::max(hi[a], x);
          }
        for (int a = 0; a < 3; ++a) {
          boxes[6 * (r0 / tile) + a] = 0.5 * (lo[a] + hi[a]);
          boxes[6 * (r0 / tile) + 3 + a] = 0.5 * (hi[a] - lo[a]);
        }
      }
    }
  });
}

}  // namespace prt_dep
