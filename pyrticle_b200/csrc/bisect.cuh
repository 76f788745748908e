// bisect.cuh -- recursive bisection of points into compact tiles (host).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
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

// The same without a width limit, on the host's cores: the parts are split in
// turn until there are some for every thread, then each is bisected by one
// (the cuts depend only on the points).
inline void bisect_parallel(const double *P, std::vector<uint32_t> &idx, uint32_t g) {
  struct Part {
    uint32_t b, e;
  };
  const unsigned threads = std::min(16u, std::max(1u, std::thread::hardware_concurrency()));
  std::vector<Part> parts{{0u, (uint32_t)idx.size()}};
  while (parts.size() < 4 * threads) {
    auto big = std::max_element(parts.begin(), parts.end(), [](const Part &x, const Part &y) {
      return x.e - x.b < y.e - y.b;
    });
    const Part t = *big;
    const uint32_t nl = t.e - t.b > 4096 ? bisect_once(P, idx, t.b, t.e, g, 0.0) : 0;
    if (!nl) break;
    *big = {t.b, t.b + nl};
    parts.push_back({t.b + nl, t.e});
  }
  if (parts.size() == 1) {
    bisect(P, idx, parts[0].b, parts[0].e, g, 0.0, nullptr);
    return;
  }
  std::vector<std::thread> pool;
  for (unsigned w = 0; w < threads; ++w)
    pool.emplace_back([&, w] {
      for (size_t i = w; i < parts.size(); i += threads)
        bisect(P, idx, parts[i].b, parts[i].e, g, 0.0, nullptr);
    });
  for (std::thread &t : pool) t.join();
}

}  // namespace prt_dep
