"""The cut of points into tiles (csrc/bisect.cuh) on host threads, compiled
here for the host alone: the cuts depend only on the points, and a process that
cannot start (all) the threads does their work itself. Without that the
exception of a thread that did not start ended the program in the C entry that
made a mesh or deposited onto a grid."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "pyrticle_b200" / "csrc"

PROGRAM = r"""
#include "bisect.cuh"
#include <cstdio>
#include <cstdlib>
#include <dlfcn.h>
#include <new>
#include <pthread.h>
#include <random>

static int allowed = -1, started = 0;  // threads that may start, -1: any
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
  static auto real = (decltype(&pthread_create))dlsym(RTLD_NEXT, "pthread_create");
  if (allowed >= 0 && started >= allowed) return 11;  // EAGAIN
  ++started;
  return real(t, a, f, x);
}

struct Cut {
  std::vector<uint32_t> rows;
  std::vector<double> pos, boxes;
};

static Cut cut(const std::vector<double> &P, int threads) {
  allowed = threads;
  started = 0;
  Cut c;
  prt_dep::cut_tiles(P.data(), P.size() / 3, 32, 128, c.rows, c.pos, c.boxes);
  return c;
}

int main(int, char **argv) {
  const size_t n = std::atoll(argv[1]);
  std::mt19937 rng(1);
  std::uniform_real_distribution<double> u(0, 1);
  std::vector<double> P(3 * n);
  for (size_t i = 0; i < n; ++i) {
    P[3 * i] = std::floor(u(rng) * 16) / 16;  // a lattice's equal coordinates too
    P[3 * i + 1] = u(rng);
    P[3 * i + 2] = 4 * u(rng);
  }
  const Cut none = cut(P, 0);
  for (int threads : {-1, 1, 3}) {
    const Cut c = cut(P, threads);
    if (threads >= 0 && started > threads) return 10;
    if (c.rows != none.rows || c.pos != none.pos || c.boxes != none.boxes) return 11;
  }
  std::vector<char> seen(n, 0);
  for (size_t r = 0; r < n; ++r) {
    const uint32_t i = none.rows[r];
    if (i >= n || seen[i]++) return 12;
    for (int a = 0; a < 3; ++a) {
      const double *b = &none.boxes[6 * (r / 32) + a];
      if (none.pos[3 * r + a] != P[3 * i + a]) return 13;
      if (std::fabs(P[3 * i + a] - b[0]) > b[3] * (1 + 1e-14) + 1e-15) return 14;
    }
  }
  if (none.boxes.size() != 6 * ((n + 31) / 32)) return 15;
  // an exception on a thread is thrown to the caller, after all have ended
  allowed = -1;
  int ended = 0;
  std::mutex m;
  try {
    prt_dep::on_threads(4, [&](unsigned w) {
      if (w == 1) throw std::bad_alloc();
      std::lock_guard<std::mutex> lock(m);
      ++ended;
    });
    return 16;
  } catch (const std::bad_alloc &) {
    if (ended != 3) return 17;
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("cuts")
    (d / "cuts.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-x", "c++", "cuts.cpp", "-o",
                    "cuts", "-pthread", "-ldl"], cwd=d, check=True)
    return d / "cuts"


@pytest.mark.parametrize("points", [1, 31, 32, 128, 129, 5000, 100_003])
def test_cuts_do_not_depend_on_the_threads(program, points):
    assert subprocess.run([str(program), str(points)], timeout=60).returncode == 0
