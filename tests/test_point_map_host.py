"""PointMap (csrc/point_map.cuh) compiled for the host: every point of a frame belongs
to one thread, and no thread, those of the table's spare tiles included, to a point
outside the frame, also for frames of nearly 2^31 points."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <climits>
#include <cstdint>
#include <cstdio>
#include <vector>
#include "point_map.cuh"
using cpetgb::PointMap;
#define CHECK(x) if (!(x)) { std::printf("line %d: %s (P %d S %d PPT %d)\n", __LINE__, #x, P, S, PPT); return 1; }

// Threads that a launch starts for the frame: its tiles of 128, spare ones included.
template <int PPT>
static int64_t started(int P) {
  const int64_t t = (int64_t(P) + PPT - 1) / PPT + 64;
  return (t + 127) / 128 * 128;
}

template <int PPT>
static int small(int P, int S) {
  PointMap m;
  m.set<PPT>(S, P);
  std::vector<int> owners(P, 0);
  CHECK(m.threads<PPT>() % 32 == 0 && m.threads<PPT>() <= started<PPT>(P));
  for (int u = 0; u < started<PPT>(P); ++u)
    for (int k = 0; k < PPT; ++k) {
      const int p = m.point<PPT>(u, k);
      CHECK(p >= -1 && p < P);
      if (p >= 0) {
        ++owners[p];
        CHECK(u < m.threads<PPT>());
        CHECK(!m.column(u) || p % S == m.point<PPT>(u, 0) % S);
      }
    }
  for (int p = 0; p < P; ++p) CHECK(owners[p] == 1);
  return 0;
}

// The last tiles of a large frame.
template <int PPT>
static int large(int P, int S) {
  PointMap m;
  m.set<PPT>(S, P);
  const int64_t lat = S ? int64_t(P) / S / PPT * S : 0, lat_end = (lat + 31) / 32 * 32, others = P - lat * PPT;
  const int64_t threads = lat_end + (others + 32 * PPT - 1) / (32 * PPT) * 32;
  CHECK(threads <= started<PPT>(P));
  CHECK(m.threads<PPT>() == threads);
  std::vector<char> owned(4096, 0);
  for (int64_t u = started<PPT>(P) - 3000; u < started<PPT>(P); ++u)
    for (int k = 0; k < PPT; ++k) {
      const int p = m.point<PPT>(int(u), k);
      CHECK(p >= -1 && p < P);
      if (p >= 0 && P - p <= 4096) ++owned[P - 1 - p];
    }
  const int64_t tail = others < 1000 ? others : 1000;  // (points of columns have their groups elsewhere)
  for (int64_t i = 0; i < tail; ++i) CHECK(owned[i] == 1);
  return 0;
}

template <int PPT>
static int all() {
  for (int P : {1, 2, 31, 32, 33, 127, 128, 129, 1000, 1331, 4096, 9261, 9262})
    for (int S : {0, 1, 3, 11, 121, 441})
      if ((S == 0 || P % S == 0) && small<PPT>(P, S)) return 1;
  for (int d : {0, 1, 5, 126, 127, 128, 254, 255, 256, 257, 1000, 2047, 2048, 4000})
    if (large<PPT>(INT_MAX - d, 0)) return 1;
  for (int S : {16384, 441, 1024})
    for (int d : {0, 1, 3})
      if (large<PPT>((INT_MAX / S - d) * S, S)) return 1;
  return 0;
}

int main() { return all<4>() || all<8>(); }
"""


def test_every_point_has_one_thread(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("needs g++")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "pycpet_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
