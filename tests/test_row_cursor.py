"""The tensor-core row hashing's walk over a row's matrices (row_cursor.cuh),
compiled for the host: every chunk of rows of several matrices, whole and
partial, and columns asked for past the last matrix, which must be counted and
read as zero without touching memory.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "row_cursor.cuh"
using namespace pico;
struct Trip {
  unsigned* n;
  void operator()(uint32_t, uint32_t) const { ++*n; }
};
// `width` columns of row r of matrices of the given widths, from chunk position pos0 on.
static int check(const std::vector<uint32_t>& widths, uint32_t width, uint32_t pos0, uint64_t r) {
  std::vector<std::vector<uint32_t>> data;
  std::vector<RowSeg> segs;
  std::vector<uint32_t> want;
  uint32_t value = 1;
  for (uint32_t w : widths) {
    data.emplace_back((r + 1) * w + 1);
    for (auto& x : data.back()) x = value++;
    segs.push_back({data.back().data(), w, 0});
    want.insert(want.end(), data.back().begin() + r * w, data.back().begin() + (r + 1) * w);
  }
  const unsigned past = width > want.size() ? width - (unsigned)want.size() : 0;
  want.resize(width, 0);
  unsigned trips = 0;
  std::vector<uint32_t> got;
  RowCursor c;
  row_cursor_begin(c, segs.data(), (uint32_t)segs.size(), r);
  const uint32_t end = pos0 + width;
  for (uint32_t base = 0; base < end; base += 8) {
    const int lo = base < pos0 ? (int)(pos0 - base) : 0, hi = end - base < 8 ? (int)(end - base) : 8;
    uint32_t v[8];
    memset(v, 0xff, sizeof v);
    row_chunk(c, segs.data(), (uint32_t)segs.size(), r, lo, hi, v, Trip{&trips});
    for (int j = 0; j < 8; j++) {
      if (j >= lo && j < hi) got.push_back(v[j]);
      else if (v[j] != 0xffffffffu) return 1;
    }
  }
  return got != want || trips != past;
}
int main() {
  int bad = 0;
  const std::vector<std::vector<uint32_t>> groups = {{1}, {7}, {8}, {9}, {16}, {3, 6, 8}, {17, 2}, {8, 8}, {40, 1, 23}, {}};
  for (const auto& g : groups) {
    uint32_t sum = 0;
    for (uint32_t w : g) sum += w;
    for (uint32_t extra : {0u, 1u, 7u, 8u, 9u, 16u, 17u, 40u})  // columns past the last matrix
      for (uint32_t pos0 : {0u, 1u, 7u})
        for (uint64_t r : {0ull, 3ull}) bad += check(g, sum + extra, pos0, r);
  }
  printf("%d\n", bad);
  return bad != 0;
}
"""


def test_chunks_stay_inside_the_rows(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "cursor.cpp", tmp_path / "cursor"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(ROOT / "pico_b200" / "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
