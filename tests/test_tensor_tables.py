"""The ranges the tensor-core Poseidon2 form relies on, checked where its tables
are built (p2_tc_tables.cu, compiled here for the host): with both fields'
diagonals every sum fits and no output of a stage can leave its range; sums of
larger coefficients are refused.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "pico_b200" / "csrc"

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "p2_tc_tables.cu"
using namespace pico;
template <class F>
static bool field(const uint32_t (&d)[16], double* used) {
  uint32_t ext[8][16], inte[24] = {0}, diag[16];
  for (auto& r : ext) for (auto& x : r) x = (uint32_t)rand() % F::P;
  for (int r = 0; r < F::ROUNDS_P; r++) inte[r] = (uint32_t)rand() % F::P;
  for (int j = 0; j < 16; j++) diag[j] = Fp<F>::to_monty(d[j]);
  std::vector<uint8_t> tables(kTcTableBytes);
  std::vector<uint32_t> lane(kLaneWords);
  P2TcConstants c;
  const bool ok = build_p2_tc_tables(F::ID, ext, inte, diag, tables.data(), &c, lane.data());
  double sum = 0;
  for (int k = 0; k < kTcBlock - 1; k++) sum += c.beta[k] < 0 ? -(double)c.beta[k] : (double)c.beta[k];
  *used = (sum * 0.75 * F::P + F::P) / 9223372036854775808.0;
  return ok;
}
int main() {
  const uint32_t k = KoalaBear::P, b = BabyBear::P;
  const uint32_t kd[16] = {k - 2, 1, 2, (k + 1) >> 1, 3, 4, (k - 1) >> 1, k - 3, k - 4, k - ((k - 1) >> 8),
                           k - ((k - 1) >> 3), k - 127, (k - 1) >> 8, (k - 1) >> 3, (k - 1) >> 4, 127};
  const uint32_t bd[16] = {b - 2, 1, 2, (b + 1) >> 1, 3, 4, (b - 1) >> 1, b - 3, b - 4, b - ((b - 1) >> 8),
                           b - ((b - 1) >> 2), b - ((b - 1) >> 3), b - 15, (b - 1) >> 8, (b - 1) >> 4, 15};
  double uk, ub;
  const bool ok = field<KoalaBear>(kd, &uk), ob = field<BabyBear>(bd, &ub);
  int32_t most[8], fits[8];
  for (int j = 0; j < 8; j++) most[j] = j % 2 ? -(int32_t)(k / 2) : (int32_t)(k / 2), fits[j] = most[j] / 10 * 9;
  printf("%d %d %.3f %.3f %d %d\n", ok, ob, uk, ub, p2_tc_sums_fit(most, k), p2_tc_sums_fit(fits, k));
}
"""


def test_sums_stay_in_range(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "tables.cpp", tmp_path / "tables"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(CSRC), str(src), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    kb, bb, used_kb, used_bb, most, fits = subprocess.run([str(exe)], check=True, capture_output=True,
                                                          text=True).stdout.split()
    assert (kb, bb) == ("1", "1")
    assert float(used_kb) <= 0.5 and float(used_bb) <= 0.5
    # six products of p / 2 leave 63 bits, of 0.45 p each they do not
    assert (most, fits) == ("0", "1")
