"""The rule that chooses the quotient kernel's form (quotient_program.h, compiled
for the host), at programs and sizes where both forms were timed: the staged
form only where it is the faster one.  It used to take every program whose rows
fit in shared memory, up to 2.8 times slower than the general form.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "quotient_program.h"
using namespace pico;
using Ops = std::vector<pico_constraint_op>;
// c columns at both rows, 8 c instructions; `reps` more constraints over random columns; ext running sums
static Ops program(uint32_t c, uint32_t reps, uint32_t ext) {
  Ops p;
  for (uint32_t i = 0; i < c; i++)
    for (pico_constraint_op o : {pico_constraint_op{PICO_Q_TRANSITION, 0, 0, 0}, {PICO_Q_MAIN, 1, i, 1}, {PICO_Q_MAIN, 2, i, 0},
                                 {PICO_Q_MAIN, 3, (i + 1) % c, 0}, {PICO_Q_MUL, 2, 2, 3}, {PICO_Q_SUB, 1, 1, 2},
                                 {PICO_Q_MUL, 0, 0, 1}, {PICO_Q_ASSERT, 0, 0, 0}})
      p.push_back(o);
  for (uint32_t i = 0; i < reps; i++) {
    for (uint32_t d = 0; d < 3; d++) p.push_back({PICO_Q_MAIN, d, (uint32_t)rand() % c, 0});
    for (pico_constraint_op o : {pico_constraint_op{PICO_Q_MUL, 0, 0, 1}, {PICO_Q_SUB, 0, 0, 2}, {PICO_Q_ASSERT, 0, 0, 0}}) p.push_back(o);
  }
  for (uint32_t i = 0; i < ext; i++)
    for (pico_constraint_op o : {pico_constraint_op{PICO_Q_PERM, 0, i, 0}, {PICO_Q_PERM, 1, i, 1}, {PICO_Q_ESUB, 1, 1, 0},
                                 {PICO_Q_CHALLENGE, 2, 0, 0}, {PICO_Q_MAIN, 0, 0, 0}, {PICO_Q_EMB, 3, 0, 0}, {PICO_Q_EADD, 2, 2, 3},
                                 {PICO_Q_EMUL, 1, 1, 2}, {PICO_Q_MAIN, 0, 1, 0}, {PICO_Q_EMB, 3, 0, 0}, {PICO_Q_ESUB, 1, 1, 3},
                                 {PICO_Q_TRANSITION, 0, 0, 0}, {PICO_Q_EMULB, 1, 1, 0}, {PICO_Q_EASSERT, 0, 1, 0}})
      p.push_back(o);
  return p;
}
static int staged(uint32_t log_points, uint32_t c, uint32_t reps, uint32_t ext) {
  const Ops p = program(c, reps, ext);
  const ProgramShape s(p.data(), (uint32_t)p.size(), c, 0, ext);
  const uint64_t points = 1ull << log_points;
  return s.prefer_staged(s.words + 3 + 4 + 4 * (ext ? 4 : 1), (points + kQThreads - 1) / kQThreads, 4 * points * (c + 4 * ext), 148);
}
int main(int argc, char** argv) {
  for (int i = 1; i + 3 < argc; i += 4) printf("%d", staged(atoi(argv[i]), atoi(argv[i + 1]), atoi(argv[i + 2]), atoi(argv[i + 3])));
}
"""

# (log2 points, columns, further constraints, extension columns): staged?
CASES = {
    (7, 2, 0, 0): True, (7, 100, 0, 0): True, (7, 200, 0, 0): True, (12, 200, 800, 0): True, (12, 40, 0, 20): True,
    (15, 100, 0, 0): True, (15, 200, 0, 0): True, (15, 40, 0, 20): False,
    (18, 8, 8, 0): True, (18, 30, 0, 0): True, (18, 45, 0, 0): True, (18, 60, 0, 0): True, (18, 60, 400, 0): True,
    (18, 100, 0, 0): False, (18, 125, 0, 0): False, (18, 150, 400, 0): False, (18, 200, 0, 0): False,
    (18, 20, 0, 10): False, (18, 40, 0, 20): False, (18, 100, 400, 0): True,
    (19, 75, 0, 0): False, (19, 100, 0, 0): False, (20, 20, 20, 0): True, (20, 30, 120, 0): True, (20, 60, 0, 0): True,
    (20, 150, 0, 0): False, (20, 200, 0, 0): False, (20, 40, 0, 20): False,
    (20, 100, 400, 0): True, (20, 150, 400, 0): True, (20, 200, 800, 0): True,
    (12, 230, 0, 0): False, (20, 300, 0, 0): False,  # rows that do not fit
}


def test_staged_only_where_it_is_faster(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(ROOT / "pico_b200" / "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    args = [str(x) for case in CASES for x in case]
    out = subprocess.run([str(exe), *args], check=True, capture_output=True, text=True).stdout
    got = dict(zip(CASES, (ch == "1" for ch in out)))
    assert got == CASES, {k: got[k] for k in CASES if got[k] != CASES[k]}
