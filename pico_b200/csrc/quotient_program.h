// What a constraint program reads and does, and from it the choice between the
// two forms of the quotient kernel (quotient.cu).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "../../include/pico_gpu.h"

namespace pico {

constexpr int kQThreads = 128;
constexpr size_t kQStagedSmem = 220 << 10;  // most shared memory per CTA of the staged form

// Of a validated program.  Lists of words read: main, preprocessed, permutation,
// each at the point and at the next row.
struct ProgramShape {
  std::vector<uint32_t> last[6];     // per column of a list: 1 + the read that read it last; 0: not read
  uint32_t words = 0;                // distinct words read
  uint64_t general = 0, staged = 0;  // instructions each form interprets, in tenths of one on base registers
  uint64_t reads = 0;                // reads in all
  uint64_t first = 0, far = 0;       // of a column not read before; of one last read more than 16 reads before
  static int list(const pico_constraint_op& o) {
    return o.op == PICO_Q_MAIN ? (int)o.b : o.op == PICO_Q_PREP ? 2 + (int)o.b : o.op == PICO_Q_PERM ? 4 + (int)o.b : -1;
  }
  ProgramShape(const pico_constraint_op* program, uint32_t n_ops, uint32_t main_w, uint32_t prep_w, uint32_t perm_cols) {
    for (int l = 0; l < 6; l++) last[l].assign(l < 2 ? main_w : l < 4 ? prep_w : perm_cols, 0);
    for (uint32_t k = 0; k < n_ops; k++) {
      const pico_constraint_op& o = program[k];
      const int l = list(o);
      if (l >= 0) {
        uint32_t& at = last[l][o.a];
        if (!at) {
          first++;
          words += l < 4 ? 1 : 4;
        } else if (reads + 1 - at > 16) {
          far++;
        }
        at = (uint32_t)++reads;
        general += 10;
        continue;
      }
      switch (o.op) {
        case PICO_Q_FIRST: case PICO_Q_LAST: case PICO_Q_TRANSITION: general += 10; break;
        case PICO_Q_ASSERT: {
          general += 10;
          const uint32_t before = k ? program[k - 1].op : 0u;  // an assertion just after its value's instruction joins it
          if (!((before == PICO_Q_ADD || before == PICO_Q_SUB || before == PICO_Q_MUL) && program[k - 1].dst == o.a))
            staged += 10;
          break;
        }
        case PICO_Q_EADD: case PICO_Q_ESUB: case PICO_Q_EMUL: case PICO_Q_EMB: case PICO_Q_EMULB: case PICO_Q_CHALLENGE:
        case PICO_Q_REGIONAL: case PICO_Q_EASSERT: general += 17, staged += 20; break;
        default: general += 10, staged += 10;
      }
    }
  }
  // Whether the staged form is the faster one.  row_words: a bound on the words of
  // a thread's row; ctas: of the launch; bytes: of the traces' rows it covers; sms.
  //
  // The costs, in 0.1 ns (instructions in tenths times ns per instruction and SM,
  // n CTAs an SM): a CTA alone takes about 280 ns per instruction in either form.
  // In the general form, whose registers are few, twelve share an SM, and n take
  // 43 n + 140.  In the staged form a row's words bound the CTAs of an SM (r):
  // ceil(n / r) rounds of 280, at best 55 n + 225.  It interprets fewer instructions
  // (no reads, no selectors, assertions joined to their values), an extension one
  // costs it 2 (the general form 1.7), a word to stage 1/4.  From 2.2 times the L2 on
  // the general form's first read of a column costs up to 3 instructions more, a
  // read of one that was read long before half as much again.
  // Measured (KoalaBear, us, call included, general / staged; c columns read at
  // both rows, 8 c instructions): 2^18 points, c = 60 (r = 3) 449 / 354, 100 (2) 674 /
  // 722, 200 (1) 1,339 / 2,810; 2^19 points 75 (2) 807 / 932; 2^20 points 60 1,214 / 1,095,
  // 200 7,617 / 11,450; 2^15 points 100 293 / 181; 40 columns and 20 extension ones,
  // 2^18 points 539 / 1,177; 100 columns with 1,200 more reads at random, 2^20 points
  // 24,350 / 8,870.  (The staged form for every row that fits was up to 2.8 times
  // slower than the general one.)
  bool prefer_staged(uint32_t row_words, uint64_t ctas, uint64_t bytes, uint32_t sms) const {
    const size_t smem = (size_t)(row_words | 1u) * kQThreads * 4;
    if (smem > kQStagedSmem) return false;
    constexpr uint64_t kSmemPerSm = 228 << 10, kSmemPerCta = 1 << 10, kMostCtas = 12, kL2 = 126 << 20;
    const uint64_t r = std::min<uint64_t>(kMostCtas, kSmemPerSm / (smem + kSmemPerCta));
    const uint64_t n = (ctas + sms - 1) / sms;
    const uint64_t extra = bytes <= kL2 * 11 / 5 ? 0 : std::min<uint64_t>(30, 15 * (bytes - kL2 * 11 / 5) / kL2);
    const uint64_t cost_general =
        (general + extra * (first + far + far / 2)) * std::max<uint64_t>(280, 43 * n + 140);
    const uint64_t cost_staged = (staged + words * 5 / 2) * std::max<uint64_t>(280 * ((n + r - 1) / r), 55 * n + 225);
    return cost_staged <= cost_general / 20 * 19;  // where they are equal, the general form
  }
};

}  // namespace pico
