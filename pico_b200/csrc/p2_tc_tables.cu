// Host construction of the tensor-core Poseidon2 tables: every linear map
// between two S-box layers as byte-limb matrices (see p2_tc.cuh), from the
// round constants and the internal diagonal.  Plain 64-bit integer arithmetic
// on canonical values.
#include <cstring>
#include <initializer_list>
#include <vector>

#include "field.cuh"
#include "p2_tc_tables.h"

namespace pico {
namespace {

struct Builder {
  uint64_t p;
  uint64_t r32;      // 2^32 mod p
  uint64_t me[16][16];
  uint64_t d[16];
  uint8_t* out;

  uint64_t mul(uint64_t a, uint64_t b) const { return a * b % p; }
  // One linear step of the internal layer (the S-box output of word 0 already in s[0]).
  void internal(std::vector<uint64_t>& s) const {
    uint64_t sum = 0;
    for (int i = 0; i < 16; i++) sum = (sum + s[i]) % p;
    for (int i = 0; i < 16; i++) s[i] = (mul(d[i], s[i]) + sum) % p;
  }
  // Row n of K byte k of a K step's table.
  static uint32_t at(uint32_t N, uint32_t n, uint32_t k) { return (k / 16) * N * 16 + (n / 8) * 128 + (n % 8) * 16 + k % 16; }
  // Source word `word` (0..7) of the K step at `table`, for output i: the
  // coefficient's limbs for each of the word's bytes.  scale carries the
  // 2^16 of the recombination and the change of Montgomery form.
  void coef(uint32_t table, uint32_t N, uint32_t i, uint32_t word, uint64_t c, uint64_t scale) const {
    uint64_t v = mul(c, scale);
    for (uint32_t b = 0; b < 4; b++) {
      for (uint32_t l = 0; l < 4; l++) out[table + at(N, 4 * i + l, 4 * word + b)] = (uint8_t)(v >> (8 * l));
      v = mul(v, 256);
    }
  }
  // S-box output j of a full round: eight bytes of the product whose
  // Montgomery reduction would give the word (scale_z = scale * 2^-32).
  void coef_z(uint32_t table, uint32_t N, uint32_t i, uint32_t j, uint64_t c, uint64_t scale_z) const {
    const uint32_t step = table + (j / 4) * N * 32;
    coef(step, N, i, 2 * (j % 4), c, scale_z);
    coef(step, N, i, 2 * (j % 4) + 1, c, mul(scale_z, r32));
  }
  // Constant of output i: byte 0 of the constant word.
  void constant_step(uint32_t table, uint32_t N, uint32_t i, uint64_t v) const {
    for (uint32_t l = 0; l < 4; l++) out[table + at(N, 4 * i + l, 4 * 7)] = (uint8_t)(v >> (8 * l));
  }
  // The same in a constant column (the second core-matrix column of a K step).
  void constant_col(uint32_t col, uint32_t i, uint64_t v) const {
    for (uint32_t l = 0; l < 4; l++) {
      const uint32_t n = 4 * i + l;
      out[col + (n / 8) * 128 + (n % 8) * 16 + 12] = (uint8_t)(v >> (8 * l));
    }
  }
  // The recombined outputs of a stage: `outputs` of them, from K steps of these
  // tables and a constant column (or 0).
  struct Part {
    uint32_t table, steps;
  };
  bool limbs_fit(uint32_t N, uint32_t outputs, std::initializer_list<Part> parts, uint32_t col) const {
    for (uint32_t i = 0; i < outputs; i++) {
      uint64_t limb[4] = {0, 0, 0, 0};
      for (uint32_t l = 0; l < 4; l++) {
        for (const Part& part : parts)
          for (uint32_t s = 0; s < part.steps; s++)
            for (uint32_t k = 0; k < 32; k++) limb[l] += 255u * out[part.table + s * N * 32 + at(N, 4 * i + l, k)];
        const uint32_t n = 4 * i + l;
        if (col) limb[l] += out[col + (n / 8) * 128 + (n % 8) * 16 + 12];
      }
      if (limb[0] + (limb[1] << 8) >= (1ull << 32) || limb[2] + (limb[3] << 8) + 65535 >= p) return false;
    }
    return true;
  }
  bool all_limbs_fit(int rounds_p) const {
    const uint32_t y_steps = rounds_p > 2 * kTcBlock ? 3 : 2;  // of the state after the partial rounds
    bool fit = limbs_fit(64, 16, {{kTcFull, 4}}, kTcC + 1024 * kTcCInit) &&
               limbs_fit(64, 16, {{kTcNew, 1}}, kTcC + 1024 * kTcCInit) &&
               limbs_fit(64, 16, {{kTcE2, 4}, {kTcNew, 1}}, kTcC + 1024 * kTcCMerged) &&
               limbs_fit(32, kTcBlock, {{kTcP1, 4}}, kTcCP1) && limbs_fit(32, kTcBlock, {{kTcP2, 5}}, 0) &&
               limbs_fit(32, kTcBlock, {{kTcP3, 6}}, 0) && limbs_fit(64, 16, {{kTcFin, 4 + y_steps}}, 0);
    for (uint32_t c = kTcCR1; c <= kTcCOut; c++) fit = fit && limbs_fit(64, 16, {{kTcFull, 4}}, kTcC + 1024 * c);
    return fit;
  }
};

template <class F>
bool build(const uint32_t ext[8][16], const uint32_t* inte, const uint32_t diag[16], uint8_t* tables,
           P2TcConstants* consts, uint32_t* lane) {
  constexpr int R = F::ROUNDS_P;
  Builder B;
  B.p = F::P;
  B.r32 = (1ull << 32) % F::P;
  B.out = tables;
  memset(tables, 0, kTcTableBytes);
  memset(consts, 0, sizeof *consts);
  consts->wait_tries = kTcWaitTries;
  consts->arrivals = 1;
  const uint64_t p = F::P;
  const uint64_t r32inv = [&] {
    uint64_t r = 1, b = B.r32, e = p - 2;
    for (; e; e >>= 1, b = b * b % p)
      if (e & 1) r = r * b % p;
    return r;
  }();
  static const int m4[4][4] = {{2, 3, 1, 1}, {1, 2, 3, 1}, {1, 1, 2, 3}, {3, 1, 1, 2}};
  for (int i = 0; i < 16; i++)
    for (int j = 0; j < 16; j++) B.me[i][j] = (uint64_t)m4[i % 4][j % 4] * (i / 4 == j / 4 ? 2 : 1);
  for (int i = 0; i < 16; i++) B.d[i] = (uint64_t)diag[i] * r32inv % p;  // from Monty form
  const uint64_t S = 1ull << 16;              // outputs in Monty form
  const uint64_t SX = B.mul(S, B.r32);        // partial-round inputs, reduced once more after the recombination
  const uint64_t SZ = B.mul(S, r32inv), SXZ = S;
  const uint64_t off = (1ull << 31) % p;      // y words carry + 2^31
  const uint64_t off_z = (1ull << 63) % p;    // z products + 2^63

  // external layer and its constants (ext / inte arrive in Monty form)
  for (uint32_t i = 0; i < 16; i++) {
    uint64_t rowsum = 0, e2sum = 0;
    for (uint32_t j = 0; j < 16; j++) {
      B.coef_z(kTcFull, 64, i, j, B.me[i][j], SZ);
      rowsum = (rowsum + B.me[i][j]) % p;
      uint64_t e2 = 0;
      for (uint32_t k = 8; k < 16; k++) e2 = (e2 + B.me[i][k] * B.me[k][j]) % p;
      B.coef_z(kTcE2, 64, i, j, e2, SZ);
      e2sum = (e2sum + e2) % p;
      if (j < 8) B.coef(kTcNew, 64, i, j, B.me[i][j], S);
    }
    auto col = [&](uint32_t which, uint64_t rc, uint64_t sum) {
      const uint64_t v = (B.mul(rc, S) + p - B.mul(B.mul(sum, SZ), off_z)) % p;
      B.constant_col(kTcC + 1024 * which, i, v);
    };
    col(kTcCInit, ext[0][i], 0);
    col(kTcCMerged, ext[0][i], e2sum);
    for (uint32_t r = 0; r < 3; r++) {
      col(kTcCR1 + r, ext[1 + r][i], rowsum);
      col(kTcCR5 + r, ext[5 + r][i], rowsum);
    }
    col(kTcCOut, 0, rowsum);
  }

  // partial rounds: alpha[r][j] = word 0 before round r from z_j; gamma from z_j to the final state
  std::vector<std::vector<uint64_t>> alpha(R, std::vector<uint64_t>(16)), gamma(16, std::vector<uint64_t>(16));
  for (uint32_t j = 0; j < 16; j++) {
    std::vector<uint64_t> s(16);
    for (int i = 0; i < 16; i++) s[i] = B.me[i][j];
    for (int r = 0; r < R; r++) {
      alpha[r][j] = s[0];
      s[0] = 0;  // replaced by y_r
      B.internal(s);
    }
    for (int i = 0; i < 16; i++) gamma[i][j] = s[i];
  }
  // beta[k]: word 0 before round r from y_(r-1-k); g[k]: the state after k + 1 rounds from y of the first
  std::vector<uint64_t> beta(R);
  std::vector<std::vector<uint64_t>> g(R, std::vector<uint64_t>(16));
  {
    std::vector<uint64_t> s(16, 0);
    s[0] = 1;
    for (int k = 0; k < R; k++) {
      B.internal(s);
      beta[k] = s[0];
      for (int i = 0; i < 16; i++) g[k][i] = s[i];
      s[0] = 0;
    }
  }
  for (int k = 0; k < 8 && k < R; k++) {
    const uint64_t m = B.mul(beta[k], B.r32);
    consts->beta[k] = m > p / 2 ? (int32_t)((int64_t)m - (int64_t)p) : (int32_t)m;
  }
  for (int blk = 0; blk * kTcBlock < R; blk++) {
    const uint32_t table = blk == 0 ? kTcP1 : blk == 1 ? kTcP2 : kTcP3;
    for (uint32_t i = 0; i < (uint32_t)kTcBlock; i++) {
      const int r = blk * kTcBlock + (int)i;
      if (r >= R) break;
      uint64_t sum = 0, sum_z = 0;
      for (uint32_t j = 0; j < 16; j++) {
        B.coef_z(table, 32, i, j, alpha[r][j], SXZ);
        sum_z = (sum_z + alpha[r][j]) % p;
      }
      for (int t = 0; t < blk * kTcBlock; t++) {
        const uint64_t c = beta[r - 1 - t];
        B.coef(table + 1024 * (kTcZSteps + t / kTcBlock), 32, i, t % kTcBlock, c, SX);
        sum = (sum + c) % p;
      }
      const uint64_t v =
          (B.mul(inte[r], SX) + 2 * p - B.mul(B.mul(sum, SX), off) - B.mul(B.mul(sum_z, SXZ), off_z)) % p;
      if (blk == 0)
        B.constant_col(kTcCP1, i, v);
      else
        B.constant_step(table + 1024 * kTcZSteps, 32, i, v);
    }
  }
  for (uint32_t i = 0; i < 16; i++) {
    uint64_t sum = 0, sum_z = 0;
    for (uint32_t j = 0; j < 16; j++) {
      B.coef_z(kTcFin, 64, i, j, gamma[i][j], SZ);
      sum_z = (sum_z + gamma[i][j]) % p;
    }
    for (int t = 0; t < R; t++) {
      const uint64_t c = g[R - 1 - t][i];
      B.coef(kTcFin + 2048 * (kTcZSteps + t / kTcBlock), 64, i, t % kTcBlock, c, S);
      sum = (sum + c) % p;
    }
    const uint64_t v = (B.mul(ext[4][i], S) + 2 * p - B.mul(B.mul(sum, S), off) - B.mul(B.mul(sum_z, SZ), off_z)) % p;
    B.constant_step(kTcFin + 2048 * kTcZSteps, 64, i, v);
  }

  // the one-word-per-lane tables: canonical values in Monty form
  memset(lane, 0, kLaneWords * 4);
  auto monty = [&](uint64_t v) { return (uint32_t)B.mul(v, B.r32); };
  for (uint32_t i = 0; i < 16; i++) {
    for (uint32_t r = 0; r < 8; r++) lane[kLaneExt + 16 * r + i] = ext[r][i];
    for (uint32_t j = 0; j < 16; j++) {
      if ((int)i < R) lane[kLaneAlpha + 16 * j + i] = monty(alpha[i][j]);
      if ((int)(16 + i) < R) lane[kLaneAlpha + 256 + 16 * j + i] = monty(alpha[16 + i][j]);
      lane[kLaneGamma + 16 * j + i] = monty(gamma[i][j]);
    }
    for (int t = 0; t < R; t++) lane[kLaneG + 16 * t + i] = monty(g[R - 1 - t][i]);
    if ((int)i < R) lane[kLaneConst + i] = monty(inte[i]);
    if ((int)(16 + i) < R) lane[kLaneConst + 16 + i] = monty(inte[16 + i]);
    lane[kLaneConst + 32 + i] = monty(ext[4][i]);
  }
  for (int k = 0; k < R; k++) lane[kLaneBeta + kLaneBetaZero + k] = monty(beta[k]);
  return p2_tc_sums_fit(consts->beta, F::P) && B.all_limbs_fit(R);
}

}  // namespace

bool p2_tc_sums_fit(const int32_t beta[8], uint32_t p) {
  uint64_t sum = 0;
  for (int k = 0; k < kTcBlock - 1; k++) sum += beta[k] < 0 ? 0u - (uint32_t)beta[k] : (uint32_t)beta[k];
  const uint64_t y = 3ull * p / 4;
  return sum <= ((1ull << 63) - 1 - p) / y;
}

bool build_p2_tc_tables(int field, const uint32_t ext[8][16], const uint32_t* inte, const uint32_t diag[16],
                        uint8_t* tables, P2TcConstants* consts, uint32_t* lane) {
  return field == 0 ? build<KoalaBear>(ext, inte, diag, tables, consts, lane)
                    : build<BabyBear>(ext, inte, diag, tables, consts, lane);
}

}  // namespace pico
