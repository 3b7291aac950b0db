// Layout of the tensor-core Poseidon2 tables (p2_tc.cuh), shared by the
// device code and the host code that builds them (p2_tc_tables.cu).
#pragma once
#include <cstdint>

namespace pico {

constexpr uint32_t kTcThreads = 128;  // states per group: M of the MMA, one TMEM lane each
constexpr uint32_t kTcGroups = 4;      // groups per CTA, sharing the tables
constexpr uint32_t kTcCtas = 2;        // CTAs per SM
constexpr uint32_t kTcResident = kTcCtas * 148;  // CTAs of a full wave (a B200's 148 SMs; fewer only share unevenly)
constexpr int kTcBlock = 7;           // partial rounds per block: 7 y words and the constant word fill a 32-byte K step
constexpr uint32_t kTcCols = 64;      // TMEM columns per group (eight groups fill an SM's 512)
// TMEM columns of a group: the S-box outputs z of a full round (16 x 64
// bits) and the accumulators of half a layer (8 words x 4 limbs).
constexpr uint32_t kTcZ = 0, kTcAcc = 32;
constexpr int kTcZSteps = 4;

// Shared-memory tables (byte offsets).  A K step is 32 bytes of K for N rows:
// two core-matrix columns (8 rows x 16 bytes, contiguous) of N / 8 each.
constexpr uint32_t kTcZero = 0;                      // a zero core-matrix column, N = 64
constexpr uint32_t kTcFull = 1024;                   // external layer of z: 4 K steps, N = 64
constexpr uint32_t kTcE2 = kTcFull + 8192;           // external layer of the capacity words of the external layer of z
constexpr uint32_t kTcNew = kTcE2 + 8192;            // external layer, 8 new rate words: 1 K step
constexpr uint32_t kTcP1 = kTcNew + 2048;            // first block of partial-round inputs: z, N = 32
constexpr uint32_t kTcP2 = kTcP1 + 4096;             // second block: z, y_0..6 and the constant (5 steps), N = 32
constexpr uint32_t kTcP3 = kTcP2 + 5120;             // third block: z, y_0..6, y_7..13 (6 steps), N = 32
constexpr uint32_t kTcFin = kTcP3 + 6144;            // state after the partial rounds: z and all y (7 steps), N = 64
constexpr uint32_t kTcC = kTcFin + 14336;            // constant columns, N = 64, 1024 bytes each
constexpr uint32_t kTcCP1 = kTcC + 9 * 1024;         // constant column of the first block, N = 32
constexpr uint32_t kTcTableBytes = kTcCP1 + 512;
// After the tables, the operand words that are not in TMEM, as K steps of 128
// rows (two core-matrix columns of 2048 bytes): a constant K step whose last
// word is 1, then per group three of 32-bit words (y of the partial rounds;
// the rate words to absorb in the second).
constexpr uint32_t kTcStepBytes = 4096;
constexpr uint32_t kTcOne = kTcTableBytes;
constexpr uint32_t kTcY = kTcOne + kTcStepBytes;
constexpr uint32_t kTcSmemBytes = kTcY + 3 * kTcStepBytes * kTcGroups;
static_assert(kTcTableBytes % 16 == 0, "operands start on 16 bytes");
// Indices of the N = 64 constant columns.
enum TcConstCol : uint32_t { kTcCInit = 0, kTcCMerged = 1, kTcCR1 = 2, kTcCR5 = 5, kTcCOut = 8 };

struct P2TcConstants {
  int32_t beta[8];     // y of k + 1 rounds ago: Monty form, centred (|.| <= p/2)
  uint32_t wait_tries; // tries of a wait for products before it gives up
  uint32_t arrivals;   // arrivals that complete a barrier: the products' one (two: no wait ever ends)
};
constexpr uint32_t kTcWaitTries = 1u << 18;  // about a second (3.9 us a try)

// Tables of the one-word-per-lane form (p2_lane.cuh), in words; entry [k][i]
// belongs to lane i.
constexpr uint32_t kLaneExt = 0;                      // full-round constants, 8 x 16
constexpr uint32_t kLaneAlpha = 128;                  // alpha_i per z_j, 16 x 16, then alpha_(16+i)
constexpr uint32_t kLaneGamma = kLaneAlpha + 512;     // Gamma, 16 x 16
constexpr uint32_t kLaneG = kLaneGamma + 256;         // state after the partial rounds per y_t, 20 x 16
constexpr uint32_t kLaneConst = kLaneG + 320;         // c_i, c_(16+i), constants of the next full round, times 2^32
constexpr uint32_t kLaneBeta = kLaneConst + 48;       // beta_k at kLaneBetaZero + k, zero elsewhere
constexpr uint32_t kLaneBetaZero = 24;
constexpr uint32_t kLaneWords = kLaneBeta + 64;
static_assert(kLaneWords % 4 == 0, "copied by 16 bytes");

// Whether the sums a block of partial rounds forms stay inside 63 bits: its last
// round adds kTcBlock - 1 products beta_k y and one recombined word.  The word is
// at most p.  |y| is below 3 p / 4: the S-box input is within p / 2 + 2^28 (the
// sum's high word is folded by 2^32 mod p < 2^29 before the reduction), below
// 0.64 p in both fields, and each product of factors below f p and g p reduces to
// (f g r + 1/2) p, r = p / 2^32, which gives 0.72 p (x^3) and 0.74 p (x^7).
bool p2_tc_sums_fit(const int32_t beta[8], uint32_t p);
// The tables of one field (kTcTableBytes) and its multiply-accumulate
// constants, and the lane tables (kLaneWords), from the canonical round constants
// and diagonal.  False if with these some sum of the tensor-core form could leave
// its range: those of p2_tc_sums_fit, or, with every byte 255, the limbs of an
// output (l0 + 2^8 l1 in 32 bits, and l2 + 2^8 l3, the recombined word's upper
// end, below p).
bool build_p2_tc_tables(int field, const uint32_t ext[8][16], const uint32_t* inte, const uint32_t diag[16],
                        uint8_t* tables, P2TcConstants* consts, uint32_t* lane);

}  // namespace pico
