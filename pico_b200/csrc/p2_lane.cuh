// Poseidon2 width-16 with one state word per lane (16 lanes per state, two
// states per warp): the latency form, for trees and rows too few to fill the
// GPU, where a chain of dependent permutations sets the time.
//
// Full rounds: the S-boxes run side by side, the external layer is two steps
// of three shuffles (column sums over the blocks, then the 4x4 block, which
// commute).  Partial rounds: only word 0 passes through S-boxes, so with z the
// S-box outputs of the last full round and y_r those of the partial rounds,
//   x_r = A_r + sum_(j<r) beta_(r-1-j) y_j,  A_r = alpha_r . z + c_r,
// and the state after them is Gamma z + sum_t G_t y_t.  Lane i keeps the sum of
// x_i (and of x_(16+i)) and of state word i and adds y_j to each as it becomes
// known; every lane runs the S-box chain itself.  Between y_(r-1) and y_r lie
// one subtraction (beta_0 = D_0 + 1 = -1) and the S-box: x_r's sum without its
// last two y leaves its lane two rounds ahead.
//
// Latency of one permutation in cycles, one thread / four lanes / this form:
// KoalaBear 11,270 / 8,400 / about 4,200, BabyBear 16,020 / 7,950 / 3,960.  In a full
// round the two shuffle steps and their six dependent additions take 115
// cycles and the S-box 50 (90).  Unrolled partial rounds: a FRI phase of 4.04
// ms, against 4.25 with loops of three.
//   commit of 2 tiny BabyBear traces 314 -> 231 us, 2^16 x 64 commit 504 -> 481 us,
//   FRI phase of 2^23 elements 4.70 -> 4.04 ms, opening of 2^26 cells 3.70 -> 3.17 ms,
//   16 requests of ~20 small traces 4.78 -> 4.3..4.6 ms.
#pragma once
#include "field.cuh"
#include "internal.h"
#include "p2_layers.cuh"
#include "p2_tc_tables.h"

namespace pico {

__device__ uint32_t g_p2_lane[2][kLaneWords];

// Copy a field's tables to shared memory (the caller synchronises) and wait
// for the kernel before this one.
template <class F>
__device__ __forceinline__ void lane_load_tables(uint32_t* tab) {
  const uint4* src = reinterpret_cast<const uint4*>(g_p2_lane[F::ID]);
  grid_release();
  for (uint32_t i = threadIdx.x; i < kLaneWords / 4; i += blockDim.x) reinterpret_cast<uint4*>(tab)[i] = __ldg(src + i);
  grid_wait();
}

// 64-bit sums of products of canonical values: four fit (4 p^2 < 2^64); a fold
// replaces the high word by its residue (below 2^61), after which three fit.
template <class F>
__device__ __forceinline__ uint64_t lane_mad(uint32_t a, uint32_t b, uint64_t c) {
  uint32_t lo, hi;
  asm("mad.lo.cc.u32 %0, %2, %3, %4;\n\tmadc.hi.u32 %1, %2, %3, %5;"
      : "=&r"(lo), "=r"(hi)
      : "r"(a), "r"(b), "r"((uint32_t)c), "r"((uint32_t)(c >> 32)));
  return ((uint64_t)hi << 32) | lo;
}
template <class F>
__device__ __forceinline__ uint64_t lane_fold(uint64_t acc) {
  return lane_mad<F>((uint32_t)(acc >> 32), (uint32_t)((1ull << 32) % F::P), (uint64_t)(uint32_t)acc);
}
// Canonical value of any 64-bit sum, times 2^-32.
template <class F>
__device__ __forceinline__ uint32_t lane_reduce(uint64_t acc) {
  return Fp<F>::canon(Fp<F>::redc(lane_fold<F>(acc)));
}

// External layer of the 16 words of a group, plus k (canonical).
template <class F>
__device__ __forceinline__ uint32_t lane_external(uint32_t v, uint32_t q, uint32_t k) {
  using B = Fp<F>;
  constexpr unsigned kAll = 0xffffffffu;
  const uint32_t v4 = __shfl_xor_sync(kAll, v, 4, 16), v8 = __shfl_xor_sync(kAll, v, 8, 16),
                 v12 = __shfl_xor_sync(kAll, v, 12, 16);
  const uint32_t u = B::add(B::add(B::add(v, v), v4), B::add(v8, v12));
  const uint32_t blk = q & ~3u;
  const uint32_t b = __shfl_sync(kAll, u, (int)(blk | ((q + 1) & 3u)), 16),
                 c = __shfl_sync(kAll, u, (int)(blk | ((q + 2) & 3u)), 16),
                 d = __shfl_sync(kAll, u, (int)(blk | ((q + 3) & 3u)), 16);
  // row q: 2 u_q + 3 u_(q+1) + u_(q+2) + u_(q+3)
  const uint32_t uk = B::add(B::add(u, u), k);
  return B::add(B::add(B::add(b, b), uk), B::add(B::add(b, c), d));
}

// The permutation of the group's state, lane q holding word q (canonical).
// All 32 lanes of a warp call it together.
template <class F>
__device__ __forceinline__ uint32_t lane_permute(uint32_t v, uint32_t q, const uint32_t* tab) {
  using B = Fp<F>;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int R = F::ROUNDS_P;
  const uint32_t* t = tab + q;
  v = lane_external<F>(v, q, t[kLaneExt]);
#pragma unroll 1
  for (int r = 1; r < 4; r++) v = lane_external<F>(p2_sbox<F>(v), q, t[kLaneExt + 16 * r]);
  v = p2_sbox<F>(v);
  // the sums of x_i, x_(16+i) and state word i, each as two chains over the
  // even and the odd words; three terms fit between folds
  uint64_t a0 = t[kLaneConst], a1 = t[kLaneConst + 16], s = t[kLaneConst + 32], a0o = 0, a1o = 0, so = 0;
#pragma unroll
  for (int j = 0; j < 16; j += 2) {
    const uint32_t z = __shfl_sync(kAll, v, j, 16), zo = __shfl_sync(kAll, v, j + 1, 16);
    a0 = lane_mad<F>(t[kLaneAlpha + 16 * j], z, a0);
    a0o = lane_mad<F>(t[kLaneAlpha + 16 * j + 16], zo, a0o);
    if (R > 16) a1 = lane_mad<F>(t[kLaneAlpha + 256 + 16 * j], z, a1);
    if (R > 16) a1o = lane_mad<F>(t[kLaneAlpha + 256 + 16 * j + 16], zo, a1o);
    s = lane_mad<F>(t[kLaneGamma + 16 * j], z, s);
    so = lane_mad<F>(t[kLaneGamma + 16 * j + 16], zo, so);
    if (j == 4 || j == 10 || j == 14) {
      a0 = lane_fold<F>(a0);
      a0o = lane_fold<F>(a0o);
      if (R > 16) a1 = lane_fold<F>(a1);
      if (R > 16) a1o = lane_fold<F>(a1o);
      s = lane_fold<F>(s);
      so = lane_fold<F>(so);
    }
  }
  a0 += a0o;
  a1 += a1o;
  s += so;
  // x_0 .. x_3 need at most two y before the last: they leave now, and lanes
  // 0 .. 3 go on with x_16 .. x_19
  const uint32_t A = lane_reduce<F>(a0);
  uint32_t x = __shfl_sync(kAll, A, 0, 16), next = __shfl_sync(kAll, A, 1, 16);
  const uint32_t A2 = __shfl_sync(kAll, A, 2, 16), A3 = __shfl_sync(kAll, A, 3, 16);
  const uint32_t beta1 = tab[kLaneBeta + kLaneBetaZero + 1], beta2 = tab[kLaneBeta + kLaneBetaZero + 2];
  const uint32_t* bt = t + kLaneBeta + kLaneBetaZero - 1;  // beta of (lane's x) - 1 - r at bt[-r]
  if (R > 16 && q < 4) {
    a0 = a1;
    bt += 16;
  }
  uint32_t y1 = 0;  // y_(r-1)
  // Round r: y_r and x_(r+1) = next + beta_1 y_(r-1) - y_r; `ahead` is x_(r+2)
  // without its last two y.  What the last rounds prepare is not used.
  auto round = [&](int r, uint32_t ahead) {
    const uint32_t y = p2_sbox<F>(x);
    x = B::sub(B::add(next, B::mul(beta1, y1)), y);
    next = ahead;
    y1 = y;
    if (r + 3 < R) a0 = lane_mad<F>(bt[-r], y, a0);
    s = lane_mad<F>(t[kLaneG + 16 * r], y, s);
  };
  auto ahead = [&](int r) { return __shfl_sync(kAll, lane_reduce<F>(a0), (r + 2) & 15, 16); };
  round(0, A2);
  round(1, B::add(A3, B::mul(beta2, y1)));
#pragma unroll
  for (int r = 2; r + 2 < R; r += 3) {
    a0 = lane_fold<F>(a0);
    s = lane_fold<F>(s);
#pragma unroll
    for (int u = 0; u < 3; u++) round(r + u, r + u + 2 < R ? ahead(r + u) : 0u);
  }
  if constexpr ((R - 2) % 3 == 2) {
    a0 = lane_fold<F>(a0);
    s = lane_fold<F>(s);
    round(R - 2, 0u);
    round(R - 1, 0u);
  }
  static_assert((R - 2) % 3 != 1, "partial rounds in threes, or two left");
  v = lane_reduce<F>(s);
#pragma unroll 1
  for (int r = 5; r < 8; r++) v = lane_external<F>(p2_sbox<F>(v), q, t[kLaneExt + 16 * r]);
  return lane_external<F>(p2_sbox<F>(v), q, 0u);
}

}  // namespace pico
