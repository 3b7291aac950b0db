// Poseidon2 width-16 on the tensor cores: a group of 128 threads owns 128
// states, every linear layer is an integer matrix product on tcgen05
// (kind::i8), the S-boxes run in registers.
//
// A word is unsigned bytes in K, and any linear map of the words is
//   out_i = sum_j sum_b (c_ij 2^(8b) mod p) byte_b(w_j)   (mod p),
// whose 31-bit constants are split into four byte limbs: four columns of N per
// output word (below 208 * 255^2 < 2^24, exact in 32 bits).  A thread owns one
// state (one TMEM lane): it writes its words (a 32-bit TMEM cell is four K
// bytes), one elected thread issues the products, and the owner reads its
// limbs back and recombines them.  The matrices are arbitrary constants, so
// what lies between two S-boxes is merged into one product:
//   - the external layer with the round constants (a constant word in K);
//   - the Montgomery reduction that ends an S-box: z holds the 64-bit product
//     as eight bytes, whose weights absorb the reduction;
//   - the external layer of the last full round with the initial one of the
//     next permutation of a sponge (the capacity words only);
//   - all partial rounds: only word 0 passes through S-boxes, so the input
//     of partial round r is linear in the S-box outputs z of the last full
//     round and y_0 .. y_(r-1) of the earlier partial rounds, and the state
//     after them is linear in z and all y.  The rounds run in blocks of
//     kTcBlock: a product gives the part of the block's inputs that comes from
//     z and earlier blocks, and the y of the same block are added by
//     multiply-accumulates in registers.
//
// Bound: the multiplier pipe (hashing 2^17 rows
// of 64 columns: fmaheavy 57% busy, issue 47%) and the latency of the 19
// (KoalaBear) or 18 (BabyBear) product stages of a permutation, plus one or two
// for its output (~280 cycles each alone: barrier, products, commit, read-back),
// which the eight groups of an SM overlap.
// Layout: the accumulators hold half a layer (32 columns), so that z (32
// columns) and they are 64 columns, eight groups fill the 512 of an SM, and
// the second half's products run under the first half's S-boxes; the 32-bit
// words (y, rate words) are shared-memory operands.  Measured on 2^23 states
// (one permutation each): 4.60 G/s before the carry-pair reduction, 5.07 with it
// (one thread per state), here 7.50 (KoalaBear); 3.72, 4.01, 5.26
// (BabyBear).  On the way: whole layers at four groups per SM 6.2; products
// issued by thread 0 instead of an elected thread under warp-uniform control
// 6.2 (the descriptors then pass through per-thread registers: ~9
// instructions a product instead of 2.5); always the same warp issuing 7.2;
// three groups per CTA 7.15; one CTA of eight groups 7.9 here but no faster on
// whole commits (65.5 against 64.9 ms), and slower where few rows are hashed.
#pragma once
#include "field.cuh"
#include "internal.h"
#include "p2_tc_tables.h"

namespace pico {

__device__ uint4 g_p2_tc[2][kTcTableBytes / 16];
__constant__ P2TcConstants c_p2_tc[2];

// ---- tcgen05 / mbarrier primitives -----------------------------------------
__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_st16(uint32_t t, const uint32_t* a) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(t),
      "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
      "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15])
      : "memory");
}
// 32 accumulator columns of this thread's lane; complete on return.
__device__ __forceinline__ void tc_ld32(uint32_t t, uint32_t* a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]),
        "=r"(a[6]), "=r"(a[7]), "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]),
        "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15]), "=r"(a[16]), "=r"(a[17]),
        "=r"(a[18]), "=r"(a[19]), "=r"(a[20]), "=r"(a[21]), "=r"(a[22]), "=r"(a[23]),
        "=r"(a[24]), "=r"(a[25]), "=r"(a[26]), "=r"(a[27]), "=r"(a[28]), "=r"(a[29]),
        "=r"(a[30]), "=r"(a[31])
      : "r"(t)
      : "memory");
}
// Products of 32 bytes of K: the states' words in TMEM (ts) or shared memory (ss).
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{.reg .pred p; setp.ne.u32 p, %4, 0; tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;}" ::"r"(d), "r"(a),
      "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{.reg .pred p; setp.ne.u32 p, %4, 0; tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;}" ::"r"(d), "l"(a),
      "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Instruction descriptor: s32 accumulators, u8 x u8, M = 128, N columns.
__host__ __device__ constexpr uint32_t tc_idesc(uint32_t n) { return (2u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

// What a permutation starts from: 16 words; 8 rate words over a zero
// capacity; 8 new rate words over the capacity of the permutation whose last
// S-boxes are in z.
enum TcInput { kTcFromState, kTcFromRate, kTcFromSponge };

// A group's handle on its tensor-core state.
template <class F>
struct P2Tc {
  uint32_t tmem;   // column base of this group
  uint32_t lane;   // the same with this warp's first lane
  uint32_t sm;     // shared-memory address of the tables
  uint32_t ybase;  // offset of this group's operand words
  uint32_t bar;    // mbarrier the products arrive on
  uint32_t phase;
  uint32_t warp;   // warp-uniform values, so that the products' operands need no per-thread registers
  uint32_t turn;   // which of the group's warps issues next
  uint32_t dead;   // not 0: a wait ran out (for phase dead - 1): no more products or waits, results are void and reported

  __device__ __forceinline__ uint64_t desc(uint32_t offset, uint32_t lbo) const {
    return (uint64_t)((sm >> 4) + (offset >> 4) + ((lbo >> 4) << 16)) | ((uint64_t)((128u >> 4) | (1u << 14)) << 32);
  }
  // z times K steps of a table of N rows, 32 of them from row `row`.
  template <uint32_t N>
  __device__ __forceinline__ void product_z(uint32_t table, uint32_t row) const {
#pragma unroll
    for (int s = 0; s < kTcZSteps; s++)
      tc_mma_ts(tmem + kTcAcc, tmem + kTcZ + 8 * s, desc(table + s * N * 32 + row * 16, N * 16), tc_idesc(32), s != 0);
  }
  // A K step of words in shared memory times one of a table.
  template <uint32_t N>
  __device__ __forceinline__ void product_s(uint32_t words, uint32_t table, uint32_t row, uint32_t accumulate) const {
    tc_mma_ss(tmem + kTcAcc, desc(words, kTcStepBytes / 2), desc(table + row * 16, N * 16), tc_idesc(32), accumulate);
  }
  // The constant column: the constant K step times zeros and the column.
  __device__ __forceinline__ void constant(uint32_t col, uint32_t row) const {
    tc_mma_ss(tmem + kTcAcc, desc(kTcOne, kTcStepBytes / 2), desc(kTcZero + row * 16, col - kTcZero), tc_idesc(32), 1u);
  }
  __device__ __forceinline__ void sync() const {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync %0, 128;" ::"r"(1 + warp / 4) : "memory");
  }
  // Every warp is past the barrier: one issues the products of a stage, each
  // warp in turn, because the issue costs the scheduler it runs on.
  template <class Issue>
  __device__ __forceinline__ void issue(Issue products) {
    if (warp % 4 == turn) {
      if (!dead && elect_one()) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        products();
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
      }
      __syncwarp();
    }
    turn = (turn + 1) % 4;
  }
  static __device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{.reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p;}" : "=r"(one));
    return one != 0;
  }
  // Every thread's words are written: their products.
  template <class Issue>
  __device__ __forceinline__ void stage(Issue products) {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    sync();
    issue(products);
    wait();
  }
  __device__ __forceinline__ void wait() {
    if (!dead && __any_sync(0xffffffffu, !arrived(phase))) dead = 1 + phase;
    __syncwarp();
    phase ^= 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  // Whether the products of a phase have arrived, after a bounded wait.
  __device__ __forceinline__ bool arrived(uint32_t parity) const {
    auto tried = [&] {
      uint32_t ok;
      asm volatile("{.reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}"
                   : "=r"(ok)
                   : "r"(bar), "r"(parity)
                   : "memory");
      return ok != 0;
    };
    bool ok = tried();
#pragma unroll 1
    for (uint32_t i = 1; !ok && i < c_p2_tc[F::ID].wait_tries; i++) ok = tried();
    return ok;
  }

  // ---- arithmetic: signed Montgomery values ---------------------------------
  static __device__ __forceinline__ uint64_t mulw(uint32_t a, uint32_t b) {
    return (uint64_t)((int64_t)(int32_t)a * (int64_t)(int32_t)b);
  }
  // a * b + c, signed; as a carry pair, which compiles to one wide
  // multiply-add (mad.wide with a 64-bit addend becomes a product and two adds).
  static __device__ __forceinline__ uint64_t madw(uint32_t a, uint32_t b, uint64_t c) {
    uint32_t lo, hi;
    asm("mad.lo.cc.s32 %0, %2, %3, %4;\n\tmadc.hi.s32 %1, %2, %3, %5;"
        : "=&r"(lo), "=r"(hi)
        : "r"(a), "r"(b), "r"((uint32_t)c), "r"((uint32_t)(c >> 32)));
    return ((uint64_t)hi << 32) | lo;
  }
  // t * 2^-32 mod p in (-p/2 - |t|/2^32, p/2 + |t|/2^32); the high word wraps.
  static __device__ __forceinline__ uint32_t redc(uint64_t t) {
    return (uint32_t)(madw((uint32_t)t * F::NEG_PINV, F::P, t) >> 32);
  }
  // x^d of a Monty-form |x| <= p, as the product whose reduction is the last
  // step, plus 2^63: the eight bytes of z are unsigned, and the next linear
  // layer, which is linear in the bytes of any integer, takes the product
  // unreduced.  With r = p / 2^32 < 0.4961, a product of factors below f p
  // and g p reduces to below (f g r + 1/2) p.
  static __device__ __forceinline__ uint64_t sbox_wide(uint32_t x) {
    const uint32_t x2 = redc(mulw(x, x));
    if constexpr (F::SBOX == 3) {
      return mulw(x2, x) ^ (1ull << 63);
    } else {
      const uint32_t x3 = redc(mulw(x2, x)), x4 = redc(mulw(x2, x2));
      return mulw(x4, x3) ^ (1ull << 63);
    }
  }
  // The reduced word plus 2^31, for the same reason.
  static __device__ __forceinline__ uint32_t sbox(uint32_t x) { return redc(sbox_wide(x)); }
  // An output word from its limbs: V = l0 + 2^8 l1 + 2^16 l2 + 2^24 l3 times
  // 2^-16 (the tables carry the 2^16), by one 16-bit Montgomery step:
  // p = 1 mod 2^16, so V - (V mod 2^16) p is divisible by 2^16.  The
  // result lies in (-p, p), which the S-boxes and canon() take: the table
  // builder checks the upper end (at most 8.8e8 with these tables).
  static __device__ __forceinline__ uint32_t recombine(const uint32_t* l) {
    const uint32_t s01 = l[0] + (l[1] << 8), s23 = l[2] + (l[3] << 8);
    return s23 + (s01 >> 16) - (s01 & 0xffffu) * ((F::P - 1) >> 16);
  }
  static __device__ __forceinline__ uint32_t canon(uint32_t v) { return min(v, v + F::P); }

  // K step k of this thread's words in shared memory.
  __device__ __forceinline__ void put_words(uint32_t k, const uint32_t* w) const {
    const uint32_t r = threadIdx.x % kTcThreads;
    const uint32_t at = sm + ybase + k * kTcStepBytes + (r / 8) * 128 + (r % 8) * 16;
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                 : "memory");
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + kTcStepBytes / 2), "r"(w[4]), "r"(w[5]),
                 "r"(w[6]), "r"(w[7])
                 : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // S-boxes of the eight words in the accumulators.
  __device__ __forceinline__ void sbox8(uint32_t* z) const {
    uint32_t a[32];
    tc_ld32(lane + kTcAcc, a);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint64_t t = sbox_wide(recombine(a + 4 * i));
      z[2 * i] = (uint32_t)t;
      z[2 * i + 1] = (uint32_t)(t >> 32);
    }
  }
  // A linear layer and the S-boxes after it, from the words the products of
  // `layer` (rows 0.. or 32.. of its tables) read, into z.  The halves share
  // the accumulators; the second half's products run under the first half's
  // S-boxes, whose results wait in registers because the products read z.
  template <class Layer>
  __device__ __forceinline__ void full_round(Layer layer) {
    uint32_t a[32], z[16];
    stage([&] { layer(0u); });
    tc_ld32(lane + kTcAcc, a);
    sync();
    issue([&] { layer(32u); });
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint64_t t = sbox_wide(recombine(a + 4 * i));
      z[2 * i] = (uint32_t)t;
      z[2 * i + 1] = (uint32_t)(t >> 32);
    }
    wait();
    tc_st16(lane + kTcZ, z);
    sbox8(z);
    tc_st16(lane + kTcZ + 16, z);
  }
  // One block of R partial rounds: inputs from the accumulators plus the
  // block's own y, which go to K step k.  Up to kTcBlock - 1 signed products are
  // added before the fold: with these fields' beta (beta_0 is -1 times 2^32) at
  // most 0.47 of 2^63 (p2_tc_sums_fit; six of p / 2 each would not fit).
  // Round r's input before the S-box is (X_r + sum_k beta_k y_(r-1-k)) 2^-32.
  template <int R>
  __device__ __forceinline__ void partial_block(uint32_t k) {
    uint32_t a[32], y[8];
    tc_ld32(lane + kTcAcc, a);
    const int32_t* beta = c_p2_tc[F::ID].beta;
    constexpr uint32_t R32 = (uint32_t)((1ull << 32) % F::P);
#pragma unroll
    for (int r = 0; r < R; r++) {
      uint64_t acc = (uint64_t)(int64_t)(int32_t)recombine(a + 4 * r);
#pragma unroll
      for (int j = r - 1; j >= 0; j--) acc = madw((uint32_t)beta[j], y[r - 1 - j], acc);
      // fold the high word (2^32 mod p is below 2^29) so that the reduced
      // value stays within p/2 + 2^28
      if (r >= 2) acc = madw((uint32_t)(acc >> 32), R32, (uint32_t)acc);
      y[r] = sbox(redc(acc)) ^ 0x80000000u;
    }
#pragma unroll
    for (int r = 0; r < R; r++) y[r] ^= 0x80000000u;
#pragma unroll
    for (int r = R; r < 8; r++) y[r] = r == 7 ? 1u : 0u;
    put_words(k, y);
  }

  // The permutation up to its last S-boxes, left in z; `from` says what it
  // starts from.  One copy of it per kernel: callers loop over one call.
  __device__ __forceinline__ void body(TcInput from) {
    full_round([&](uint32_t row) {
      if (from == kTcFromState) {
        product_z<64>(kTcFull, row);
      } else if (from == kTcFromRate) {
        product_s<64>(ybase + kTcStepBytes, kTcNew, row, 0u);
      } else {
        product_z<64>(kTcE2, row);
        product_s<64>(ybase + kTcStepBytes, kTcNew, row, 1u);
      }
      constant(kTcC + 1024 * (from == kTcFromSponge ? kTcCMerged : kTcCInit), row);
    });
    external(kTcCR1);
    stage([&] {
      product_z<32>(kTcP1, 0);
      constant(kTcCP1, 0);
    });
    partial_block<kTcBlock>(0);
    stage([&] {
      product_z<32>(kTcP2, 0);
      product_s<32>(ybase, kTcP2 + kTcZSteps * 1024, 0, 1u);
    });
    if constexpr (F::ROUNDS_P == 20) {
      partial_block<kTcBlock>(1);
      stage([&] {
        product_z<32>(kTcP3, 0);
#pragma unroll
        for (uint32_t k = 0; k < 2; k++)
          product_s<32>(ybase + k * kTcStepBytes, kTcP3 + (kTcZSteps + k) * 1024, 0, 1u);
      });
      partial_block<6>(2);
    } else {
      static_assert(F::ROUNDS_P == 13, "partial rounds in blocks of 7, 7, 6 or 7, 6");
      partial_block<6>(1);
    }
    full_round([&](uint32_t row) {
      product_z<64>(kTcFin, row);
#pragma unroll
      for (uint32_t k = 0; k < (F::ROUNDS_P == 20 ? 3u : 2u); k++)
        product_s<64>(ybase + k * kTcStepBytes, kTcFin + (kTcZSteps + k) * 2048, row, 1u);
    });
    external(kTcCR5);
  }
  // Three full rounds with the constant columns from `col`.
  __device__ __forceinline__ void external(uint32_t col) {
#pragma unroll 1
    for (uint32_t r = 0; r < 3; r++)
      full_round([&](uint32_t row) {
        product_z<64>(kTcFull, row);
        constant(kTcC + 1024 * (col + r), row);
      });
  }
  // The words body() starts from: a state (canonical, or any 32-bit
  // representative), or eight rate words.
  __device__ __forceinline__ void put_state(const uint32_t* s) const {
    __syncwarp();
    // a word w stands for the product w * 2^32
    uint32_t z[16];
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        z[2 * i] = 0;
        z[2 * i + 1] = s[8 * h + i];
      }
      tc_st16(lane + kTcZ + 16 * h, z);
    }
  }
  __device__ __forceinline__ void put_rate(const uint32_t* s) const {
    __syncwarp();
    put_words(1, s);
  }
  // Words 8h .. 8h + 7 of the permutation's output, canonical.
  __device__ __forceinline__ void output8(uint32_t h, uint32_t* s) {
    stage([&] {
      product_z<64>(kTcFull, 32 * h);
      constant(kTcC + 1024 * kTcCOut, 32 * h);
    });
    uint32_t a[32];
    tc_ld32(lane + kTcAcc, a);
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = canon(recombine(a + 4 * i));
  }
  __device__ __forceinline__ void digest(uint32_t* s) { output8(0, s); }
  __device__ __forceinline__ void output(uint32_t* s) {
    output8(0, s);
    output8(1, s + 8);
  }

  // Tiles of 128 states go to groups in order, a CTA's groups taking
  // neighbours; with no more tiles than resident groups they go one to a CTA
  // first, so that the SMs share them evenly.  Warp-uniform.
  __device__ __forceinline__ uint64_t first_tile(uint64_t tiles) const {
    return tiles <= kTcResident * kTcGroups ? blockIdx.x + (uint64_t)gridDim.x * (warp / 4) : (uint64_t)blockIdx.x * kTcGroups + warp / 4;
  }
  static __device__ __forceinline__ uint64_t tile_stride() { return (uint64_t)gridDim.x * kTcGroups; }
  // Set-up and tear-down, by the whole CTA: tables into shared memory, TMEM
  // columns, a barrier per group, the constant word.
  __device__ __forceinline__ void open(uint8_t* tables, uint64_t* mbar, uint32_t* tmem_slot) {
    const uint4* src = g_p2_tc[F::ID];
    for (uint32_t i = threadIdx.x; i < kTcTableBytes / 16; i += kTcThreads * kTcGroups)
      reinterpret_cast<uint4*>(tables)[i] = __ldg(src + i);
    warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    turn = 0;
    const uint32_t group = warp / 4;
    sm = tc_smem(tables);
    ybase = kTcY + 3 * kTcStepBytes * group;
    for (uint32_t i = threadIdx.x; i < kTcStepBytes / 16; i += kTcThreads * kTcGroups)
      reinterpret_cast<uint4*>(tables + kTcOne)[i] = make_uint4(0u, 0u, 0u, i >= kTcStepBytes / 32 ? 1u : 0u);
    bar = tc_smem(mbar + group);
    phase = 0;
    dead = 0;
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_slot)),
                   "n"(512 / kTcCtas)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
      for (uint32_t g = 0; g < kTcGroups; g++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(mbar + g)), "r"(c_p2_tc[F::ID].arrivals)
                     : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // Only now: a successor's CTAs hold TMEM while they wait for this kernel, so
    // every CTA of it has its own first.
    grid_release();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(tmem_slot), 0) + kTcCols * group;
    lane = tmem + ((warp % 4) << 21);
    grid_wait();
  }
  __device__ __forceinline__ void close() {
    // A warp that gave up waits once more, as long again: products still in
    // flight write TMEM columns and a barrier that are about to be given back.
    if (dead) arrived(dead - 1);
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512 / kTcCtas));
    }
  }
};

}  // namespace pico
