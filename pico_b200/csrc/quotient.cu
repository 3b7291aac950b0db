// compute_quotient_values on the GPU (vm/src/machine/utils.rs:201-350).
//
// One thread per point x_i = GENERATOR * w_Q^i of the quotient domain
// (Q = 2^(log_trace + log_qd), i in natural order).  The traces are the
// commit's resident LDEs: the quotient domain is the first Q points of the
// LDE domain, so natural point i is committed row rev_Q(i) (the rows
// get_evaluations_on_domain returns, prover.rs:469-489), and the next row is
// point i + 2^log_qd (mod Q).  The chip's constraints come as a straight-line
// register program (pico_constraint_op, see include/pico_gpu.h) that every
// thread runs over its own registers, which live in shared memory, in one of
// two forms, k_quotient_staged or k_quotient, by what the program reads and does
// (ProgramShape, quotient_program.h).  Assertions fold as acc = acc * alpha + c
// (ProverConstraintFolder::assert_zero / assert_zero_ext,
// vm/src/machine/folder.rs:223-227,321-327); the quotient is acc * inv_zerofier.
// The Lagrange selectors for the trace domain H = <w_n> (shift 1) follow vm/src/compiler/recursion/circuit/domain.rs:48-66:
// Z_H(x) = x^n - 1, is_first_row = Z_H / (x - 1), is_last_row =
// Z_H / (x - w_n^-1), is_transition = x - w_n^-1, inv_zerofier = 1 / Z_H; the
// three inverses share one Fermat inversion per point.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/pico_gpu.h"
#include "field.cuh"
#include "internal.h"
#include "quotient_program.h"
#include "runtime.h"

namespace pico {

constexpr uint32_t kQBaseRegs = 64;  // register file limits of a program
constexpr uint32_t kQExtRegs = 16;
constexpr size_t kQGeneralSmem = (kQBaseRegs + 4 * kQExtRegs) * kQThreads * 4;  // every register in use
// k_quotient_staged: a base operation whose result is only asserted, the
// assertion's index in dst.
constexpr uint32_t kQAssertOf = 32;

// The fold in the staged form: the sum of alpha^(m-1-k) c_k over the m
// assertions, one 64-bit sum per coefficient, its high word kept below p (p^2 +
// p 2^32 < 2^64).  A base value costs four wide multiply-adds and eight
// additions; the product acc * alpha it stands for is 19 Montgomery products.
// The general form folds as written: there the powers are one more read per
// assertion that the column reads push out of the L1 (2^18 points, 300 columns and
// assertions 2,290 us, with the sum 3,010; 2^20 points, 200 columns 7.7 / 9.4 ms).
template <class F>
struct AssertSum {
  uint32_t lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
  __device__ __forceinline__ void add_base(const uint4& p, uint32_t c) {
    const uint32_t pw[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, %1;" : "+r"(lo[j]), "+r"(hi[j]) : "r"(pw[j]), "r"(c));
      hi[j] = min(hi[j], hi[j] - F::P);
    }
  }
  __device__ __forceinline__ void add_ext(const uint4& p, const Ext4& c) {
    const Ext4 v = Ef<F>::mul(Ext4{{p.x, p.y, p.z, p.w}}, c);
#pragma unroll
    for (int j = 0; j < 4; j++) hi[j] = Fp<F>::add(hi[j], v.c[j]);
  }
  __device__ __forceinline__ Ext4 value() const {
    Ext4 v;
#pragma unroll
    for (int j = 0; j < 4; j++) v.c[j] = Fp<F>::canon(Fp<F>::redc(((uint64_t)hi[j] << 32) | lo[j]));
    return v;
  }
};

struct QuotientArgs {
  const uint32_t* main;
  const uint32_t* prep;
  const uint32_t* perm;
  uint32_t main_w, prep_w, perm_w;  // words per row (perm: 4 per extension column)
  const uint4* ops;
  uint32_t n_ops;
  uint32_t alpha[4];
  const uint4* powers;      // k_quotient_staged: alpha^(m-1-k) for the k-th of m assertions, whose dst is k
  const uint32_t* pub;      // public values
  const uint32_t* chal;     // permutation challenges, 4 words each
  const uint32_t* consts;   // regional sum (4), global sum (14)
  uint32_t log_trace, log_qd;
  uint32_t n_base;          // base registers the program uses; the extension registers follow them
  uint32_t shift_n;         // GENERATOR^(2^log_trace)
  uint32_t stride;          // k_quotient_staged: words of a thread's row (odd)
  uint32_t cols_end[6];     //   ends of the lists of cols: main, prep, perm, each at the point and at the next row
  const uint32_t* cols;     //   staged words' columns
  uint32_t chunks;          // 1: point i at out row (i mod D) n + i / D (split_evals order); 0: row i
  uint32_t* out;            // Q x 4
};

// Selectors at x = GENERATOR * w_Q^i.  x^n depends on i mod 2^log_qd only:
// GENERATOR^n times a power of w_(2^log_qd).
struct Selectors {
  uint32_t first, last, transition, inv_zh;
};
// a^(p-2) for p = C 2^S + 1 with C - 1 = 2 (2^K - 1) and K dividing S: the
// exponent's bits are K ones, a zero and S ones.
template <class F>
__device__ __forceinline__ uint32_t inverse(uint32_t a) {
  using B = Fp<F>;
  constexpr int K = F::PS % 6 ? 3 : 6;
  static_assert(F::PC - 1 == 2 * ((1u << K) - 1) && F::PS % K == 0, "exponent p - 2");
  uint32_t ones = B::mul(B::sqr(a), a);  // a^3
  ones = B::mul(B::sqr(ones), a);        // a^7
  if (K == 6) {
    uint32_t t = ones;
#pragma unroll
    for (int i = 0; i < 3; i++) t = B::sqr(t);
    ones = B::mul(t, ones);  // a^63
  }
  uint32_t v = B::sqr(ones);
#pragma unroll 1
  for (int g = 0; g < F::PS / K; g++) {
#pragma unroll
    for (int i = 0; i < K; i++) v = B::sqr(v);
    v = B::mul(v, ones);
  }
  return v;
}
template <class F>
__device__ __forceinline__ Selectors selectors(uint64_t i, const QuotientArgs& A, const TwiddleTables& tw) {
  using B = Fp<F>;
  constexpr uint32_t mask = (1u << F::TWO_ADICITY) - 1u;
  auto root = [&](uint32_t e) { return B::mul(__ldg(tw.hi + (e >> 14)), __ldg(tw.lo + (e & 0x3fffu))); };
  const uint32_t log_q = A.log_trace + A.log_qd;
  const uint32_t x = B::mul(B::to_monty(F::GENERATOR), root((uint32_t)(i << (F::TWO_ADICITY - log_q)) & mask));
  const uint32_t xn = B::mul(A.shift_n, root((uint32_t)(i << (F::TWO_ADICITY - A.log_qd)) & mask));
  const uint32_t wn_inv = root((0u - (1u << (F::TWO_ADICITY - A.log_trace))) & mask);
  const uint32_t zh = B::sub(xn, F::ONE);
  const uint32_t d1 = B::sub(x, F::ONE), d2 = B::sub(x, wn_inv);
  const uint32_t d12 = B::mul(d1, d2);
  const uint32_t inv = inverse<F>(B::mul(d12, zh));  // nonzero: the quotient domain is disjoint from H
  const uint32_t zi = B::mul(zh, inv);
  return {B::mul(zh, B::mul(d2, zi)), B::mul(zh, B::mul(d1, zi)), d2, B::mul(inv, d12)};
}
template <class F>
__device__ __forceinline__ void store_quotient(const Ext4& acc, uint32_t inv_zh, uint64_t i, const QuotientArgs& A) {
  using B = Fp<F>;
  const uint64_t orow =
      A.chunks ? ((i & ((1ull << A.log_qd) - 1)) << A.log_trace) + (i >> A.log_qd) : i;  // a permutation of [0, Q)
  reinterpret_cast<uint4*>(A.out)[orow] = make_uint4(B::mul(acc.c[0], inv_zh), B::mul(acc.c[1], inv_zh),
                                                     B::mul(acc.c[2], inv_zh), B::mul(acc.c[3], inv_zh));
}

template <class F>
__global__ void __launch_bounds__(kQThreads) k_quotient(const __grid_constant__ QuotientArgs A,
                                                         const __grid_constant__ TwiddleTables tw) {
  using B = Fp<F>;
  using E = Ef<F>;
  extern __shared__ uint32_t qsm[];
  uint32_t* rb = qsm + threadIdx.x;                               // base register r at rb[r * kQThreads]
  uint32_t* re = qsm + A.n_base * kQThreads + threadIdx.x;        // ext register r, coeff j at re[(4r+j) * kQThreads]
  const uint32_t log_q = A.log_trace + A.log_qd;
  const uint64_t Q = 1ull << log_q;
  const uint64_t i = (uint64_t)blockIdx.x * kQThreads + threadIdx.x;
  const bool active = i < Q;
  const uint64_t ii = active ? i : 0;
  const uint64_t row_l = bitrev64(ii, (int)log_q);
  const uint64_t row_n = bitrev64((ii + (1ull << A.log_qd)) & (Q - 1), (int)log_q);

  const Selectors sel = selectors<F>(ii, A, tw);
  Ext4 acc{{0, 0, 0, 0}};
  const Ext4 alpha{{A.alpha[0], A.alpha[1], A.alpha[2], A.alpha[3]}};

  auto ext_get = [&](uint32_t r) {
    Ext4 v;
#pragma unroll
    for (int j = 0; j < 4; j++) v.c[j] = re[(4 * r + j) * kQThreads];
    return v;
  };
  auto ext_set = [&](uint32_t r, const Ext4& v) {
#pragma unroll
    for (int j = 0; j < 4; j++) re[(4 * r + j) * kQThreads] = v.c[j];
  };
  for (uint32_t k = 0; k < A.n_ops; k++) {
    const uint4 o = __ldg(A.ops + k);  // the same instruction for every thread: a broadcast
    const uint32_t d = o.y, a = o.z, b = o.w;
    const uint64_t row = b ? row_n : row_l;
    switch (o.x) {
      case PICO_Q_MAIN: rb[d * kQThreads] = __ldg(A.main + row * A.main_w + a); break;
      case PICO_Q_PREP: rb[d * kQThreads] = __ldg(A.prep + row * A.prep_w + a); break;
      case PICO_Q_PERM: {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(A.perm + row * A.perm_w + 4 * a));
        ext_set(d, Ext4{{v.x, v.y, v.z, v.w}});
        break;
      }
      case PICO_Q_CONST: rb[d * kQThreads] = a; break;
      case PICO_Q_PUBLIC: rb[d * kQThreads] = __ldg(A.pub + a); break;
      case PICO_Q_FIRST: rb[d * kQThreads] = sel.first; break;
      case PICO_Q_LAST: rb[d * kQThreads] = sel.last; break;
      case PICO_Q_TRANSITION: rb[d * kQThreads] = sel.transition; break;
      case PICO_Q_ADD: rb[d * kQThreads] = B::add(rb[a * kQThreads], rb[b * kQThreads]); break;
      case PICO_Q_SUB: rb[d * kQThreads] = B::sub(rb[a * kQThreads], rb[b * kQThreads]); break;
      case PICO_Q_MUL: rb[d * kQThreads] = B::mul(rb[a * kQThreads], rb[b * kQThreads]); break;
      case PICO_Q_EADD: ext_set(d, E::add(ext_get(a), ext_get(b))); break;
      case PICO_Q_ESUB: ext_set(d, E::sub(ext_get(a), ext_get(b))); break;
      case PICO_Q_EMUL: ext_set(d, E::mul(ext_get(a), ext_get(b))); break;
      case PICO_Q_EMB: ext_set(d, Ext4{{rb[a * kQThreads], 0u, 0u, 0u}}); break;
      case PICO_Q_EMULB: ext_set(d, E::scale(ext_get(a), rb[b * kQThreads])); break;
      case PICO_Q_CHALLENGE:
        ext_set(d, Ext4{{__ldg(A.chal + 4 * a), __ldg(A.chal + 4 * a + 1), __ldg(A.chal + 4 * a + 2),
                         __ldg(A.chal + 4 * a + 3)}});
        break;
      case PICO_Q_REGIONAL:
        ext_set(d, Ext4{{__ldg(A.consts), __ldg(A.consts + 1), __ldg(A.consts + 2), __ldg(A.consts + 3)}});
        break;
      case PICO_Q_GLOBAL: rb[d * kQThreads] = __ldg(A.consts + 4 + a); break;
      case PICO_Q_ASSERT: {
        acc = E::mul(acc, alpha);
        acc.c[0] = B::add(acc.c[0], rb[a * kQThreads]);
        break;
      }
      case PICO_Q_EASSERT: acc = E::add(E::mul(acc, alpha), ext_get(a)); break;
      default: break;  // validated on the host
    }
  }
  if (active) store_quotient<F>(acc, sel.inv_zh, i, A);
}

// The staged form: thread t of CTA b
// owns the point of committed row 128 b + t and a row of shared memory
// that holds the trace words the program reads (each copied once, a row's
// words side by side), the selectors and the program's registers; the odd
// stride spreads a warp over the banks.  The host has renamed operands to
// words of that row, so that reading a column is no instruction; operands come
// as byte offsets.
//
// Bound: instruction issue (55% of cycles, 2^21 points x 32 columns) and the
// latency of the interpreter's dependent steps at 28 warps per SM.  The general
// form reads a column from 32 lines per warp and instruction, for which the L1
// is busy 83% of the time, and dispatches 215 instructions where 90 are left here.  KoalaBear, host call included:
// 2^20 points x 33 columns 591 -> 345 us, 2^19 x 100 354 -> 290, 2^11 x 8 132 -> 106.
template <class F>
__global__ void __launch_bounds__(kQThreads) k_quotient_staged(const __grid_constant__ QuotientArgs A,
                                                                const __grid_constant__ TwiddleTables tw) {
  using B = Fp<F>;
  using E = Ef<F>;
  extern __shared__ uint32_t qsm[];
  const uint32_t log_q = A.log_trace + A.log_qd;
  const uint32_t Q = 1u << log_q;  // at most 2^27
  const uint32_t row0 = blockIdx.x * kQThreads;
  const uint32_t sub = threadIdx.x & 7;
  for (uint32_t t = threadIdx.x >> 3; t < kQThreads; t += kQThreads / 8) {  // eight lanes per row
    const uint32_t row = row0 + t;
    if (row >= Q) break;
    const uint32_t next = bitrev32((bitrev32(row, (int)log_q) + (1u << A.log_qd)) & (Q - 1), (int)log_q);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(qsm + t * A.stride);
    uint32_t j0 = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const uint32_t* base = k < 2 ? A.main : k < 4 ? A.prep : A.perm;
      const uint32_t w = k < 2 ? A.main_w : k < 4 ? A.prep_w : A.perm_w;
      const uint32_t j1 = A.cols_end[k];
      if (j1 == j0) continue;
      const uint32_t* src = base + (uint64_t)(k & 1 ? next : row) * w;
      for (uint32_t j = j0 + sub; j < j1; j += 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * j), "l"(src + __ldg(A.cols + j))
                     : "memory");
      j0 = j1;
    }
  }
  const uint32_t row = row0 + threadIdx.x;
  const bool active = row < Q;
  const uint32_t i = bitrev32(active ? row : 0u, (int)log_q);
  const Selectors sel = selectors<F>(i, A, tw);
  char* own = reinterpret_cast<char*>(qsm + threadIdx.x * A.stride);
  auto word = [&](uint32_t off) -> uint32_t& { return *reinterpret_cast<uint32_t*>(own + off); };
  word(4 * A.cols_end[5]) = sel.first;
  word(4 * A.cols_end[5] + 4) = sel.last;
  word(4 * A.cols_end[5] + 8) = sel.transition;
  AssertSum<F> acc;
  auto ext_get = [&](uint32_t off) { return Ext4{{word(off), word(off + 4), word(off + 8), word(off + 12)}}; };
  auto ext_set = [&](uint32_t off, const Ext4& v) {
#pragma unroll
    for (int j = 0; j < 4; j++) word(off + 4 * j) = v.c[j];
  };
  uint4 o = __ldg(A.ops);  // the host appends one instruction
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (uint32_t k = 0; k < A.n_ops; k++) {
    const uint4 following = __ldg(A.ops + k + 1);
    const uint32_t d = o.y, a = o.z, b = o.w;
    switch (o.x) {
      case PICO_Q_CONST: word(d) = a; break;
      case PICO_Q_ADD: word(d) = B::add(word(a), word(b)); break;
      case PICO_Q_SUB: word(d) = B::sub(word(a), word(b)); break;
      case PICO_Q_MUL: word(d) = B::mul(word(a), word(b)); break;
      case kQAssertOf + PICO_Q_ADD: acc.add_base(__ldg(A.powers + d), B::add(word(a), word(b))); break;
      case kQAssertOf + PICO_Q_SUB: acc.add_base(__ldg(A.powers + d), B::sub(word(a), word(b))); break;
      case kQAssertOf + PICO_Q_MUL: acc.add_base(__ldg(A.powers + d), B::mul(word(a), word(b))); break;
      case PICO_Q_EADD: ext_set(d, E::add(ext_get(a), ext_get(b))); break;
      case PICO_Q_ESUB: ext_set(d, E::sub(ext_get(a), ext_get(b))); break;
      case PICO_Q_EMUL: ext_set(d, E::mul(ext_get(a), ext_get(b))); break;
      case PICO_Q_EMB: ext_set(d, Ext4{{word(a), 0u, 0u, 0u}}); break;
      case PICO_Q_EMULB: ext_set(d, E::scale(ext_get(a), word(b))); break;
      case PICO_Q_CHALLENGE:
        ext_set(d, Ext4{{__ldg(A.chal + 4 * a), __ldg(A.chal + 4 * a + 1), __ldg(A.chal + 4 * a + 2),
                         __ldg(A.chal + 4 * a + 3)}});
        break;
      case PICO_Q_REGIONAL:
        ext_set(d, Ext4{{__ldg(A.consts), __ldg(A.consts + 1), __ldg(A.consts + 2), __ldg(A.consts + 3)}});
        break;
      case PICO_Q_ASSERT: acc.add_base(__ldg(A.powers + d), word(a)); break;
      case PICO_Q_EASSERT: acc.add_ext(__ldg(A.powers + d), ext_get(a)); break;
      default: break;  // renamed or folded on the host
    }
    o = following;
  }
  if (active) store_quotient<F>(acc.value(), sel.inv_zh, i, A);
}

}  // namespace pico

using namespace pico;

namespace {

// GENERATOR^(2^log_n).
template <class F>
uint32_t shift_power(uint32_t log_n) {
  uint32_t v = Fp<F>::to_monty(F::GENERATOR);
  for (uint32_t k = 0; k < log_n; k++) v = Fp<F>::sqr(v);
  return v;
}

// alpha^(m-1-k) at powers + 4 k.
template <class F>
void assertion_powers(const uint32_t alpha[4], uint32_t m, uint32_t* powers) {
  const Ext4 a{{alpha[0], alpha[1], alpha[2], alpha[3]}};
  Ext4 v{{F::ONE, 0, 0, 0}};
  for (uint32_t k = m; k-- > 0; v = Ef<F>::mul(v, a)) memcpy(powers + 4 * k, v.c, 16);
}

// A validated program for k_quotient_staged: per list of QuotientArgs::cols_end
// the words read, and the instructions left once every read of a column or
// selector is renamed to its word (registers that other instructions write get
// words of their own) and public values and global sums are constants.
struct StagedProgram {
  std::vector<uint32_t> cols;
  uint32_t cols_end[6] = {};
  std::vector<pico_constraint_op> ops;
  uint32_t stride = 1;
  // For each assertion of a base register: its value comes from the addition,
  // subtraction or product just before it, and nothing reads that register
  // again before it is written.
  static std::vector<bool> sole_uses(const pico_constraint_op* program, uint32_t n_ops) {
    std::vector<bool> sole(n_ops, false);
    bool read_later[kQBaseRegs] = {};
    for (uint32_t k = n_ops; k-- > 0;) {
      const pico_constraint_op& o = program[k];
      switch (o.op) {
        case PICO_Q_MAIN: case PICO_Q_PREP: case PICO_Q_CONST: case PICO_Q_PUBLIC: case PICO_Q_FIRST:
        case PICO_Q_LAST: case PICO_Q_TRANSITION: case PICO_Q_GLOBAL: read_later[o.dst] = false; break;
        case PICO_Q_ADD: case PICO_Q_SUB: case PICO_Q_MUL:
          read_later[o.dst] = false;
          read_later[o.a] = read_later[o.b] = true;
          break;
        case PICO_Q_EMB: read_later[o.a] = true; break;
        case PICO_Q_EMULB: read_later[o.b] = true; break;
        case PICO_Q_ASSERT: {
          const uint32_t before = k ? program[k - 1].op : 0u;
          sole[k] = !read_later[o.a] && (before == PICO_Q_ADD || before == PICO_Q_SUB || before == PICO_Q_MUL) &&
                    program[k - 1].dst == o.a;
          read_later[o.a] = true;
          break;
        }
        default: break;
      }
    }
    return sole;
  }
  StagedProgram() = default;
  StagedProgram(const pico_constraint_op* program, uint32_t n_ops, const ProgramShape& shape,
                const uint32_t* public_values, const uint32_t* global_sum) {
    std::vector<uint32_t> word[6];  // per column of a list, its (first) word
    cols.reserve(shape.words);
    for (uint32_t l = 0; l < 6; l++) {
      word[l].assign(shape.last[l].size(), 0);
      for (uint32_t c = 0; c < word[l].size(); c++) {
        if (!shape.last[l][c]) continue;
        word[l][c] = (uint32_t)cols.size();
        for (uint32_t j = 0; j < (l < 4 ? 1u : 4u); j++) cols.push_back(l < 4 ? c : 4 * c + j);
      }
      cols_end[l] = (uint32_t)cols.size();
    }
    ops.reserve(n_ops + 1);
    const uint32_t selectors = (uint32_t)cols.size();
    uint32_t words = selectors + 3;
    constexpr uint32_t kNone = 0xffffffffu;
    // per register its own word and the word that holds its value now
    std::vector<uint32_t> home[2] = {std::vector<uint32_t>(kQBaseRegs, kNone), std::vector<uint32_t>(kQExtRegs, kNone)};
    std::vector<uint32_t> now[2] = {home[0], home[1]};
    auto own = [&](int ext, uint32_t r) {
      if (home[ext][r] == kNone) {
        home[ext][r] = words;
        words += ext ? 4 : 1;
      }
      return home[ext][r];
    };
    auto from = [&](int ext, uint32_t r) {  // a register that nothing wrote: its own word, undefined as ever
      if (now[ext][r] == kNone) now[ext][r] = own(ext, r);
      return 4 * now[ext][r];
    };
    auto into = [&](int ext, uint32_t r) { return 4 * (now[ext][r] = own(ext, r)); };
    uint32_t asserts = 0;
    const std::vector<bool> sole = sole_uses(program, n_ops);
    for (uint32_t k = 0; k < n_ops; k++) {
      pico_constraint_op o = program[k];
      switch (o.op) {
        case PICO_Q_MAIN: case PICO_Q_PREP: case PICO_Q_PERM: {
          const int l = ProgramShape::list(o);
          now[l < 4 ? 0 : 1][o.dst] = word[l][o.a];
          continue;
        }
        case PICO_Q_FIRST: case PICO_Q_LAST: case PICO_Q_TRANSITION:
          now[0][o.dst] = selectors + (o.op - PICO_Q_FIRST);
          continue;
        case PICO_Q_CONST: o.dst = into(0, o.dst); break;
        case PICO_Q_PUBLIC: o = {PICO_Q_CONST, into(0, o.dst), public_values[o.a], 0}; break;
        case PICO_Q_GLOBAL: o = {PICO_Q_CONST, into(0, o.dst), global_sum[o.a], 0}; break;
        case PICO_Q_ADD: case PICO_Q_SUB: case PICO_Q_MUL:
          o.a = from(0, o.a), o.b = from(0, o.b), o.dst = into(0, o.dst);
          break;
        case PICO_Q_EADD: case PICO_Q_ESUB: case PICO_Q_EMUL:
          o.a = from(1, o.a), o.b = from(1, o.b), o.dst = into(1, o.dst);
          break;
        case PICO_Q_EMB: o.a = from(0, o.a), o.dst = into(1, o.dst); break;
        case PICO_Q_EMULB: o.a = from(1, o.a), o.b = from(0, o.b), o.dst = into(1, o.dst); break;
        case PICO_Q_CHALLENGE: case PICO_Q_REGIONAL: o.dst = into(1, o.dst); break;
        case PICO_Q_ASSERT: o.a = from(0, o.a), o.dst = asserts++; break;
        case PICO_Q_EASSERT: o.a = from(1, o.a), o.dst = asserts++; break;
        default: break;
      }
      if (sole[k]) {
        o = {kQAssertOf + ops.back().op, o.dst, ops.back().a, ops.back().b};
        ops.pop_back();
      }
      ops.push_back(o);
    }
    ops.push_back({0, 0, 0, 0});
    stride = words | 1u;
  }
};

// The LDE behind a trace reference, with its checks: a matrix of a resident
// commit of this context and field, tall enough for the quotient domain.
pico_status trace_view(pico_ctx* ctx, const pico_trace_ref& r, int field, uint32_t log_q, const char* what,
                       bool required, const uint32_t** ptr, uint32_t* width) {
  *ptr = nullptr;
  *width = 0;
  if (!r.commit) {
    if (required) {
      set_error("quotient_values: the %s trace is required", what);
      return PICO_ERR_INVALID_ARG;
    }
    return PICO_OK;
  }
  const pico_commit* c = r.commit;
  if (c->ctx != ctx || c->field != field || r.mat_idx >= c->n_mats) {
    set_error("quotient_values: the %s trace is not a matrix of a commit of this context and field", what);
    return PICO_ERR_INVALID_ARG;
  }
  if (c->shard_log) {
    set_error("quotient_values: the %s trace's commitment is one shard of a row-split commit", what);
    return PICO_ERR_UNSUPPORTED;
  }
  if (c->log_N[r.mat_idx] < log_q) {
    set_error("quotient_values: the %s LDE has 2^%u rows, fewer than the quotient domain's 2^%u", what,
              c->log_N[r.mat_idx], log_q);
    return PICO_ERR_INVALID_ARG;
  }
  *ptr = c->lde[r.mat_idx];
  *width = c->width[r.mat_idx];
  return PICO_OK;
}

}  // namespace

extern "C" pico_status pico_gpu_quotient_values(pico_ctx* ctx, pico_trace_ref preprocessed, pico_trace_ref main,
                                                pico_trace_ref permutation, uint32_t log_trace_height,
                                                uint32_t log_quotient_degree, const pico_constraint_op* program,
                                                uint32_t n_ops, const uint32_t* public_values, uint32_t n_public,
                                                const uint32_t* perm_challenges, uint32_t n_challenges,
                                                const uint32_t regional_sum[4], const uint32_t global_sum[14],
                                                const uint32_t alpha[4], uint32_t* out, uint32_t flags) {
  if (!ctx || !main.commit || (!program && n_ops) || !alpha || !out || (n_public && !public_values) ||
      (n_challenges && !perm_challenges)) {
    set_error("quotient_values: null argument");
    return PICO_ERR_INVALID_ARG;
  }
  if (flags & ~(PICO_OUTPUT_DEVICE | PICO_QUOTIENT_CHUNKS)) {
    set_error("quotient_values: unknown flags 0x%x", flags);
    return PICO_ERR_INVALID_ARG;
  }
  const int field = main.commit->field;
  const uint32_t S = field == PICO_KOALABEAR ? 24u : 27u;
  const uint32_t log_q = log_trace_height + log_quotient_degree;
  if (log_trace_height == 0 || log_q > S || log_quotient_degree > kLdeMaxLogBlowup) {
    set_error("quotient_values: trace 2^%u with quotient degree 2^%u is not supported", log_trace_height,
              log_quotient_degree);
    return PICO_ERR_INVALID_ARG;
  }
  pico_status s;
  const uint32_t *pm, *pp, *pe;
  uint32_t wm, wp, we;
  if ((s = trace_view(ctx, main, field, log_q, "main", true, &pm, &wm)) ||
      (s = trace_view(ctx, preprocessed, field, log_q, "preprocessed", false, &pp, &wp)) ||
      (s = trace_view(ctx, permutation, field, log_q, "permutation", false, &pe, &we)))
    return s;
  if (we % 4) {
    set_error("quotient_values: the permutation trace has %u words per row, not whole extension elements", we);
    return PICO_ERR_INVALID_ARG;
  }
  // the program: every register, column and table index in range; the
  // register files are sized to the highest register it names, so a small
  // program leaves shared memory for more resident CTAs
  uint32_t n_base = 1, n_ext = 1, n_asserts = 0;
  for (uint32_t k = 0; k < n_ops; k++) {
    const pico_constraint_op& o = program[k];
    bool ok;
    const bool db = o.dst < kQBaseRegs, de = o.dst < kQExtRegs;
    switch (o.op) {
      case PICO_Q_MAIN: ok = db && o.a < wm && o.b <= 1; break;
      case PICO_Q_PREP: ok = db && pp && o.a < wp && o.b <= 1; break;
      case PICO_Q_PERM: ok = de && pe && o.a < we / 4 && o.b <= 1; break;
      case PICO_Q_CONST: ok = db && o.a < (field == PICO_KOALABEAR ? KoalaBear::P : BabyBear::P); break;
      case PICO_Q_PUBLIC: ok = db && o.a < n_public; break;
      case PICO_Q_FIRST: case PICO_Q_LAST: case PICO_Q_TRANSITION: ok = db; break;
      case PICO_Q_ADD: case PICO_Q_SUB: case PICO_Q_MUL: ok = db && o.a < kQBaseRegs && o.b < kQBaseRegs; break;
      case PICO_Q_EADD: case PICO_Q_ESUB: case PICO_Q_EMUL: ok = de && o.a < kQExtRegs && o.b < kQExtRegs; break;
      case PICO_Q_EMB: ok = de && o.a < kQBaseRegs; break;
      case PICO_Q_EMULB: ok = de && o.a < kQExtRegs && o.b < kQBaseRegs; break;
      case PICO_Q_CHALLENGE: ok = de && o.a < n_challenges; break;
      case PICO_Q_REGIONAL: ok = de && regional_sum; break;
      case PICO_Q_GLOBAL: ok = db && o.a < 14 && global_sum; break;
      case PICO_Q_ASSERT: ok = o.a < kQBaseRegs; break;
      case PICO_Q_EASSERT: ok = o.a < kQExtRegs; break;
      default: ok = false;
    }
    if (!ok) {
      set_error("quotient_values: program instruction %u (op %u, dst %u, a %u, b %u) is out of range", k, o.op,
                o.dst, o.a, o.b);
      return PICO_ERR_INVALID_ARG;
    }
    // registers named (in range, checked above): which operands are base or extension registers
    auto base = [&](uint32_t r) { n_base = std::max(n_base, r + 1); };
    auto ext = [&](uint32_t r) { n_ext = std::max(n_ext, r + 1); };
    switch (o.op) {
      case PICO_Q_MAIN: case PICO_Q_PREP: case PICO_Q_CONST: case PICO_Q_PUBLIC: case PICO_Q_FIRST:
      case PICO_Q_LAST: case PICO_Q_TRANSITION: case PICO_Q_GLOBAL: base(o.dst); break;
      case PICO_Q_ADD: case PICO_Q_SUB: case PICO_Q_MUL: base(o.dst); base(o.a); base(o.b); break;
      case PICO_Q_PERM: case PICO_Q_CHALLENGE: case PICO_Q_REGIONAL: ext(o.dst); break;
      case PICO_Q_EADD: case PICO_Q_ESUB: case PICO_Q_EMUL: ext(o.dst); ext(o.a); ext(o.b); break;
      case PICO_Q_EMB: ext(o.dst); base(o.a); break;
      case PICO_Q_EMULB: ext(o.dst); ext(o.a); base(o.b); break;
      case PICO_Q_ASSERT: base(o.a); n_asserts++; break;
      case PICO_Q_EASSERT: ext(o.a); n_asserts++; break;
      default: break;
    }
  }
  size_t smem = (size_t)(n_base + 4 * n_ext) * kQThreads * 4;  // at most kQGeneralSmem
  const uint64_t Q = 1ull << log_q;
  const unsigned grid = (unsigned)((Q + kQThreads - 1) / kQThreads);
  const ProgramShape shape(program, n_ops, wm, wp, we / 4);
  const bool staged = shape.prefer_staged(shape.words + 3 + n_base + 4 * n_ext, grid, 4 * Q * ((uint64_t)wm + wp + we),
                                          (uint32_t)ctx->sm_count);
  const StagedProgram sp = staged ? StagedProgram(program, n_ops, shape, public_values, global_sum) : StagedProgram();
  const bool out_dev = flags & PICO_OUTPUT_DEVICE;
  // one device block: program, assertion powers, public values, challenges, constants, then the output if on the host
  const uint64_t w_ops = 4ull * (staged ? sp.ops.size() : n_ops), w_pow = staged ? 4ull * n_asserts : 0, w_pub = n_public, w_chal = 4ull * n_challenges;
  const uint64_t w_const = 18;
  const uint64_t o_pub = w_ops + w_pow, o_chal = o_pub + w_pub, o_const = o_chal + w_chal, o_cols = o_const + w_const;
  const uint64_t w_in = o_cols + (staged ? sp.cols.size() : 0);
  const uint64_t off_out = (w_in + 63) & ~63ull;
  const uint64_t bytes = 4 * (off_out + (out_dev ? 0 : 4 * Q));
  if (!try_reserve(ctx, bytes)) {
    set_error("quotient_values: HBM budget exceeded");
    return PICO_ERR_OUT_OF_MEMORY;
  }
  cudaSetDevice(ctx->device);
  cudaStream_t st = pick_stream(ctx);
  uint32_t* blk = nullptr;
  if ((s = device_alloc((void**)&blk, bytes, st))) {
    unreserve(ctx, bytes);
    return s;
  }
  std::vector<uint32_t> host(w_in, 0);
  if (staged) {
    memcpy(host.data(), sp.ops.data(), 4 * w_ops);
    if (!sp.cols.empty()) memcpy(host.data() + o_cols, sp.cols.data(), 4 * sp.cols.size());
    smem = (size_t)sp.stride * kQThreads * 4;
    if (field == PICO_KOALABEAR) assertion_powers<KoalaBear>(alpha, n_asserts, host.data() + w_ops);
    else assertion_powers<BabyBear>(alpha, n_asserts, host.data() + w_ops);
  } else {
    if (n_ops) memcpy(host.data(), program, 16ull * n_ops);
  }
  if (n_public) memcpy(host.data() + o_pub, public_values, 4ull * n_public);
  if (n_challenges) memcpy(host.data() + o_chal, perm_challenges, 16ull * n_challenges);
  uint32_t* cst = host.data() + o_const;
  if (regional_sum) memcpy(cst, regional_sum, 16);
  if (global_sum) memcpy(cst + 4, global_sum, 56);
  s = cuda_status(cudaMemcpyAsync(blk, host.data(), 4 * w_in, cudaMemcpyHostToDevice, st), "program upload");
  QuotientArgs A;
  A.main = pm;
  A.prep = pp;
  A.perm = pe;
  A.main_w = wm;
  A.prep_w = wp;
  A.perm_w = we;
  A.ops = reinterpret_cast<const uint4*>(blk);
  A.n_ops = staged ? (uint32_t)sp.ops.size() - 1 : n_ops;
  A.powers = reinterpret_cast<const uint4*>(blk + w_ops);
  A.pub = blk + o_pub;
  A.chal = blk + o_chal;
  A.consts = blk + o_const;
  A.log_trace = log_trace_height;
  A.log_qd = log_quotient_degree;
  A.n_base = n_base;
  memcpy(A.alpha, alpha, 16);
  A.shift_n = field == PICO_KOALABEAR ? shift_power<KoalaBear>(log_trace_height) : shift_power<BabyBear>(log_trace_height);
  A.stride = sp.stride;
  memcpy(A.cols_end, sp.cols_end, sizeof(A.cols_end));
  A.cols = blk + o_cols;
  A.chunks = (flags & PICO_QUOTIENT_CHUNKS) ? 1u : 0u;
  A.out = out_dev ? out : blk + off_out;
  const TwiddleTables tw = twiddles(ctx, field);
  if (!s) {
    void (*const kernel)(QuotientArgs, TwiddleTables) =
        field == PICO_KOALABEAR ? (staged ? k_quotient_staged<KoalaBear> : k_quotient<KoalaBear>)
                                : (staged ? k_quotient_staged<BabyBear> : k_quotient<BabyBear>);
    // the form's maximum and not this program's size: the attribute is the
    // process's, and another thread may set it between here and the launch
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(staged ? kQStagedSmem : kQGeneralSmem));
    if (!e) kernel<<<grid, kQThreads, smem, st>>>(A, tw);
    s = cuda_status(e ? e : cudaGetLastError(), "quotient kernel");
  }
  if (!s && !out_dev)
    s = cuda_status(cudaMemcpyAsync(out, blk + off_out, 16 * Q, cudaMemcpyDeviceToHost, st), "quotient read-back");
  cudaFreeAsync(blk, st);
  pico_status s2 = cuda_status(cudaStreamSynchronize(st), "quotient_values");
  unreserve(ctx, bytes);
  return s ? s : s2;
}
