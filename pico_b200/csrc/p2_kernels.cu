// Poseidon2 kernels: batch permutation, Merkle row hashing (PaddingFreeSponge
// rate 8, overwrite mode), 2-to-1 compression with mixed-height injection,
// FRI fold, and the device-side duplex challenger.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <vector>

#include "field.cuh"
#include "internal.h"
#include "open.h"
#include "p2_lane.cuh"
#include "p2_tc.cuh"
#include "poseidon2.cuh"

namespace pico {

cudaError_t upload_p2_constants(int field, const uint32_t ext[8][16], const uint32_t* inte, int rounds_p,
                                const uint32_t diag[16]) {
  P2Constants h{};
  for (int r = 0; r < 8; r++)
    for (int j = 0; j < 16; j++) h.ext[r][j] = ext[r][j];
  for (int r = 0; r < rounds_p && r < 24; r++) h.inte[r] = inte[r];
  for (int j = 0; j < 16; j++) h.diag[j] = diag[j];
  cudaError_t e = cudaMemcpyToSymbol(c_p2, &h, sizeof h, sizeof(P2Constants) * (field ? 1 : 0));
  if (e) return e;
  std::vector<uint8_t> tables(kTcTableBytes);
  P2TcConstants tc;
  std::vector<uint32_t> lane(kLaneWords);
  if (!build_p2_tc_tables(field, h.ext, h.inte, h.diag, tables.data(), &tc, lane.data())) return cudaErrorInvalidValue;
  if ((e = cudaMemcpyToSymbol(g_p2_lane, lane.data(), kLaneWords * 4, (size_t)kLaneWords * 4 * (field ? 1 : 0)))) return e;
  if ((e = cudaMemcpyToSymbol(g_p2_tc, tables.data(), kTcTableBytes, (size_t)kTcTableBytes * (field ? 1 : 0)))) return e;
  return cudaMemcpyToSymbol(c_p2_tc, &tc, sizeof tc, sizeof tc * (field ? 1 : 0));
}

// From now on (tries >= 0) a wait for tensor-core products gives up after that
// many tries and none ever succeeds: the barriers need an arrival that nothing
// makes.  tries < 0: as built.
cudaError_t expire_tensor_waits(int64_t tries) {
  const uint32_t w[2] = {tries < 0 ? kTcWaitTries : (uint32_t)std::min<int64_t>(tries, kTcWaitTries), tries < 0 ? 1u : 2u};
  static_assert(offsetof(P2TcConstants, arrivals) == offsetof(P2TcConstants, wait_tries) + 4, "copied together");
  cudaError_t e = cudaSuccess;
  for (size_t f = 0; f < 2 && !e; f++)
    e = cudaMemcpyToSymbol(c_p2_tc, w, sizeof w, f * sizeof(P2TcConstants) + offsetof(P2TcConstants, wait_tries));
  return e ? e : cudaDeviceSynchronize();
}

// ---------------------------------------------------------------------------
template <class F>
__global__ void k_permute(uint32_t* states, uint64_t n) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[16];
  uint4* p = reinterpret_cast<uint4*>(states + 16 * i);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint4 v = p[k];
    s[4 * k] = v.x;
    s[4 * k + 1] = v.y;
    s[4 * k + 2] = v.z;
    s[4 * k + 3] = v.w;
  }
  p2_permute<F>(s);
#pragma unroll
  for (int k = 0; k < 4; k++) p[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
}

// Absorb row r of the concatenated group into a zeroed sponge state
// (PaddingFreeSponge<_,16,8,8>: overwrite s[0..k) with each chunk of up to 8
// elements, permute after each chunk; hash.rs:40-52).
// Bounds guard of the row hashing: a read stays inside its row segment by
// construction (rows are bounded by the launch, columns by the segment
// widths), so the guard sits where the cursor moves to the next segment: a
// move past the last segment is skipped (reads as zero), recorded in
// g_hash_guard, and reported by the entry points after their final
// synchronisation.
__device__ GuardRecord g_hash_guard;
__device__ __forceinline__ void hash_guard_trip(unsigned long long seg, unsigned long long col,
                                                unsigned long long tag = kGuardRowRead) {
  if (atomicAdd(&g_hash_guard.count, 1ull) == 0) {
    g_hash_guard.tag = tag;
    g_hash_guard.offset = seg;
    g_hash_guard.extent = col;
    g_hash_guard.block = blockIdx.x;
    g_hash_guard.thread = threadIdx.x;
  }
}
// For row_chunk: a read past the last segment.
struct RowReadTrip {
  __device__ __forceinline__ void operator()(uint32_t seg, uint32_t col) const { hash_guard_trip(seg, col); }
};
template <class F>
__device__ __forceinline__ void hash_row_segs(const RowSeg* segs, uint32_t n_segs, uint32_t W, uint64_t r,
                                              uint32_t s[16]) {
  uint32_t seg = 0, col = 0;
  uint32_t segw = n_segs ? segs[0].width : 0u;
  const uint32_t* rowp = n_segs ? segs[0].ptr + r * segw : nullptr;
  for (uint32_t base = 0; base < W; base += 8) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (base + j < W) {
        while (col == segw && seg < n_segs) {
          seg++;
          col = 0;
          segw = seg < n_segs ? segs[seg].width : 0u;
          rowp = seg < n_segs ? segs[seg].ptr + r * segw : nullptr;
        }
        if (seg >= n_segs) {
          hash_guard_trip(seg, col);
          s[j] = 0;
        } else {
          s[j] = __ldg(rowp + col);
        }
        col++;
      }
    }
    p2_permute<F>(s);
  }
}

template <class F>
__device__ __forceinline__ void hash_row(const RowGroup& g, uint64_t r, uint32_t s[16], uint64_t rows) {
  (void)rows;
  hash_row_segs<F>(g.segs, g.n_segs, g.total_width, r, s);
}

__device__ __forceinline__ void store_digest(uint32_t* out, const uint32_t s[16]) {
  uint4* o = reinterpret_cast<uint4*>(out);
  o[0] = make_uint4(s[0], s[1], s[2], s[3]);
  o[1] = make_uint4(s[4], s[5], s[6], s[7]);
}

// Row digests of several height groups, one thread per row of any group:
// the groups' sponges, short and latency-bound when a group has few rows,
// run side by side instead of one launch after another.
template <class F>
__global__ void __launch_bounds__(256, 5) k_hash_groups(const __grid_constant__ GroupBatch b) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (b.n_groups == 0 || b.n_groups > (uint32_t)kBatchGroups || t >= b.row_end[b.n_groups - 1]) return;
  uint32_t g = 0;
  while (g + 1 < b.n_groups && t >= b.row_end[g]) g++;
  const uint64_t r = t - (g ? b.row_end[g - 1] : 0ull);
  const uint32_t s0 = b.seg_begin[g], s1 = b.seg_begin[g + 1];
  if (s1 < s0 || s1 > (uint32_t)kBatchSegs) {
    hash_guard_trip(s0, s1);
    return;
  }
  uint32_t s[16];
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = 0;
  hash_row_segs<F>(b.segs + s0, s1 - s0, b.width[g], r, s);
  store_digest(b.out[g] + 8 * r, s);
}

template <class F>
// (256, 5): 48 registers at 5/8 occupancy.  Measured on a 2^30-cell commit,
// leaf hashing takes 34.4 ms at (256, 8) (32 registers, full occupancy),
// 34.1 at (256, 6), 33.2 here and 33.4 at (256, 4): the permutation's
// instruction scheduling gains more from registers than from warps.
__global__ void __launch_bounds__(256, 5) k_hash_rows(const __grid_constant__ RowGroup g, uint64_t rows, uint32_t* out) {
  uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r >= rows) return;
  uint32_t s[16];
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = 0;
  hash_row<F>(g, r, s, rows);
  store_digest(out + 8 * r, s);
}

// The same sponge, resumable: absorb the group's columns into a state that a
// previous call left in state_in (nullptr: the zero state), the first column
// going to rate position pos0 of the current chunk (the previous call's
// columns mod 8).  A call that is not the last stores the whole state to
// state_out, including a partly overwritten chunk that is not yet permuted;
// the last call permutes after its final (possibly partial) chunk, as the
// one-pass sponge does, and writes the digest.  Absorbing a row's matrices
// one call at a time gives the one-pass digest exactly.
template <class F>
__global__ void __launch_bounds__(256, 5)
    k_absorb_rows(const __grid_constant__ RowGroup g, uint64_t rows, uint32_t pos0, const uint32_t* state_in,
                  uint32_t* state_out, uint32_t* digest_out) {
  uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r >= rows) return;
  uint32_t s[16];
  if (state_in) {
    // plain loads: state_in may be state_out (each thread rereads its own row)
    const uint4* p = reinterpret_cast<const uint4*>(state_in + 16 * r);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 v = p[k];
      s[4 * k] = v.x;
      s[4 * k + 1] = v.y;
      s[4 * k + 2] = v.z;
      s[4 * k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; i++) s[i] = 0;
  }
  const int W = (int)g.total_width;
  const int end = (int)pos0 + W;  // positions pos0 .. end-1 of the chunk sequence
  uint32_t seg = 0, col = 0;
  uint32_t segw = g.segs[0].width;
  const uint32_t* rowp = g.segs[0].ptr + r * segw;
  for (int base = 0; base < end; base += 8) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int c = base + j;  // chunk position; column c - pos0 of this call
      if (c >= (int)pos0 && c < end) {
        while (col == segw && seg < g.n_segs) {
          seg++;
          col = 0;
          segw = seg < g.n_segs ? g.segs[seg].width : 0u;
          rowp = g.segs[seg < g.n_segs ? seg : 0].ptr + r * segw;
        }
        if (seg >= g.n_segs) {
          hash_guard_trip(seg, col);
          s[j] = 0;
        } else {
          s[j] = __ldg(rowp + col);
        }
        col++;
      }
    }
    if (base + 8 <= end || digest_out) p2_permute<F>(s);
  }
  if (digest_out) {
    store_digest(digest_out + 8 * r, s);
  } else {
    uint4* o = reinterpret_cast<uint4*>(state_out + 16 * r);
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
  }
}

// next[i] = compress(prev[2i], prev[2i+1]); where a matrix height meets this
// level, next[i] = compress(next[i], inj[i]) with inj[i] the digest of the
// concatenated rows i of those matrices (TruncatedPermutation, hash.rs:89-94;
// injection order of the verifier, fri.rs:389-436).
template <class F>
__global__ void __launch_bounds__(256)
    k_compress(const uint32_t* prev, uint32_t* next, uint64_t n, const uint32_t* inj) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t s[16];
  const uint4* p = reinterpret_cast<const uint4*>(prev + 16 * i);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint4 v = __ldg(p + k);
    s[4 * k] = v.x;
    s[4 * k + 1] = v.y;
    s[4 * k + 2] = v.z;
    s[4 * k + 3] = v.w;
  }
  p2_permute<F>(s);
  if (inj) {
    const uint4* q = reinterpret_cast<const uint4*>(inj + 8 * i);
    const uint4 a = __ldg(q), b = __ldg(q + 1);
    s[8] = a.x;
    s[9] = a.y;
    s[10] = a.z;
    s[11] = a.w;
    s[12] = b.x;
    s[13] = b.y;
    s[14] = b.z;
    s[15] = b.w;
    p2_permute<F>(s);
  }
  store_digest(next + 8 * i, s);
}

// ---------------------------------------------------------------------------
// One word per lane (p2_lane.cuh): 16 lanes per state, for the levels and
// rows too few to fill the GPU.
constexpr uint32_t kLaneThreads = 256;  // 16 states per CTA

// Row digests of a GroupBatch, 16 lanes per row (k_hash_groups' sponges): lanes
// 0..7 carry the rate, so a chunk's eight words are one load.
template <class F>
__global__ void __launch_bounds__(kLaneThreads) k_hash_groups_lane(const __grid_constant__ GroupBatch b) {
  __shared__ __align__(16) uint32_t tab[kLaneWords];
  lane_load_tables<F>(tab);
  __syncthreads();
  if (b.n_groups == 0 || b.n_groups > (uint32_t)kBatchGroups) return;
  const uint64_t t = blockIdx.x * (uint64_t)kLaneThreads + threadIdx.x;
  const uint64_t row = t >> 4;
  const uint32_t q = (uint32_t)(t & 15);
  const bool live = row < b.row_end[b.n_groups - 1];
  uint32_t g = 0;
  while (g + 1 < b.n_groups && row >= b.row_end[g]) g++;
  const uint64_t r = row - (g ? b.row_end[g - 1] : 0ull);
  const uint32_t s0 = b.seg_begin[g], s1 = b.seg_begin[g + 1];
  uint32_t W = live ? b.width[g] : 0u;
  if (s1 < s0 || s1 > (uint32_t)kBatchSegs) {
    hash_guard_trip(s0, s1);
    W = 0;
  }
  // the two rows of a warp may differ in width: the warp runs the longer one's
  // chunks, the other keeps its digest
  const uint32_t chunks = (W + 7) / 8;
  const uint32_t steps = max(chunks, __shfl_xor_sync(0xffffffffu, chunks, 16));
  uint32_t seg = s0, begin = 0;  // this lane's segment and its first column
  uint32_t v = 0;
  for (uint32_t c = 0; c < steps; c++) {
    const uint32_t col = 8 * c + q;
    uint32_t w = v;
    if (q < 8 && col < W) {
      while (seg < s1 && col - begin >= b.segs[seg].width) begin += b.segs[seg++].width;
      if (seg >= s1) {
        hash_guard_trip(seg, col);
        w = 0;
      } else {
        w = __ldg(b.segs[seg].ptr + r * b.segs[seg].width + (col - begin));
      }
    }
    w = lane_permute<F>(w, q, tab);
    if (c < chunks) v = w;
  }
  if (live && q < 8) b.out[g][8 * r + q] = v;
}

// k_absorb_rows with 16 lanes per row.
template <class F>
__global__ void __launch_bounds__(kLaneThreads)
    k_absorb_rows_lane(const __grid_constant__ RowGroup g, uint64_t rows, uint32_t pos0, const uint32_t* state_in,
                       uint32_t* state_out, uint32_t* digest_out) {
  __shared__ __align__(16) uint32_t tab[kLaneWords];
  lane_load_tables<F>(tab);
  __syncthreads();
  const uint64_t t = blockIdx.x * (uint64_t)kLaneThreads + threadIdx.x;
  const uint64_t r = t >> 4;
  const uint32_t q = (uint32_t)(t & 15);
  const bool live = r < rows;
  uint32_t v = live && state_in ? state_in[16 * r + q] : 0u;
  const uint32_t end = pos0 + g.total_width;
  uint32_t seg = 0, begin = 0;  // this lane's segment and its first column
  for (uint32_t base = 0; base < end; base += 8) {
    const uint32_t c = base + q;  // chunk position; column c - pos0 of this call
    if (live && q < 8 && c >= pos0 && c < end) {
      const uint32_t col = c - pos0;
      while (seg < g.n_segs && col - begin >= g.segs[seg].width) begin += g.segs[seg++].width;
      if (seg >= g.n_segs) {
        hash_guard_trip(seg, col);
        v = 0;
      } else {
        v = __ldg(g.segs[seg].ptr + r * g.segs[seg].width + (col - begin));
      }
    }
    if (base + 8 <= end || digest_out) v = lane_permute<F>(v, q, tab);
  }
  if (!live) return;
  if (!digest_out)
    state_out[16 * r + q] = v;
  else if (q < 8)
    digest_out[8 * r + q] = v;
}

// Duplex challenger (challenger.rs:89-115, 202-237) held by the 16 lanes of a
// warp's halves: lane q has sponge word q and buffer words q mod 8.
template <class F>
struct LaneChallenger {
  uint32_t sponge, in, out, in_len, out_len;
  __device__ __forceinline__ void load(const DevChallenger* ch, uint32_t q) {
    sponge = ch->sponge[q];
    in = ch->in_buf[q & 7];
    out = ch->out_buf[q & 7];
    in_len = ch->in_len;
    out_len = ch->out_len;
  }
  __device__ __forceinline__ void store(DevChallenger* ch, uint32_t q) const {
    ch->sponge[q] = sponge;
    if (q < 8) {
      ch->in_buf[q] = in;
      ch->out_buf[q] = out;
    }
    if (q == 0) {
      ch->in_len = in_len;
      ch->out_len = out_len;
    }
  }
  __device__ __forceinline__ void duplex(uint32_t q, const uint32_t* tab) {
    sponge = lane_permute<F>(q < in_len ? in : sponge, q, tab);
    in_len = 0;
    out = __shfl_sync(0xffffffffu, sponge, (int)(q & 7), 16);
    out_len = 8;
  }
  __device__ __forceinline__ void observe(uint32_t value, uint32_t q, const uint32_t* tab) {
    out_len = 0;
    if ((q & 7) == in_len) in = value;
    if (++in_len == 8) duplex(q, tab);
  }
  __device__ __forceinline__ uint32_t sample(uint32_t q, const uint32_t* tab) {
    if (in_len != 0 || out_len == 0) duplex(q, tab);
    return __shfl_sync(0xffffffffu, out, (int)--out_len, 16);
  }
};

// Levels of a tree above `n` nodes (a power of two), in one CTA, in shared
// memory: cur holds the nodes, spare is as large as half of them; every level is written
// after the previous one (in the whole tree the level holds total nodes, this
// CTA's are those from c * n).  Returns the buffer that holds the last node.
constexpr uint32_t kSubtreeThreads = 512;
template <class F>
__device__ __forceinline__ uint32_t* lane_subtree(uint32_t* cur, uint32_t* spare, uint32_t n, uint32_t* level,
                                                  uint64_t total, uint64_t c, const SubtreeInj* inj,
                                                  const uint32_t* tab) {
  const uint32_t q = threadIdx.x & 15, g = threadIdx.x >> 4;
  uint32_t lvl = 0;
  while (n > 1) {
    const uint32_t m = n >> 1;
    uint32_t* out = level + 8 * total;
    const uint32_t* d = inj ? inj->digests[lvl] : nullptr;
    for (uint32_t s = 0; s < m; s += kSubtreeThreads / 16) {
      if (s + (threadIdx.x >> 5) * 2 >= m) break;  // warp-uniform
      const uint32_t node = s + g;
      const bool live = node < m;
      uint32_t v = live ? cur[16 * node + q] : 0u;
      uint32_t w = 0;
      if (d && live && q >= 8) w = d[(c * m + node) * 8 + q - 8];
      v = lane_permute<F>(v, q, tab);
      if (d) {
        if (q >= 8) v = w;
        v = lane_permute<F>(v, q, tab);
      }
      if (live && q < 8) {
        spare[8 * node + q] = v;
        out[(c * m + node) * 8 + q] = v;
      }
    }
    __syncthreads();
    uint32_t* t = cur;
    cur = spare;
    spare = t;
    level = out;
    total >>= 1;
    n = m;
    lvl++;
  }
  return cur;
}

// The levels above CTA c's nodes [c * n, (c + 1) * n) of a level of n_in nodes;
// with a challenger (one CTA only), then observe the root and sample the EF4
// challenge into beta_out.
template <class F>
__global__ void __launch_bounds__(kSubtreeThreads)
    k_subtree_lane(uint32_t* level, uint32_t n_in, uint32_t n, const __grid_constant__ SubtreeInj inj,
                   DevChallenger* ch, uint32_t* beta_out) {
  __shared__ __align__(16) uint32_t tab[kLaneWords];
  __shared__ __align__(16) uint32_t buf[(kSubtreeMaxIn + kSubtreeMaxIn / 2) * 8];
  lane_load_tables<F>(tab);
  if (n > kSubtreeMaxIn || (uint64_t)(blockIdx.x + 1) * n > n_in) return;  // the launcher checks both
  const uint32_t* src = level + (size_t)blockIdx.x * n * 8;
  for (uint32_t i = threadIdx.x; i < n * 8; i += kSubtreeThreads) buf[i] = src[i];
  __syncthreads();
  const uint32_t* root = lane_subtree<F>(buf, buf + kSubtreeMaxIn * 8, n, level, n_in, blockIdx.x, &inj, tab);
  if (ch && threadIdx.x < 32) {
    const uint32_t q = threadIdx.x & 15;
    LaneChallenger<F> c;
    c.load(ch, q);
    for (int i = 0; i < 8; i++) c.observe(root[i], q, tab);
    uint32_t beta = 0;
    for (uint32_t i = 0; i < 4; i++) {
      const uint32_t b = c.sample(q, tab);
      if (q == i) beta = b;
    }
    if (threadIdx.x < 4) beta_out[threadIdx.x] = beta;
    if (threadIdx.x < 16) c.store(ch, q);
  }
}

template <class F>
__global__ void k_challenger_observe(DevChallenger* ch, const uint32_t* vals, uint32_t n) {
  __shared__ __align__(16) uint32_t tab[kLaneWords];
  lane_load_tables<F>(tab);
  __syncthreads();
  const uint32_t q = threadIdx.x & 15;
  LaneChallenger<F> c;
  c.load(ch, q);
  for (uint32_t i = 0; i < n; i++) c.observe(vals[i], q, tab);
  if (threadIdx.x < 16) c.store(ch, q);
}

// ---------------------------------------------------------------------------
// Tensor-core forms (p2_tc.cuh): groups of 128 threads own 128 states each; a
// CTA of 512 threads holds four groups, which share the tables, and an SM two
// CTAs (eight groups of 64 TMEM columns).

__host__ __device__ static inline uint64_t tc_tiles(uint64_t n) { return (n + kTcThreads - 1) / kTcThreads; }
#define PICO_TC_OPEN(F)                                  \
  extern __shared__ __align__(128) uint8_t tc_tables[];  \
  __shared__ __align__(8) uint64_t tc_bar[kTcGroups];    \
  __shared__ uint32_t tc_slot;                           \
  P2Tc<F> tc;                                            \
  tc.open(tc_tables, tc_bar, &tc_slot)
#define PICO_TC_CLOSE()                                          \
  tc.close();                                                    \
  if (tc.dead) hash_guard_trip(0, 0, kGuardTensorWait)

template <class F>
__global__ void __launch_bounds__(kTcThreads * kTcGroups, kTcCtas) k_permute_tc(uint32_t* states, uint64_t n, volatile uint32_t* expired) {
  PICO_TC_OPEN(F);
  for (uint64_t t0 = tc.first_tile(tc_tiles(n)) * kTcThreads; t0 < n; t0 += tc.tile_stride() * kTcThreads) {
    const uint64_t i = t0 + threadIdx.x % kTcThreads;
    uint32_t s[16];
    uint4* p = reinterpret_cast<uint4*>(states + 16 * (i < n ? i : n - 1));
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 v = p[k];
      s[4 * k] = v.x;
      s[4 * k + 1] = v.y;
      s[4 * k + 2] = v.z;
      s[4 * k + 3] = v.w;
    }
    tc.put_state(s);
    tc.body(kTcFromState);
    tc.output(s);
    if (i < n) {
#pragma unroll
      for (int k = 0; k < 4; k++) p[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
    }
  }
  tc.close();
  if (tc.dead) *expired = *expired + 1;  // the host looks for any change
}

// Row digests of a GroupBatch (k_hash_groups' sponges).  Tiles of 128 rows do
// not cross groups, so a CTA's rows have one width.
template <class F>
__global__ void __launch_bounds__(kTcThreads * kTcGroups, kTcCtas) k_hash_groups_tc(const __grid_constant__ GroupBatch b, uint64_t tiles_all) {
  PICO_TC_OPEN(F);
  uint64_t tile = tc.first_tile(tiles_all);
  uint32_t g = 0;
  uint64_t row0 = 0, first = 0;  // of group g: its first global row, its first tile
  const uint32_t n_groups = b.n_groups <= (uint32_t)kBatchGroups ? b.n_groups : 0u;
  for (; g < n_groups;) {
    const uint64_t rows = b.row_end[g] - row0, tiles = (rows + kTcThreads - 1) / kTcThreads;
    if (tile >= first + tiles) {
      first += tiles;
      row0 = b.row_end[g];
      g++;
      continue;
    }
    const uint64_t r = (tile - first) * kTcThreads + threadIdx.x % kTcThreads;
    const uint64_t rr = r < rows ? r : rows - 1;
    const uint32_t s0 = b.seg_begin[g], s1 = b.seg_begin[g + 1], W = b.width[g];
    uint32_t s[16];
#pragma unroll
    for (int k = 0; k < 16; k++) s[k] = 0;
    if (s1 < s0 || s1 > (uint32_t)kBatchSegs) {
      hash_guard_trip(s0, s1);
    } else {
      const RowSeg* segs = b.segs + s0;
      RowCursor cur;
      row_cursor_begin(cur, segs, s1 - s0, rr);
      for (uint32_t base = 0; base < W; base += 8) {
        const int hi = W - base < 8 ? (int)(W - base) : 8;
        TcInput from = base ? kTcFromSponge : kTcFromRate;
        if (base && hi < 8) {  // a partial chunk keeps the other rate words: through registers
          tc.output(s);
          from = kTcFromState;
        }
        row_chunk(cur, segs, s1 - s0, rr, 0, hi, s, RowReadTrip());
        if (from == kTcFromState)
          tc.put_state(s);
        else
          tc.put_rate(s);
        tc.body(from);
      }
      if (W) tc.digest(s);
    }
    if (r < rows) store_digest(b.out[g] + 8 * r, s);
    tile += tc.tile_stride();
  }
  PICO_TC_CLOSE();
}

// k_absorb_rows on the tensor cores.
template <class F>
__global__ void __launch_bounds__(kTcThreads * kTcGroups, kTcCtas)
    k_absorb_rows_tc(const __grid_constant__ RowGroup g, uint64_t rows, uint32_t pos0, const uint32_t* state_in,
                     uint32_t* state_out, uint32_t* digest_out) {
  PICO_TC_OPEN(F);
  for (uint64_t t0 = tc.first_tile(tc_tiles(rows)) * kTcThreads; t0 < rows; t0 += tc.tile_stride() * kTcThreads) {
    const uint64_t r = t0 + threadIdx.x % kTcThreads, rr = r < rows ? r : rows - 1;
    uint32_t s[16];
    if (state_in) {
      const uint4* p = reinterpret_cast<const uint4*>(state_in + 16 * rr);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint4 v = p[k];
        s[4 * k] = v.x;
        s[4 * k + 1] = v.y;
        s[4 * k + 2] = v.z;
        s[4 * k + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 16; k++) s[k] = 0;
    }
    const int end = (int)(pos0 + g.total_width);
    bool held = true;  // the state is in s (else its last S-boxes are in TMEM)
    RowCursor cur;
    row_cursor_begin(cur, g.segs, g.n_segs, rr);
    for (int base = 0; base < end; base += 8) {
      const int lo = base < (int)pos0 ? (int)pos0 - base : 0, hi = end - base < 8 ? end - base : 8;
      const bool permute = base + 8 <= end || digest_out;
      const bool full = lo == 0 && hi == 8;
      if (!held && !full) {
        tc.output(s);
        held = true;
      }
      row_chunk(cur, g.segs, g.n_segs, rr, lo, hi, s, RowReadTrip());
      if (!permute) break;
      if (held)
        tc.put_state(s);
      else
        tc.put_rate(s);
      tc.body(held ? kTcFromState : kTcFromSponge);
      held = false;
    }
    if (digest_out) {
      if (!held) tc.digest(s);
      if (r < rows) store_digest(digest_out + 8 * r, s);
    } else {
      if (!held) tc.output(s);
      if (r < rows) {
        uint4* o = reinterpret_cast<uint4*>(state_out + 16 * r);
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = make_uint4(s[4 * k], s[4 * k + 1], s[4 * k + 2], s[4 * k + 3]);
      }
    }
  }
  PICO_TC_CLOSE();
}

// k_compress on the tensor cores.
template <class F>
__global__ void __launch_bounds__(kTcThreads * kTcGroups, kTcCtas)
    k_compress_tc(const uint32_t* prev, uint32_t* next, uint64_t n, const uint32_t* inj) {
  PICO_TC_OPEN(F);
  for (uint64_t t0 = tc.first_tile(tc_tiles(n)) * kTcThreads; t0 < n; t0 += tc.tile_stride() * kTcThreads) {
    const uint64_t i = t0 + threadIdx.x % kTcThreads, ii = i < n ? i : n - 1;
    uint32_t s[16];
    const uint4* p = reinterpret_cast<const uint4*>(prev + 16 * ii);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 v = p[k];
      s[4 * k] = v.x;
      s[4 * k + 1] = v.y;
      s[4 * k + 2] = v.z;
      s[4 * k + 3] = v.w;
    }
    for (int pass = 0;; pass++) {
      tc.put_state(s);
      tc.body(kTcFromState);
      tc.digest(s);
      if (!inj || pass) break;
      const uint4* q = reinterpret_cast<const uint4*>(inj + 8 * ii);
      const uint4 a = q[0], c = q[1];
      s[8] = a.x;
      s[9] = a.y;
      s[10] = a.z;
      s[11] = a.w;
      s[12] = c.x;
      s[13] = c.y;
      s[14] = c.z;
      s[15] = c.w;
    }
    if (i < n) store_digest(next + 8 * i, s);
  }
  PICO_TC_CLOSE();
}

// Row hashing takes a CTA per kTcGroups tiles from this many permutations a
// row on: the hardware then balances groups of different widths, and the
// set-up (the tables into shared memory) is a small part.  A commit of 2^30
// cells and 16 requests of small traces: 65.5 and 4.72 ms with 4, 66.4 and 5.03
// with 16; with 48 recursion traces a full wave of looping CTAs took 420 ms
// against 405.
constexpr uint64_t kTcWholeChunks = 4;
// Launch a tensor-core kernel over `tiles` tiles: a full wave of CTAs, each
// looping over its share, or (whole) a CTA per kTcGroups tiles.
template <class... P, class... A>
static cudaError_t tc_launch(bool chained, void (*kernel)(P...), uint64_t tiles, bool whole, cudaStream_t st, A... args) {
  uint64_t ctas = tiles;
  if (ctas > kTcResident) ctas = whole ? std::max<uint64_t>((tiles + kTcGroups - 1) / kTcGroups, kTcResident) : kTcResident;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmemBytes);
  if (e) return e;
  return launch_chained(chained, kernel, (unsigned)ctas, kTcThreads * kTcGroups, kTcSmemBytes, st, args...);
}

// ---------------------------------------------------------------------------
static inline unsigned blocks_for(uint64_t n, unsigned bs) { return (unsigned)((n + bs - 1) / bs); }

// Four threads per state (the latency form).  Every thread of a launched warp
// takes part in the shuffles; threads past the last state permute zeros and
// store nothing.
template <class F>
__global__ void __launch_bounds__(256) k_permute_quad(uint32_t* states, uint64_t n) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t i = t >> 2;
  const uint32_t q = (uint32_t)(t & 3);
  const bool live = i < n;
  uint32_t v[4];
  if (live) {
    const uint4 a = reinterpret_cast<const uint4*>(states + 16 * i)[q];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  } else {
    v[0] = v[1] = v[2] = v[3] = 0;
  }
  p2_permute_quad<F>(v, q, 0xffffffffu);
  if (live) reinterpret_cast<uint4*>(states + 16 * i)[q] = make_uint4(v[0], v[1], v[2], v[3]);
}

cudaError_t launch_permute(int field, uint32_t* states, uint64_t n, cudaStream_t st, bool four_lanes,
                           uint32_t* expired) {
  if (n == 0) return cudaSuccess;
  if (four_lanes) {
    if (field == 0)
      k_permute_quad<KoalaBear><<<blocks_for(4 * n, 256), 256, 0, st>>>(states, n);
    else
      k_permute_quad<BabyBear><<<blocks_for(4 * n, 256), 256, 0, st>>>(states, n);
    return cudaGetLastError();
  }
  if (n >= kTcMinStates) {
    return tc_launch(false, field == 0 ? k_permute_tc<KoalaBear> : k_permute_tc<BabyBear>, tc_tiles(n), false, st, states,
                     n, expired);
  }
  if (field == 0)
    k_permute<KoalaBear><<<blocks_for(n, 256), 256, 0, st>>>(states, n);
  else
    k_permute<BabyBear><<<blocks_for(n, 256), 256, 0, st>>>(states, n);
  return cudaGetLastError();
}

cudaError_t hash_guard_fetch(GuardRecord* dst, cudaStream_t st) {
  return cudaMemcpyFromSymbolAsync(dst, g_hash_guard, sizeof(GuardRecord), 0, cudaMemcpyDeviceToHost, st);
}
cudaError_t hash_guard_clear() {
  const GuardRecord z{};
  return cudaMemcpyToSymbol(g_hash_guard, &z, sizeof z);
}

// Rows are hashed on the tensor cores when there are enough states for one
// permutation, or, where each takes several, from kTcMinRows on.
static bool use_tensor_rows(uint64_t rows, uint64_t chunks) {
  return rows >= kTcMinStates || (rows >= kTcMinRows && chunks >= 2);
}
// A batch of one group.
static GroupBatch one_group(const RowGroup& g, uint64_t rows, uint32_t* out) {
  GroupBatch b;
  memset(&b, 0, sizeof b);
  b.n_groups = 1;
  b.n_segs = g.n_segs;
  b.row_end[0] = rows;
  b.out[0] = out;
  b.seg_begin[1] = g.n_segs;
  b.width[0] = g.total_width;
  for (uint32_t k = 0; k < g.n_segs; k++) b.segs[k] = g.segs[k];
  return b;
}

// block: threads per CTA, 32 .. 256 (the kernels are bounded to 256), where
// rows are hashed one thread each.
cudaError_t launch_hash_rows(int field, const RowGroup& g, uint64_t rows, uint32_t* out, cudaStream_t st,
                             unsigned block) {
  if (rows == 0) return cudaSuccess;
  if (use_tensor_rows(rows, (g.total_width + 7) / 8) || rows <= kLaneMaxStates)
    return launch_hash_groups(field, one_group(g, rows, out), st, block);
  if (block < 32 || block > 256) block = 256;
  if (field == 0)
    k_hash_rows<KoalaBear><<<blocks_for(rows, block), block, 0, st>>>(g, rows, out);
  else
    k_hash_rows<BabyBear><<<blocks_for(rows, block), block, 0, st>>>(g, rows, out);
  return cudaGetLastError();
}

cudaError_t launch_hash_groups(int field, const GroupBatch& b, cudaStream_t st, unsigned block) {
  if (b.n_groups == 0) return cudaSuccess;
  if (b.n_groups > (uint32_t)kBatchGroups || b.n_segs > (uint32_t)kBatchSegs) return cudaErrorInvalidValue;
  const uint64_t rows = b.row_end[b.n_groups - 1];
  if (rows == 0) return cudaSuccess;
  uint64_t tiles = 0, chunks = 0;
  for (uint32_t g = 0; g < b.n_groups; g++) {
    const uint64_t t = tc_tiles(b.row_end[g] - (g ? b.row_end[g - 1] : 0ull));
    tiles += t;
    chunks += t * ((b.width[g] + 7) / 8);
  }
  if (use_tensor_rows(rows, chunks / tiles)) {
    return tc_launch(false, field == 0 ? k_hash_groups_tc<KoalaBear> : k_hash_groups_tc<BabyBear>, tiles,
                     chunks >= kTcWholeChunks * tiles, st, b, tiles);
  }
  if (rows <= kLaneMaxStates) {
    return launch_chained(false, field == 0 ? k_hash_groups_lane<KoalaBear> : k_hash_groups_lane<BabyBear>,
                          blocks_for(16 * rows, kLaneThreads), kLaneThreads, 0, st, b);
  }
  if (block < 32 || block > 256) block = 256;
  if (field == 0)
    k_hash_groups<KoalaBear><<<blocks_for(rows, block), block, 0, st>>>(b);
  else
    k_hash_groups<BabyBear><<<blocks_for(rows, block), block, 0, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_absorb_rows(int field, const RowGroup& g, uint64_t rows, uint32_t pos0, const uint32_t* state_in,
                               uint32_t* state_out, uint32_t* digest_out, cudaStream_t st, unsigned block) {
  if (rows == 0) return cudaSuccess;
  const uint64_t absorbed = pos0 + g.total_width;
  if (use_tensor_rows(rows, absorbed / 8)) {
    return tc_launch(false, field == 0 ? k_absorb_rows_tc<KoalaBear> : k_absorb_rows_tc<BabyBear>, tc_tiles(rows),
                     absorbed >= 8 * kTcWholeChunks, st,
                     g, rows, pos0, state_in, state_out, digest_out);
  }
  if (rows <= kLaneMaxStates) {
    return launch_chained(false, field == 0 ? k_absorb_rows_lane<KoalaBear> : k_absorb_rows_lane<BabyBear>,
                          blocks_for(16 * rows, kLaneThreads), kLaneThreads, 0, st, g, rows, pos0, state_in, state_out, digest_out);
  }
  if (block < 32 || block > 256) block = 256;
  if (field == 0)
    k_absorb_rows<KoalaBear><<<blocks_for(rows, block), block, 0, st>>>(g, rows, pos0, state_in, state_out,
                                                                        digest_out);
  else
    k_absorb_rows<BabyBear><<<blocks_for(rows, block), block, 0, st>>>(g, rows, pos0, state_in, state_out,
                                                                       digest_out);
  return cudaGetLastError();
}

// The same compression, four threads per node (the level of 2^14 nodes, too few
// to fill the GPU: one permutation's latency sets the launch's time).
template <class F>
__global__ void __launch_bounds__(256) k_compress_quad(const uint32_t* prev, uint32_t* next, uint64_t n,
                                                       const uint32_t* inj) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t i = t >> 2;
  const uint32_t q = (uint32_t)(t & 3);
  const bool live = i < n;
  uint32_t v[4] = {0, 0, 0, 0};
  if (live) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(prev + 16 * i) + q);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
  p2_permute_quad<F>(v, q, 0xffffffffu);
  if (inj) {
    // compress(digest, injected digest): lanes 0, 1 keep the digest, lanes 2, 3 load the injection
    if (q >= 2) {
      if (live) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(inj + 8 * i) + (q - 2));
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      } else {
        v[0] = v[1] = v[2] = v[3] = 0;
      }
    }
    p2_permute_quad<F>(v, q, 0xffffffffu);
  }
  if (live && q < 2) reinterpret_cast<uint4*>(next + 8 * i)[q] = make_uint4(v[0], v[1], v[2], v[3]);
}

cudaError_t launch_compress(int field, const uint32_t* prev, uint32_t* next, uint64_t n_next,
                            const uint32_t* inj_digests, cudaStream_t st, bool chained) {
  if (n_next == 0) return cudaSuccess;
  if (n_next <= kQuadMaxNodes) {
    if (field == 0)
      k_compress_quad<KoalaBear><<<blocks_for(4 * n_next, 256), 256, 0, st>>>(prev, next, n_next, inj_digests);
    else
      k_compress_quad<BabyBear><<<blocks_for(4 * n_next, 256), 256, 0, st>>>(prev, next, n_next, inj_digests);
    return cudaGetLastError();
  }
  if (n_next >= kTcMinStates) {
    return tc_launch(chained, field == 0 ? k_compress_tc<KoalaBear> : k_compress_tc<BabyBear>, tc_tiles(n_next), false, st,
                     prev, next, n_next, inj_digests);
  }
  if (field == 0)
    k_compress<KoalaBear><<<blocks_for(n_next, 256), 256, 0, st>>>(prev, next, n_next, inj_digests);
  else
    k_compress<BabyBear><<<blocks_for(n_next, 256), 256, 0, st>>>(prev, next, n_next, inj_digests);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FRI fold (TwoAdicFriGenericConfig::fold_matrix, mirrored by the verifier at
// vm/src/compiler/recursion/circuit/fri.rs:345-377): row r of the (len/2) x 2
// matrix (lo, hi) folds to
//   (lo + hi)/2 + (beta/2) * g_inv^rev(r) * (lo - hi),
// g = two_adic_generator(log len), rev over log(len/2) bits.  The pair is read
// at rows 2r, 2r+1 of cw; rg is its row in the whole codeword (r itself,
// except for one shard of a codeword split by rows).  Ordinary loads here and
// in half_beta: chained kernels call both (launch_chained).
template <class F>
__device__ __forceinline__ Ext4 fri_fold_row(const uint32_t* cw, uint32_t log_len, uint64_t r, const Ext4& hb,
                                             const TwiddleTables& tw, uint64_t rg) {
  using B = Fp<F>;
  using E = Ef<F>;
  // g_inv^rev(rg) = w_max^(-(rev(rg) << (S - log_len)))
  const uint32_t mask = (1u << F::TWO_ADICITY) - 1u;
  uint32_t e = (uint32_t)bitrev64(rg, (int)log_len - 1) << (F::TWO_ADICITY - log_len);
  e = (0u - e) & mask;
  uint32_t t = B::mul(__ldg(tw.hi + (e >> 14)), __ldg(tw.lo + (e & 0x3fffu)));
  const uint4 lo4 = reinterpret_cast<const uint4*>(cw)[2 * r];
  const uint4 hi4 = reinterpret_cast<const uint4*>(cw)[2 * r + 1];
  Ext4 lo{{lo4.x, lo4.y, lo4.z, lo4.w}}, hi{{hi4.x, hi4.y, hi4.z, hi4.w}};
  Ext4 sum = E::add(lo, hi), dif = E::sub(lo, hi);
  Ext4 res;
  Ext4 pd = E::mul(hb, E::scale(dif, t));
#pragma unroll
  for (int i = 0; i < 4; i++) res.c[i] = B::add(B::half(sum.c[i]), pd.c[i]);
  return res;
}

template <class F>
__device__ __forceinline__ Ext4 half_beta(const uint32_t* beta) {
  Ext4 hb;
#pragma unroll
  for (int i = 0; i < 4; i++) hb.c[i] = Fp<F>::half(beta[i]);
  return hb;
}

template <class F>
__global__ void k_fri_fold(const uint32_t* cw, uint32_t log_len, const uint32_t* beta, TwiddleTables tw,
                           uint32_t* out, const uint32_t* inject) {
  const uint64_t h = 1ull << (log_len - 1);
  uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r >= h) return;
  Ext4 res = fri_fold_row<F>(cw, log_len, r, half_beta<F>(beta), tw, r);
  if (inject) {
    const uint4 v = reinterpret_cast<const uint4*>(inject)[r];
    res = Ef<F>::add(res, Ext4{{v.x, v.y, v.z, v.w}});
  }
  reinterpret_cast<uint4*>(out)[r] = make_uint4(res.c[0], res.c[1], res.c[2], res.c[3]);
}

// Fold, then hash the next round's leaves in the same pass: thread k folds
// rows 2k and 2k+1 (adding the injected reduced opening), stores them, and
// hashes the pair as one 8-element leaf (one permutation: the rate block is
// the row, PaddingFreeSponge over 8 elements).
template <class F>
__global__ void __launch_bounds__(256) k_fri_fold_hash(const uint32_t* cw, uint32_t log_len, const uint32_t* beta,
                                                       TwiddleTables tw, uint32_t* out, const uint32_t* inject,
                                                       uint32_t* leaves) {
  const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (k >= (1ull << (log_len - 2))) return;
  const Ext4 hb = half_beta<F>(beta);
  uint32_t s[16];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const uint64_t r = 2 * k + u;
    Ext4 res = fri_fold_row<F>(cw, log_len, r, hb, tw, r);
    if (inject) {
      const uint4 v = reinterpret_cast<const uint4*>(inject)[r];
      res = Ef<F>::add(res, Ext4{{v.x, v.y, v.z, v.w}});
    }
    reinterpret_cast<uint4*>(out)[r] = make_uint4(res.c[0], res.c[1], res.c[2], res.c[3]);
#pragma unroll
    for (int i = 0; i < 4; i++) s[4 * u + i] = res.c[i];
  }
#pragma unroll
  for (int i = 8; i < 16; i++) s[i] = 0;
  p2_permute<F>(s);
  uint4* lp = reinterpret_cast<uint4*>(leaves + 8 * k);
  lp[0] = make_uint4(s[0], s[1], s[2], s[3]);
  lp[1] = make_uint4(s[4], s[5], s[6], s[7]);
}

// One shard's part of k_fri_fold_hash for a codeword split by rows: the
// shard holds rows [2 row0, 2 row0 + 4 n_leaves) of the 2^log_len-row
// codeword at cw; it folds them into rows [row0, row0 + 2 n_leaves) (stored
// from out) and hashes their n_leaves leaves.
template <class F>
__global__ void __launch_bounds__(256) k_fri_fold_hash_rows(const uint32_t* cw, uint32_t log_len, uint64_t row0,
                                                            uint64_t n_leaves, const uint32_t* beta,
                                                            TwiddleTables tw, uint32_t* out, uint32_t* leaves) {
  const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (k >= n_leaves) return;
  const Ext4 hb = half_beta<F>(beta);
  uint32_t s[16];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const uint64_t r = 2 * k + u;
    const Ext4 res = fri_fold_row<F>(cw, log_len, r, hb, tw, row0 + r);
    reinterpret_cast<uint4*>(out)[r] = make_uint4(res.c[0], res.c[1], res.c[2], res.c[3]);
#pragma unroll
    for (int i = 0; i < 4; i++) s[4 * u + i] = res.c[i];
  }
#pragma unroll
  for (int i = 8; i < 16; i++) s[i] = 0;
  p2_permute<F>(s);
  uint4* lp = reinterpret_cast<uint4*>(leaves + 8 * k);
  lp[0] = make_uint4(s[0], s[1], s[2], s[3]);
  lp[1] = make_uint4(s[4], s[5], s[6], s[7]);
}

// The same with 16 lanes per leaf (p2_lane.cuh): lane q < 8 folds the row of
// the leaf's word q (every lane of a row computes the whole element).
template <class F>
__global__ void __launch_bounds__(kLaneThreads)
    k_fri_fold_hash_lane(const uint32_t* cw, uint32_t log_len, uint64_t row0, uint64_t n_leaves, const uint32_t* beta,
                         const __grid_constant__ TwiddleTables tw, uint32_t* out, const uint32_t* inject,
                         uint32_t* leaves) {
  __shared__ __align__(16) uint32_t tab[kLaneWords];
  lane_load_tables<F>(tab);
  const uint64_t t = blockIdx.x * (uint64_t)kLaneThreads + threadIdx.x;
  const uint64_t k = t >> 4;
  const uint32_t q = (uint32_t)(t & 15);
  const bool live = k < n_leaves;
  uint32_t v = 0;
  if (live && q < 8) {
    const uint64_t r = 2 * k + (q >> 2);
    const Ext4 res = fri_fold_row<F>(cw, log_len, r, half_beta<F>(beta), tw, row0 + r);
    v = (q & 2) ? ((q & 1) ? res.c[3] : res.c[2]) : ((q & 1) ? res.c[1] : res.c[0]);
    if (inject) v = Fp<F>::add(v, inject[4 * r + (q & 3)]);
    out[4 * r + (q & 3)] = v;
  }
  __syncthreads();
  v = lane_permute<F>(v, q, tab);
  if (live && q < 8) leaves[8 * k + q] = v;
}

// k_fri_fold_hash and k_fri_fold_hash_rows with the leaves hashed on the
// tensor cores (p2_tc.cuh).
template <class F>
__global__ void __launch_bounds__(kTcThreads * kTcGroups, kTcCtas)
    k_fri_fold_hash_tc(const uint32_t* cw, uint32_t log_len, uint64_t row0, uint64_t n_leaves, const uint32_t* beta,
                       const __grid_constant__ TwiddleTables tw, uint32_t* out, const uint32_t* inject,
                       uint32_t* leaves) {
  PICO_TC_OPEN(F);
  for (uint64_t t0 = tc.first_tile(tc_tiles(n_leaves)) * kTcThreads; t0 < n_leaves; t0 += tc.tile_stride() * kTcThreads) {
    const uint64_t k = t0 + threadIdx.x % kTcThreads;
    uint32_t s[8];
    if (k < n_leaves) {
      const Ext4 hb = half_beta<F>(beta);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint64_t r = 2 * k + u;
        Ext4 res = fri_fold_row<F>(cw, log_len, r, hb, tw, row0 + r);
        if (inject) {
          const uint4 v = reinterpret_cast<const uint4*>(inject)[r];
          res = Ef<F>::add(res, Ext4{{v.x, v.y, v.z, v.w}});
        }
        reinterpret_cast<uint4*>(out)[r] = make_uint4(res.c[0], res.c[1], res.c[2], res.c[3]);
#pragma unroll
        for (int i = 0; i < 4; i++) s[4 * u + i] = res.c[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) s[i] = 0;
    }
    tc.put_rate(s);
    tc.body(kTcFromRate);
    tc.digest(s);
    if (k < n_leaves) store_digest(leaves + 8 * k, s);
  }
  PICO_TC_CLOSE();
}

static cudaError_t launch_fri_fold_hash_lane(int field, const uint32_t* cw, uint32_t log_len, uint64_t row0, uint64_t n,
                                             const uint32_t* beta, TwiddleTables tw, uint32_t* out,
                                             const uint32_t* inject, uint32_t* leaves, cudaStream_t st) {
  return launch_chained(true, field == 0 ? k_fri_fold_hash_lane<KoalaBear> : k_fri_fold_hash_lane<BabyBear>,
                        blocks_for(16 * n, kLaneThreads), kLaneThreads, 0, st, cw, log_len, row0, n, beta, tw, out, inject,
                        leaves);
}

cudaError_t launch_fri_fold_hash_rows(int field, const uint32_t* cw, uint32_t log_len, uint64_t row0,
                                      uint64_t n_leaves, const uint32_t* beta, TwiddleTables tw, uint32_t* out,
                                      uint32_t* leaves, cudaStream_t st) {
  if (n_leaves == 0) return cudaSuccess;
  if (log_len < 2 || 2 * (row0 + 2 * n_leaves) > (1ull << log_len)) return cudaErrorInvalidValue;
  if (n_leaves >= kTcMinStates)
    return tc_launch(true, field == 0 ? k_fri_fold_hash_tc<KoalaBear> : k_fri_fold_hash_tc<BabyBear>, tc_tiles(n_leaves), false,
                     st, cw, log_len, row0, n_leaves, beta, tw, out, (const uint32_t*)nullptr, leaves);
  if (n_leaves <= kLaneMaxStates)
    return launch_fri_fold_hash_lane(field, cw, log_len, row0, n_leaves, beta, tw, out, nullptr, leaves, st);
  if (field == 0)
    k_fri_fold_hash_rows<KoalaBear><<<blocks_for(n_leaves, 256), 256, 0, st>>>(cw, log_len, row0, n_leaves, beta,
                                                                               tw, out, leaves);
  else
    k_fri_fold_hash_rows<BabyBear><<<blocks_for(n_leaves, 256), 256, 0, st>>>(cw, log_len, row0, n_leaves, beta,
                                                                              tw, out, leaves);
  return cudaGetLastError();
}

cudaError_t launch_fri_fold_hash(int field, const uint32_t* cw, uint32_t log_len, const uint32_t* beta,
                                 TwiddleTables tw, uint32_t* out, const uint32_t* inject, uint32_t* leaves,
                                 cudaStream_t st) {
  if (log_len < 2) return cudaErrorInvalidValue;
  const uint64_t n = 1ull << (log_len - 2);
  if (n >= kTcMinStates)
    return tc_launch(true, field == 0 ? k_fri_fold_hash_tc<KoalaBear> : k_fri_fold_hash_tc<BabyBear>, tc_tiles(n), false, st, cw,
                     log_len, (uint64_t)0, n, beta, tw, out, inject, leaves);
  if (n <= kLaneMaxStates)
    return launch_fri_fold_hash_lane(field, cw, log_len, 0, n, beta, tw, out, inject, leaves, st);
  if (field == 0)
    k_fri_fold_hash<KoalaBear><<<blocks_for(n, 256), 256, 0, st>>>(cw, log_len, beta, tw, out, inject, leaves);
  else
    k_fri_fold_hash<BabyBear><<<blocks_for(n, 256), 256, 0, st>>>(cw, log_len, beta, tw, out, inject, leaves);
  return cudaGetLastError();
}

cudaError_t launch_fri_fold_tw(int field, const uint32_t* cw, uint32_t log_len, const uint32_t* beta,
                               TwiddleTables tw, uint32_t* out, cudaStream_t st, const uint32_t* inject) {
  uint64_t h = 1ull << (log_len - 1);
  if (field == 0)
    k_fri_fold<KoalaBear><<<blocks_for(h, 256), 256, 0, st>>>(cw, log_len, beta, tw, out, inject);
  else
    k_fri_fold<BabyBear><<<blocks_for(h, 256), 256, 0, st>>>(cw, log_len, beta, tw, out, inject);
  return cudaGetLastError();
}

cudaError_t launch_subtree(int field, uint32_t* level, uint32_t n_in, uint32_t n, const SubtreeInj& inj,
                           cudaStream_t st, DevChallenger* ch, uint32_t* beta_out, bool chained) {
  if (n == 0 || n > kSubtreeMaxIn || (n & (n - 1)) || n_in % n || (ch && n != n_in)) return cudaErrorInvalidValue;
  return launch_chained(chained, field == 0 ? k_subtree_lane<KoalaBear> : k_subtree_lane<BabyBear>, n_in / n, kSubtreeThreads, 0, st,
                        level, n_in, n, inj, ch, beta_out);
}

cudaError_t launch_challenger_observe(int field, DevChallenger* ch, const uint32_t* vals, uint32_t n,
                                      cudaStream_t st) {
  return launch_chained(true, field == 0 ? k_challenger_observe<KoalaBear> : k_challenger_observe<BabyBear>, 1, 32, 0, st, ch, vals,
                        n);
}

// Proof-of-work search (the challenger's grind; checked by check_witness,
// challenger.rs:210-221).  Observing candidate c and sampling always permutes
// once: the state with its pending inputs and c written over lanes
// 0..in_len, and the sample is lane 7 of the result (the last output popped).
// A candidate passes when the sample's canonical value has `bits` low zero
// bits; the smallest passing candidate of the launch wins (atomicMin).
template <class F>
__global__ void __launch_bounds__(256) k_grind(const DevChallenger* ch, uint32_t bits, uint32_t base,
                                               uint32_t count, uint32_t* best) {
  using B = Fp<F>;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (*reinterpret_cast<volatile uint32_t*>(best) != 0xffffffffu) return;  // found by an earlier launch
  if (k >= count) return;
  const uint64_t c = (uint64_t)base + k;
  if (c >= F::P) return;
  uint32_t s[16];
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = ch->sponge[i];
  const uint32_t n_in = ch->in_len;  // below 8: a full buffer is absorbed when it fills
  for (uint32_t i = 0; i < n_in && i < 8; i++) s[i] = ch->in_buf[i];
  const uint32_t v = B::to_monty((uint32_t)c);
#pragma unroll
  for (int i = 0; i < 8; i++)
    if ((uint32_t)i == n_in) s[i] = v;
  p2_permute<F>(s);
  const uint32_t mask = bits >= 32 ? 0xffffffffu : ((1u << bits) - 1u);
  if ((B::from_monty(s[7]) & mask) == 0) atomicMin(best, (uint32_t)c);
}

cudaError_t launch_grind(int field, const DevChallenger* ch, uint32_t bits, uint32_t base, uint32_t count,
                         uint32_t* best, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const unsigned blocks = (count + 255) / 256;
  if (field == 0)
    k_grind<KoalaBear><<<blocks, 256, 0, st>>>(ch, bits, base, count, best);
  else
    k_grind<BabyBear><<<blocks, 256, 0, st>>>(ch, bits, base, count, best);
  return cudaGetLastError();
}

}  // namespace pico

namespace pico {

// Final polynomial of the commit phase when folding stops early: the
// remaining codeword holds 2^log_len evaluations in bit-reversed order; its
// coefficients over the subgroup are c_i = (1/len) sum_j v[rev(j)] w^(-ij).
// Coefficients at i >= 2^log_keep must vanish (low-degree check): a nonzero
// one sets *err.
template <class F>
__global__ void k_fri_final_poly(const uint32_t* cw, uint32_t log_len, uint32_t log_keep, TwiddleTables tw,
                                 uint32_t* coeffs, uint32_t* err) {
  using B = Fp<F>;
  const uint32_t len = 1u << log_len;
  const uint32_t mask = (1u << F::TWO_ADICITY) - 1u;
  const uint32_t len_inv = B::inv(B::to_monty(len));
  for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
    uint32_t acc[4] = {0, 0, 0, 0};
    for (uint32_t j = 0; j < len; j++) {
      uint32_t e = (uint32_t)(((uint64_t)i * j) & (len - 1)) << (F::TWO_ADICITY - log_len);
      e = (0u - e) & mask;
      const uint32_t wv = B::mul(__ldg(tw.hi + (e >> 14)), __ldg(tw.lo + (e & 0x3fffu)));
      const uint32_t* v = cw + 4 * bitrev32(j, log_len);
#pragma unroll
      for (int k = 0; k < 4; k++) acc[k] = B::add(acc[k], B::mul(v[k], wv));
    }
#pragma unroll
    for (int k = 0; k < 4; k++) acc[k] = B::mul(acc[k], len_inv);
    if (i < (1u << log_keep)) {
#pragma unroll
      for (int k = 0; k < 4; k++) coeffs[4 * i + k] = acc[k];
    } else if (acc[0] | acc[1] | acc[2] | acc[3]) {
      atomicExch(err, 1u);
    }
  }
}

cudaError_t launch_fri_final_poly(int field, const uint32_t* cw, uint32_t log_len, uint32_t log_keep,
                                  TwiddleTables tw, uint32_t* coeffs, uint32_t* err, cudaStream_t st) {
  if (field == 0)
    k_fri_final_poly<KoalaBear><<<1, 256, 0, st>>>(cw, log_len, log_keep, tw, coeffs, err);
  else
    k_fri_final_poly<BabyBear><<<1, 256, 0, st>>>(cw, log_len, log_keep, tw, coeffs, err);
  return cudaGetLastError();
}

}  // namespace pico
