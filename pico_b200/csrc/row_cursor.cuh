// Walking a row across the matrices of its group, eight columns at a time
// (tensor-core row hashing), for host and device.
#pragma once
#include <cstdint>

#include "field.cuh"

namespace pico {

// One matrix segment of a concatenated Merkle row: `rows` x `width`,
// row-major, rows at ptr + r * width.
struct RowSeg {
  const uint32_t* ptr;
  uint32_t width;
  uint32_t pad;
};

struct RowCursor {
  uint32_t seg, col, segw;
  const uint32_t* rowp;
};
PICO_HD void row_cursor_begin(RowCursor& c, const RowSeg* segs, uint32_t n_segs, uint64_t r) {
  c.seg = c.col = 0;
  c.segw = n_segs ? segs[0].width : 0u;
  c.rowp = n_segs ? segs[0].ptr + r * c.segw : nullptr;
}
PICO_HD uint32_t row_word(const uint32_t* p) {
#if defined(__CUDA_ARCH__)
  return __ldg(p);
#else
  return *p;
#endif
}
// The next columns of row r: words of chunk positions [lo, hi) into v, through
// the cursor.  A column past the last segment (where segw is 0, so that no chunk
// fits) is not read: it counts as zero and trip(seg, col)
// records it.
template <class Trip>
PICO_HD void row_chunk(RowCursor& c, const RowSeg* segs, uint32_t n_segs, uint64_t r, int lo, int hi, uint32_t v[8],
                       Trip trip) {
  if (lo == 0 && hi == 8 && c.col + 8 <= c.segw) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int j = 0; j < 8; j++) v[j] = row_word(c.rowp + c.col + j);
    c.col += 8;
    return;
  }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int j = 0; j < 8; j++) {
    if (j >= lo && j < hi) {
      while (c.col == c.segw && c.seg < n_segs) {
        c.seg++;
        c.col = 0;
        c.segw = c.seg < n_segs ? segs[c.seg].width : 0u;
        c.rowp = c.seg < n_segs ? segs[c.seg].ptr + r * c.segw : nullptr;
      }
      if (c.seg >= n_segs) {
        trip(c.seg, c.col);
        v[j] = 0;
      } else {
        v[j] = row_word(c.rowp + c.col);
      }
      c.col++;
    }
  }
}

}  // namespace pico
