// Word operations of the bit-row kernels (bit_rows.cuh), for host and device.
//
// Inside a string vertex neighbouring chars' scores differ by -1, 0 or 1 in
// every row, so a row is the first score of each vertex and two bits per
// chain char: P (one above the char before) and N (one below). The chain
// update
//     T[c] = min(D[c] + 1, D[c-1] + delta, T[c-1] + 1)
// over the differences is Myers' bit-vector step (J. ACM 46(3), 1999) with
// the block boundary of Hyyro (Nordic J. Computing 10, 2003): 32 chars of
// one read a word, the change of the first char's score carried in.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define CHSGA_HD __host__ __device__ __forceinline__
#else
#define CHSGA_HD inline
#endif

namespace chsga {
namespace bits {

struct PN {
  uint32_t p, n;
};

// Chars of a word whose label scores a substitution against the read base;
// mask bit k = label key k (0..3 A,C,G,T, 4 the special byte) mismatches.
CHSGA_HD uint32_t mismatch_word(uint32_t b0, uint32_t b1, uint32_t sp, uint32_t mask) {
  const uint32_t m0 = 0u - (mask & 1u), m1 = 0u - ((mask >> 1) & 1u), m2 = 0u - ((mask >> 2) & 1u),
                 m3 = 0u - ((mask >> 3) & 1u), m4 = 0u - ((mask >> 4) & 1u);
  const uint32_t lo = (m0 & ~b0) | (m1 & b0), hi = (m2 & ~b0) | (m3 & b0);
  return ((((lo & ~b1) | (hi & b1)) & ~sp) | (m4 & sp));
}

// Lowers a word of differences under the line that starts g below the
// word's left neighbour and climbs by 1 a char: the row becomes
// min(row, line). `valid` = the word's chars. g is what is left of the gap
// at the word's end. A char whose difference is +1 keeps the gap, 0 closes
// it by one, -1 by two (to -1 at most: then the lowered row meets the row
// one char early and the difference is 0).
CHSGA_HD PN under_line(PN w, uint32_t valid, uint32_t& g) {
  uint32_t z = ~w.p & valid;
  while (g && z) {
    const uint32_t bit = z & (0u - z);
    z ^= bit;
    if (w.n & bit) {
      w.n &= ~bit;
      if (g == 1) {
        g = 0;
      } else {
        w.p |= bit;
        g -= 2;
      }
    } else {
      w.p |= bit;
      --g;
    }
  }
  return w;
}

// One row update of a word: differences of the previous row, d = mismatching
// chars, h = the change of the score left of the word (-1, 0, 1). Returns
// the new differences; h becomes the change of the score of char `top`.
CHSGA_HD PN step(PN w, uint32_t d, int& h, uint32_t top) {
  const uint32_t eq0 = ~d;
  const uint32_t xv = eq0 | w.n;
  const uint32_t eq = eq0 | (h < 0 ? 1u : 0u);
  const uint32_t xh = (((eq & w.p) + w.p) ^ w.p) | eq;
  uint32_t ph = w.n | ~(xh | w.p);
  uint32_t mh = w.p & xh;
  const uint32_t pin = h > 0 ? 1u : 0u, nin = h < 0 ? 1u : 0u;
  h = (int)((ph >> top) & 1u) - (int)((mh >> top) & 1u);
  ph = (ph << 1) | pin;
  mh = (mh << 1) | nin;
  return PN{mh | ~(xv | ph), ph & xv};
}

// Row 0: the differences of the mismatch bits themselves; `left` = the
// mismatch of the char left of the word, replaced by that of char `top`.
CHSGA_HD PN first_row(uint32_t d, uint32_t& left, uint32_t top) {
  const uint32_t before = (d << 1) | left;
  left = (d >> top) & 1u;
  return PN{d & ~before, before & ~d};
}

}  // namespace bits
}  // namespace chsga
