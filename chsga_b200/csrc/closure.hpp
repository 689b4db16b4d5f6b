// The hierarchy closure of a row as one independent minimum per string
// vertex, and the vertex records of the bit-row kernels (bit_rows.cuh).
//
// The sweeps of align.hpp:279-345 lower the first score of every string
// vertex over the hierarchy, level by level, and read the *last* score of
// each edge's source. They never refresh a last score from a lowered first
// score, so the source of an edge is a value the row update left -- a
// constant of the sweep -- unless the source is a one-char vertex, whose
// first and last score are one. Only one-char sources chain, and replacing
// such a source by its own sources (weights added) removes the chain: after
// expansion every swept first score is
//     F(v) = min(first(v), min over A(v) of raw_last(x) + w)
// over raw scores only, with no order between vertices. On the variation
// graphs measured (labels of 1..32 chars) the expansion adds 5-21 % to the
// hierarchy's edges, and the sweeps' 30-45 dependent levels become one pass.
//
// The row update takes a first char's in-edges from the final last scores,
//     M(v) = min over in-edges u of min(raw_last(u), F(u) + len(u) - 1),
// expanded the same way into a list B(v) of raw last scores (raw_last(u) is
// never above raw_first(u) + len(u) - 1, so F(u)'s own raw first drops out).
// T(first) = min(F + 1, M + delta), so an entry of B whose weight is above
// that of the same source in A can never win and is dropped; a source with
// w_B = w_A - 1 (the usual case: x reaches v through u) is read once for both.
//
// Graphs of one-char vertices chain without bound; there the lists would
// grow far beyond the edges, build_closure gives up (ok = false) and the
// engine sweeps the levels instead.
#pragma once

#include <cstddef>
#include <cstdint>
#include <memory>

#include "device_graph.hpp"

namespace chsga {

// Longest list a vertex may have, and entries per hierarchy edge above which
// the level sweeps are kept.
// A list is cut down to one entry a source whenever it is longer than
// kClosureTidy on the way, and the totals are watched while the lists grow, so
// a graph that is refused costs little time and no more memory than one that
// is not.
constexpr uint32_t kClosureMaxList = 192;
constexpr uint32_t kClosureMaxGrowth = 6;
constexpr uint32_t kClosureTidy = 1024;
constexpr uint32_t kWordWindow = 512, kWordLight = 8;

// An array that is not cleared first: it is filled by all threads, which then
// share its page faults too (a quarter of the build's time where one thread
// cleared it).
template <typename T>
class RawArray {
 public:
  void alloc(size_t n) {
    p_.reset(new T[n]);
    n_ = n;
  }
  T& operator[](size_t i) { return p_[i]; }
  const T& operator[](size_t i) const { return p_[i]; }
  T* data() { return p_.get(); }
  const T* data() const { return p_.get(); }
  size_t size() const { return n_; }

 private:
  std::unique_ptr<T[]> p_;
  size_t n_ = 0;
};

struct HostClosure {
  bool ok = false;
  // 4 words per string vertex: first char; length | label key of the first
  // char << 29; first entry; entries of each class (both | M only << 8 | F
  // only << 16)
  RawArray<uint32_t> rec;
  // {source vertex, weight}, classes in that order; the weight counts for M
  // (a "both" entry has weight w + 1 for F), for F-only entries for F
  RawArray<EdgeW> ent;

  // The one-read-a-word kernel works in an order of its own. Vertices with
  // more than kWordLight entries come first (several lanes share such a
  // list); the others follow, by list length inside every window of
  // kWordWindow vertices, so that the 32 vertices of a warp end together and
  // lie side by side in the arrays of that order (the scores stay by string
  // vertex, where neighbours are near).
  //   heavy     vertices of the first kind
  //   order     4 words per position: first bit word, string vertex, first of
  //             its n_went entries, 0. A long list is contiguous, entry k of a
  //             short one lies at first + 32 k (a group of 32 vertices side
  //             by side)
  //   words     bit words (32 chain chars each)
  // The arrays themselves are made on the device (k_closure_arrays).
  uint32_t heavy = 0;
  RawArray<uint32_t> order;
  uint64_t n_went = 0, words = 0;
};

// Throws std::bad_alloc like a vector would, whichever thread ran out.
HostClosure build_closure(const HostLayout& L);

}  // namespace chsga
