// Closure lists and vertex records of the bit-row kernels (closure.hpp).
#include "closure.hpp"

#include <algorithm>
#include <atomic>
#include <exception>
#include <vector>

namespace chsga {

namespace {

constexpr int64_t kMaxWeight = 1 << 30;  // sums stay below int32 with any score

// An entry as one number (source vertex above, weight below), so that lists
// sort by source, then weight.
using Entry = uint64_t;
using List = std::vector<Entry>;

Entry entry(uint32_t src, int32_t w) { return (Entry)src << 32 | (uint32_t)w; }
uint32_t src_of(Entry e) { return (uint32_t)(e >> 32); }
int32_t w_of(Entry e) { return (int32_t)(uint32_t)e; }
Entry heavier(Entry e, int32_t by) {
  return entry(src_of(e), (int32_t)std::min<int64_t>((int64_t)w_of(e) + by, kMaxWeight));
}

// Lists by index, many to an allocation.
struct Lists {
  std::vector<const Entry*> first{nullptr};  // list 0 is empty
  std::vector<uint32_t> n{0};
  std::vector<List> store;
};

// One entry per source, the smallest weight; `self` (a one-char vertex's own
// score, which a positive weight cannot lower) is dropped.
void tidy(List& l, int64_t self) {
  std::sort(l.begin(), l.end());
  size_t k = 0;
  for (const Entry e : l) {
    if (src_of(e) == self || (k && src_of(l[k - 1]) == src_of(e))) continue;
    l[k++] = e;
  }
  l.resize(k);
}

// out = the union of two tidy lists, b's weights raised by `by`.
void merge(const List& a, const Entry* b, const Entry* b_end, int32_t by, List& out) {
  out.clear();
  auto i = a.begin();
  while (i != a.end() || b != b_end) {
    if (b == b_end || (i != a.end() && src_of(*i) < src_of(*b))) {
      out.push_back(*i++);
    } else if (i == a.end() || src_of(*b) < src_of(*i)) {
      out.push_back(heavier(*b++, by));
    } else {
      out.push_back(std::min(*i++, heavier(*b, by)));
      ++b;
    }
  }
}

// f(i) for i in [0, n), on all threads when there are many; what one of them
// throws is thrown here when all are done.
template <typename F>
void parallel(int64_t n, bool many, F&& f) {
  std::exception_ptr err;
  std::atomic<bool> failed{false};
#pragma omp parallel for schedule(dynamic) if (many)
  for (int64_t i = 0; i < n; ++i) {
    if (failed.load(std::memory_order_relaxed)) continue;
    try {
      f(i);
    } catch (...) {
      if (!failed.exchange(true)) err = std::current_exception();
    }
  }
  if (err) std::rethrow_exception(err);
}

}  // namespace

HostClosure build_closure(const HostLayout& L) {
  HostClosure c;
  const uint32_t S = L.S;
  const bool many = S > 2048;
  std::atomic<bool> refused{false};
  auto single = [&](uint32_t d) { return L.dv_len[d] == 1; };
  // expanded lists of one-char vertices that are sources, by hierarchy
  // position: after the upward sweep (what upward edges read) and final
  // (what downward edges read). An even source index of an edge names the
  // only score of a one-char vertex.
  std::vector<uint8_t> up_src(S, 0), dn_src(S, 0);
  auto mark = [&](const std::vector<EdgeW>& in, std::vector<uint8_t>& src) {
#pragma omp parallel for schedule(static) if (many)
    for (int64_t k = 0; k < (int64_t)in.size(); ++k)
      if (!(in[k].src & 1) && single(in[k].src >> 1)) __atomic_store_n(&src[in[k].src >> 1], 1, __ATOMIC_RELAXED);
  };
  mark(L.up_in, up_src);
  mark(L.dn_in, dn_src);
  std::vector<uint32_t> slot(S, 0);
  Lists ups, fins;
  auto self_of = [&](uint32_t d) { return single(d) ? (int64_t)L.dv_s[d] : -1; };
  // the source of an edge and, through a one-char source, that one's sources
  auto take = [&](uint32_t d, const EdgeW& e, bool through, const Lists& lists, const std::vector<uint32_t>& at,
                  List& l) {
    const uint32_t x = (uint32_t)e.src >> 1;
    l.push_back(entry(L.dv_s[x], e.w));
    if (!through) return;
    const Entry* y = lists.first[at[x]];
    for (uint32_t k = 0; k < lists.n[at[x]]; ++k) l.push_back(heavier(y[k], e.w));
    if (l.size() > kClosureTidy) {
      tidy(l, self_of(d));
      if (l.size() > kClosureMaxList) refused = true;
    }
  };
  auto expand_up = [&](uint32_t d, List& l) {
    for (uint32_t k = L.up_off[d]; k < L.up_off[d + 1] && !refused; ++k) {
      const uint32_t x = (uint32_t)L.up_in[k].src >> 1;
      take(d, L.up_in[k], single(x) && L.up_off[x + 1] > L.up_off[x], ups, slot, l);
    }
  };
  auto finish = [&](uint32_t d, List& l) {
    tidy(l, self_of(d));
    if (l.size() > kClosureMaxList) refused = true;
  };
  // the one-char vertices of a level that `want` picks, in pieces of 64
  auto by_level = [&](uint32_t level, Lists& lists, std::vector<uint32_t>& at, auto&& want, auto&& make) {
    const size_t first = lists.n.size(), piece = lists.store.size();
    std::vector<uint32_t> todo;
    for (uint32_t d = L.lvl_off[level]; d < L.lvl_off[level + 1]; ++d)
      if (want(d)) {
        at[d] = (uint32_t)(first + todo.size());
        todo.push_back(d);
      }
    const size_t pieces = (todo.size() + 63) / 64;
    lists.first.resize(first + todo.size());
    lists.n.resize(first + todo.size());
    lists.store.resize(piece + pieces);
    parallel((int64_t)pieces, todo.size() > 256, [&](int64_t q) {
      const size_t lo = 64 * (size_t)q, hi = std::min(todo.size(), lo + 64);
      List l, out;
      uint32_t n[64];
      for (size_t i = lo; i < hi && !refused; ++i) {
        l.clear();
        make(todo[i], l);
        finish(todo[i], l);
        n[i - lo] = (uint32_t)l.size();
        out.insert(out.end(), l.begin(), l.end());
      }
      if (refused) return;
      const Entry* p = out.data();
      for (size_t i = lo; i < hi; p += n[i - lo], ++i) {
        lists.first[first + i] = p;
        lists.n[first + i] = n[i - lo];
      }
      lists.store[piece + q] = std::move(out);  // its entries stay where they are
    });
  };
  // one-char vertices with upward in-edges, by rising level
  for (uint32_t l = 0; l < L.levels && !refused; ++l)
    by_level(l, ups, slot,
             [&](uint32_t d) { return single(d) && (up_src[d] || dn_src[d]) && L.up_off[d + 1] > L.up_off[d]; },
             expand_up);
  if (refused) return HostClosure{};
  // final lists of one-char sources of downward edges, by falling level
  std::vector<uint32_t> fslot(S, 0);
  auto expand_final = [&](uint32_t d, List& l) {
    expand_up(d, l);
    for (uint32_t k = L.dn_off[d]; k < L.dn_off[d + 1] && !refused; ++k)
      take(d, L.dn_in[k], single((uint32_t)L.dn_in[k].src >> 1), fins, fslot, l);
  };
  for (uint32_t l = L.levels; l-- > 0 && !refused;)
    by_level(l, fins, fslot, [&](uint32_t d) { return dn_src[d] != 0; }, expand_final);
  if (refused) return HostClosure{};
  // A(v) of every vertex, in chunks of string vertices
  // log2 of a chunk: some hundred chunks, whose lists stay below the size at
  // which the allocator maps and unmaps memory for each
  uint32_t shift = 6;
  while (shift < 10 && (S >> shift) > 256) ++shift;
  const int64_t chunks = ((int64_t)S + (1 << shift) - 1) >> shift;
  auto chunk_end = [&](int64_t q) { return (uint32_t)std::min<int64_t>(S, (q + 1) << shift); };
  RawArray<uint32_t> a_off, a_n;
  a_off.alloc(S);
  a_n.alloc(S);
  std::vector<List> a_chunk(chunks);
  std::atomic<uint64_t> total{0};
  const uint64_t limit = (uint64_t)kClosureMaxGrowth * (L.up_in.size() + L.dn_in.size()) + 1024;
  auto grow = [&](uint64_t n, uint64_t most) {
    const uint64_t now = total.fetch_add(n, std::memory_order_relaxed) + n;
    if (now > most || now > (1u << 30)) refused = true;
  };
  parallel(chunks, many, [&](int64_t q) {
    List l, out;  // local: neighbouring chunks' lists share cache lines
    out.reserve((size_t)4 << shift);
    for (uint32_t s = (uint32_t)(q << shift); s < chunk_end(q) && !refused; ++s) {
      l.clear();
      expand_final(L.sv_dev[s], l);
      finish(L.sv_dev[s], l);
      a_off[s] = (uint32_t)out.size();
      a_n[s] = (uint32_t)l.size();
      out.insert(out.end(), l.begin(), l.end());
    }
    grow(out.size(), limit);
    a_chunk[q] = std::move(out);
  });
  if (refused) return HostClosure{};
  auto a_list = [&](uint32_t s) { return a_chunk[s >> shift].data() + a_off[s]; };
  // merged entries: both, M only, F only
  auto key = [&](uint32_t ch) { return (L.lab4[ch >> 3] >> ((ch & 7) * 4)) & 0xFu; };
  auto len_of = [&](uint32_t s) { return L.sv_off[s + 1] - L.sv_off[s]; };
  c.rec.alloc((size_t)4 * S);
  std::vector<std::vector<EdgeW>> e_chunk(chunks);
  std::vector<uint32_t> h_chunk(chunks + 1, 0);  // long lists
  total = 0;
  parallel(chunks, many, [&](int64_t q) {
    List b, t, cls[3];
    std::vector<EdgeW> out;
    uint32_t heavy = 0;
    out.reserve((size_t)6 << shift);
    for (uint32_t s = (uint32_t)(q << shift); s < chunk_end(q) && !refused; ++s) {
      b.clear();
      for (List& l : cls) l.clear();
      for (uint32_t k = L.vin_off[s]; k < L.vin_off[s + 1]; ++k) {
        const uint32_t u = L.vin_srcv[k];
        merge(b, a_list(u), a_list(u) + a_n[u], (int32_t)(len_of(u) - 1), t);
        const Entry last = entry(u, 0);
        merge(t, &last, &last + 1, 0, b);
        // more than the three classes and the dropped ones can hold
        if (b.size() > kClosureTidy) refused = true;
        if (refused) return;
      }
      const Entry *a = a_list(s), *const a_end = a + a_n[s];
      for (const Entry e : b) {
        for (; a != a_end && src_of(*a) < src_of(e); ++a) cls[2].push_back(*a);
        if (a != a_end && src_of(*a) == src_of(e)) {
          if (w_of(e) == w_of(*a) - 1) {
            cls[0].push_back(e);
          } else {
            if (w_of(e) <= w_of(*a)) cls[1].push_back(e);
            cls[2].push_back(*a);
          }
          ++a;
        } else {
          cls[1].push_back(e);
        }
      }
      cls[2].insert(cls[2].end(), a, a_end);
      if (std::max({cls[0].size(), cls[1].size(), cls[2].size()}) > 255) refused = true;
      const uint32_t at = (uint32_t)out.size();
      // light entries first: the sources that win are near
      for (List& l : cls) {
        for (Entry& e : l) e = e << 32 | e >> 32;
        std::sort(l.begin(), l.end());
        for (const Entry e : l) out.push_back(EdgeW{(int32_t)(uint32_t)e, (int32_t)(e >> 32)});
      }
      uint32_t* r = &c.rec[4 * (size_t)s];
      r[0] = L.sv_off[s];
      r[1] = len_of(s) | key(L.sv_off[s]) << 29;
      r[2] = at;
      r[3] = (uint32_t)(cls[0].size() | cls[1].size() << 8 | cls[2].size() << 16);
      heavy += out.size() - at > kWordLight;
    }
    grow(out.size(), 3 * limit);
    e_chunk[q] = std::move(out);
    h_chunk[q + 1] = heavy;
  });
  if (refused) return HostClosure{};
  std::vector<uint32_t> e_base(chunks + 1, 0);
  for (int64_t q = 0; q < chunks; ++q) {
    e_base[q + 1] = e_base[q] + (uint32_t)e_chunk[q].size();
    h_chunk[q + 1] += h_chunk[q];
  }
  c.heavy = h_chunk[chunks];
  c.ent.alloc(e_base[chunks]);
  RawArray<uint32_t> at;
  at.alloc(S);
  auto count = [&](uint32_t s) {
    const uint32_t n = c.rec[4 * (size_t)s + 3];
    return (n & 255) + ((n >> 8) & 255) + (n >> 16);
  };
  parallel(chunks, many, [&](int64_t q) {
    std::copy(e_chunk[q].begin(), e_chunk[q].end(), c.ent.data() + e_base[q]);
    const uint32_t s0 = (uint32_t)(q << shift);
    uint32_t h = h_chunk[q], l = c.heavy + s0 - h;
    for (uint32_t s = s0; s < chunk_end(q); ++s) {
      c.rec[4 * (size_t)s + 2] += e_base[q];
      at[count(s) > kWordLight ? h++ : l++] = s;
    }
  });
  // the word kernel's order: segments of up to kWordWindow positions, those of
  // the long lists first
  const int64_t hs = ((int64_t)c.heavy + kWordWindow - 1) / kWordWindow,
                segs = hs + ((int64_t)S - c.heavy + kWordWindow - 1) / kWordWindow;
  auto seg = [&](int64_t q) {
    const int64_t lo = q < hs ? q * kWordWindow : c.heavy + (q - hs) * kWordWindow,
                  end = q < hs ? c.heavy : S;
    return std::pair<uint32_t, uint32_t>((uint32_t)lo, (uint32_t)std::min<int64_t>(end, lo + kWordWindow));
  };
  std::vector<uint64_t> w_base(segs + 1, 0), n_base(segs + 1, 0);
  parallel(segs, many, [&](int64_t q) {
    const auto [lo, hi] = seg(q);
    if (q >= hs) {
      // by list length, then vertices without chain chars together, else in
      // their order: a counting sort
      uint32_t first[2 * kWordLight + 3] = {}, s_of[kWordWindow];
      auto rank = [&](uint32_t s) { return 2 * (kWordLight - count(s)) + (len_of(s) > 1 ? 0 : 1); };
      for (uint32_t i = lo; i < hi; ++i) ++first[rank(at[i]) + 1];
      for (uint32_t r = 1; r < 2 * kWordLight + 2; ++r) first[r + 1] += first[r];
      for (uint32_t i = lo; i < hi; ++i) s_of[first[rank(at[i])]++] = at[i];
      std::copy(s_of, s_of + (hi - lo), at.data() + lo);
    }
    uint64_t w = 0, n = 0;
    for (uint32_t i = lo; i < hi; ++i) {
      w += (len_of(at[i]) - 1 + 31) / 32;
      // a group of short lists is as wide as its longest, which is its first
      if (q < hs || (i - lo) % 32 == 0) n += (q < hs ? 1 : 32) * count(at[i]);
    }
    w_base[q + 1] = w;
    n_base[q + 1] = n;
  });
  for (int64_t q = 0; q < segs; ++q) {
    w_base[q + 1] += w_base[q];
    n_base[q + 1] += n_base[q];
  }
  if (w_base[segs] >= (1ull << 31) || n_base[segs] >= (1ull << 31)) return HostClosure{};
  c.words = w_base[segs];
  c.n_went = n_base[segs];
  c.order.alloc((size_t)4 * S);
  parallel(segs, many, [&](int64_t q) {
    const auto [lo, hi] = seg(q);
    uint64_t w = w_base[q], n = n_base[q], wide = 0;
    for (uint32_t i = lo; i < hi; ++i) {
      const uint32_t k = (i - lo) % 32;
      if (q >= hs && k == 0) {
        n += wide;
        wide = 32ull * count(at[i]);
      }
      uint32_t* r = &c.order[4 * (size_t)i];
      r[0] = (uint32_t)w;
      r[1] = at[i];
      r[2] = (uint32_t)(q < hs ? n : n + k);
      r[3] = 0;
      w += (len_of(at[i]) - 1 + 31) / 32;
      if (q < hs) n += count(at[i]);
    }
  });
  c.ok = true;
  return c;
}

}  // namespace chsga
