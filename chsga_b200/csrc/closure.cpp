// Closure lists and vertex records of the bit-row kernels (closure.hpp).
#include "closure.hpp"

#include <algorithm>
#include <atomic>
#include <numeric>

namespace chsga {

namespace {

constexpr int64_t kMaxWeight = 1 << 30;  // sums stay below int32 with any score

using List = std::vector<EdgeW>;  // {source vertex, weight}

// One entry per source, the smallest weight; `self` (a one-char vertex's own
// score, which a positive weight cannot lower) is dropped.
void tidy(List& l, int32_t self) {
  std::sort(l.begin(), l.end(), [](const EdgeW& a, const EdgeW& b) {
    return a.src != b.src ? a.src < b.src : a.w < b.w;
  });
  size_t k = 0;
  for (const EdgeW& e : l) {
    if (e.src == self || (k && l[k - 1].src == e.src)) continue;
    l[k++] = e;
  }
  l.resize(k);
}

int32_t add_w(int32_t a, int32_t b) { return (int32_t)std::min<int64_t>((int64_t)a + b, kMaxWeight); }

}  // namespace

HostClosure build_closure(const HostLayout& L) {
  HostClosure c;
  const uint32_t S = L.S;
  std::atomic<bool> too_long{false};
  // expanded lists of one-char vertices that are sources, by hierarchy
  // position: after the upward sweep (what upward edges read) and final
  // (what downward edges read)
  std::vector<uint8_t> up_src(S, 0), dn_src(S, 0);
  for (const EdgeW& e : L.up_in)
    if (!(e.src & 1)) up_src[e.src >> 1] = 1;
  for (const EdgeW& e : L.dn_in)
    if (!(e.src & 1)) dn_src[e.src >> 1] = 1;
  for (uint32_t d = 0; d < S; ++d)  // an even index names the only score of a one-char vertex
    if (L.dv_len[d] != 1) up_src[d] = dn_src[d] = 0;
  std::vector<uint32_t> slot(S, 0);
  std::vector<List> ups(1), fins(1);
  auto single = [&](uint32_t d) { return L.dv_len[d] == 1; };
  auto expand_up = [&](uint32_t d, List& l) {
    for (uint32_t k = L.up_off[d]; k < L.up_off[d + 1]; ++k) {
      const uint32_t x = (uint32_t)L.up_in[k].src >> 1;
      l.push_back({(int32_t)L.dv_s[x], L.up_in[k].w});
      if (single(x) && L.up_off[x + 1] > L.up_off[x])
        for (const EdgeW& e : ups[slot[x]]) l.push_back({e.src, add_w(e.w, L.up_in[k].w)});
    }
  };
  auto finish = [&](uint32_t d, List& l) {
    tidy(l, single(d) ? (int32_t)L.dv_s[d] : -1);
    if (l.size() > kClosureMaxList) too_long = true;
  };
  // one-char vertices with upward in-edges, by rising level
  for (uint32_t l = 0; l < L.levels && !too_long; ++l) {
    const uint32_t lo = L.lvl_off[l], hi = L.lvl_off[l + 1];
    const size_t first = ups.size();
    std::vector<uint32_t> todo;
    for (uint32_t d = lo; d < hi; ++d)
      if (single(d) && (up_src[d] || dn_src[d]) && L.up_off[d + 1] > L.up_off[d]) {
        slot[d] = (uint32_t)(first + todo.size());
        todo.push_back(d);
      }
    ups.resize(first + todo.size());
#pragma omp parallel for schedule(dynamic, 64) if (todo.size() > 256)
    for (int64_t i = 0; i < (int64_t)todo.size(); ++i) {
      if (too_long) continue;
      expand_up(todo[i], ups[first + i]);
      finish(todo[i], ups[first + i]);
    }
  }
  if (too_long) return HostClosure{};
  // final lists of one-char sources of downward edges, by falling level
  std::vector<uint32_t> fslot(S, 0);
  auto expand_final = [&](uint32_t d, List& l) {
    expand_up(d, l);
    for (uint32_t k = L.dn_off[d]; k < L.dn_off[d + 1]; ++k) {
      const uint32_t x = (uint32_t)L.dn_in[k].src >> 1;
      l.push_back({(int32_t)L.dv_s[x], L.dn_in[k].w});
      if (single(x))
        for (const EdgeW& e : fins[fslot[x]]) l.push_back({e.src, add_w(e.w, L.dn_in[k].w)});
    }
    finish(d, l);
  };
  for (uint32_t l = L.levels; l-- > 0 && !too_long;) {
    const size_t first = fins.size();
    std::vector<uint32_t> todo;
    for (uint32_t d = L.lvl_off[l]; d < L.lvl_off[l + 1]; ++d)
      if (dn_src[d]) {
        fslot[d] = (uint32_t)(first + todo.size());
        todo.push_back(d);
      }
    fins.resize(first + todo.size());
#pragma omp parallel for schedule(dynamic, 64) if (todo.size() > 256)
    for (int64_t i = 0; i < (int64_t)todo.size(); ++i)
      if (!too_long) expand_final(todo[i], fins[first + i]);
  }
  if (too_long) return HostClosure{};
  // A(v) of every vertex, by string vertex
  constexpr int64_t kChunk = 4096;
  const int64_t chunks = ((int64_t)S + kChunk - 1) / kChunk;
  std::vector<uint32_t> a_off((size_t)S + 1, 0);
  std::vector<List> a_chunk(chunks);
  uint64_t total = 0;
  const uint64_t limit = (uint64_t)kClosureMaxGrowth * (L.up_in.size() + L.dn_in.size()) + 1024;
#pragma omp parallel for schedule(dynamic) reduction(+ : total)
  for (int64_t q = 0; q < chunks; ++q) {
    List l;
    for (int64_t s = q * kChunk; s < std::min<int64_t>(S, (q + 1) * kChunk) && !too_long; ++s) {
      l.clear();
      expand_final(L.sv_dev[s], l);
      a_off[s + 1] = (uint32_t)l.size();
      a_chunk[q].insert(a_chunk[q].end(), l.begin(), l.end());
      total += l.size();
    }
  }
  if (too_long || total > limit || total > (1u << 30)) return HostClosure{};
  for (uint32_t s = 0; s < S; ++s) a_off[s + 1] += a_off[s];
  List a(total);
#pragma omp parallel for schedule(static)
  for (int64_t q = 0; q < chunks; ++q)
    std::copy(a_chunk[q].begin(), a_chunk[q].end(), a.begin() + a_off[q * kChunk]);
  a_chunk = std::vector<List>();
  // merged entries: both, M only, F only
  c.rec.assign((size_t)4 * S, 0);
  std::vector<List> e_chunk(chunks);
  std::vector<uint32_t> e_cnt((size_t)S + 1, 0);
  total = 0;
#pragma omp parallel for schedule(dynamic) reduction(+ : total)
  for (int64_t q = 0; q < chunks; ++q) {
    List b, both, m, f;
    for (int64_t s = q * kChunk; s < std::min<int64_t>(S, (q + 1) * kChunk) && !too_long; ++s) {
      b.clear();
      both.clear();
      m.clear();
      f.clear();
      for (uint32_t k = L.vin_off[s]; k < L.vin_off[s + 1]; ++k) {
        const uint32_t u = L.vin_srcv[k], len = L.sv_off[u + 1] - L.sv_off[u];
        b.push_back({(int32_t)u, 0});
        for (uint32_t j = a_off[u]; j < a_off[u + 1]; ++j)
          b.push_back({a[j].src, add_w(a[j].w, (int32_t)(len - 1))});
      }
      tidy(b, -1);
      uint32_t j = a_off[s];
      for (const EdgeW& e : b) {
        for (; j < a_off[s + 1] && a[j].src < e.src; ++j) f.push_back(a[j]);
        if (j < a_off[s + 1] && a[j].src == e.src) {
          if (e.w == a[j].w - 1) {
            both.push_back(e);
          } else {
            if (e.w <= a[j].w) m.push_back(e);
            f.push_back(a[j]);
          }
          ++j;
        } else {
          m.push_back(e);
        }
      }
      for (; j < a_off[s + 1]; ++j) f.push_back(a[j]);
      const size_t n = both.size() + m.size() + f.size();
      if (std::max({both.size(), m.size(), f.size()}) > 255) too_long = true;
      // light entries first: the sources that win are near
      for (List* l : {&both, &m, &f}) {
        std::stable_sort(l->begin(), l->end(), [](const EdgeW& x, const EdgeW& y) { return x.w < y.w; });
        e_chunk[q].insert(e_chunk[q].end(), l->begin(), l->end());
      }
      e_cnt[s + 1] = (uint32_t)n;
      c.rec[4 * s + 3] = (uint32_t)(both.size() | m.size() << 8 | f.size() << 16);
      total += n;
    }
  }
  if (too_long || total > 3 * limit || total > (1u << 30)) return HostClosure{};
  for (uint32_t s = 0; s < S; ++s) e_cnt[s + 1] += e_cnt[s];
  c.ent.resize(total);
#pragma omp parallel for schedule(static)
  for (int64_t q = 0; q < chunks; ++q)
    std::copy(e_chunk[q].begin(), e_chunk[q].end(), c.ent.begin() + e_cnt[q * kChunk]);
  auto key = [&](uint32_t ch) { return (L.lab4[ch >> 3] >> ((ch & 7) * 4)) & 0xFu; };
  auto len_of = [&](uint32_t s) { return L.sv_off[s + 1] - L.sv_off[s]; };
  c.ent16.resize(2 * c.ent.size());
#pragma omp parallel for schedule(static)
  for (int64_t s = 0; s < (int64_t)S; ++s) {
    uint32_t* r = &c.rec[4 * (size_t)s];
    r[0] = L.sv_off[s];
    r[1] = len_of((uint32_t)s) | key(L.sv_off[s]) << 29;
    r[2] = e_cnt[s];
    const uint32_t n = r[3], kb = e_cnt[s] + (n & 255), km = kb + ((n >> 8) & 255);
    for (uint32_t k = e_cnt[s]; k < e_cnt[s + 1]; ++k) {
      const uint32_t w = std::min<uint32_t>((uint32_t)c.ent[k].w, 0xFFFE), none = 0xFFFF;
      const uint32_t wm = k < km ? w : none, wf = k < kb ? w + 1 : k >= km ? w : none;
      c.ent16[2 * (size_t)k] = (uint32_t)c.ent[k].src;
      c.ent16[2 * (size_t)k + 1] = wm | wf << 16;
    }
  }
  for (int i = 0; i < 3; ++i) {
    const uint32_t W = 32u << i;
    std::vector<uint8_t>& out = c.by_len[i];
    out.resize(S);
#pragma omp parallel for schedule(static)
    for (int64_t w0 = 0; w0 < (int64_t)S; w0 += W) {
      const uint32_t n = std::min<uint32_t>(W, S - (uint32_t)w0);
      uint8_t* o = &out[w0];
      std::iota(o, o + n, (uint8_t)0);
      std::stable_sort(o, o + n, [&](uint8_t x, uint8_t y) {
        return len_of((uint32_t)w0 + x) > len_of((uint32_t)w0 + y);
      });
    }
  }
  // the word kernel's order and arrays
  c.pos.resize(S);
  std::vector<uint32_t> at(S);
  auto count = [&](uint32_t s) { return e_cnt[s + 1] - e_cnt[s]; };
  {
    uint32_t h = 0;
    for (uint32_t s = 0; s < S; ++s)
      if (count(s) > kWordLight) at[h++] = s;
    c.heavy = h;
    for (uint32_t s = 0; s < S; ++s)
      if (count(s) <= kWordLight) at[h++] = s;
  }
#pragma omp parallel for schedule(static)
  for (int64_t w0 = c.heavy; w0 < (int64_t)S; w0 += kWordWindow) {
    const auto b = at.begin() + w0, e = at.begin() + std::min<int64_t>(S, w0 + kWordWindow);
    // by list length, then vertices without chain chars together
    auto rank = [&](uint32_t s) { return 2 * count(s) + (len_of(s) > 1 ? 1u : 0u); };
    std::stable_sort(b, e, [&](uint32_t x, uint32_t y) { return rank(x) > rank(y); });
  }
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < (int64_t)S; ++i) c.pos[at[i]] = (uint32_t)i;
  c.wsv.resize((size_t)2 * S);
  c.wrec.resize((size_t)4 * S);
  // groups of 32 positions, counted from the first short list on
  const uint32_t groups = c.heavy / 32 + 1 + (S - c.heavy + 31) / 32;
  auto g_lo = [&](uint32_t q) {  // positions [g_lo(q), g_lo(q + 1))
    const uint32_t hg = c.heavy / 32 + 1;
    return q < hg ? std::min(32 * q, c.heavy) : std::min<uint32_t>(S, c.heavy + 32 * (q - hg));
  };
  std::vector<uint64_t> g_words((size_t)groups + 1, 0), g_ent((size_t)groups + 1, 0);
#pragma omp parallel for schedule(static)
  for (int64_t q = 0; q < (int64_t)groups; ++q) {
    uint64_t w = 0, n = 0;
    for (uint32_t i = g_lo((uint32_t)q); i < g_lo((uint32_t)q + 1); ++i) {
      w += (len_of(at[i]) - 1 + 31) / 32;
      n = i < c.heavy ? n + count(at[i]) : std::max<uint64_t>(n, 32ull * count(at[i]));
    }
    g_words[q + 1] = w;
    g_ent[q + 1] = n;
  }
  for (uint32_t q = 0; q < groups; ++q) {
    g_words[q + 1] += g_words[q];
    g_ent[q + 1] += g_ent[q];
  }
  if (g_words[groups] >= (1ull << 31) || g_ent[groups] >= (1ull << 31)) return HostClosure{};
  c.words = g_words[groups];
  c.lab.assign(4 * (size_t)std::max<uint64_t>(c.words, 1), 0);
  c.went.assign((size_t)g_ent[groups], EdgeW{0, 0});
#pragma omp parallel for schedule(static)
  for (int64_t q = 0; q < (int64_t)groups; ++q) {
    uint64_t wo = g_words[q], eo = g_ent[q];
    const uint32_t lo = g_lo((uint32_t)q);
    for (uint32_t i = lo; i < g_lo((uint32_t)q + 1); ++i) {
      const uint32_t s = at[i], f = L.sv_off[s], len = len_of(s), n = count(s);
      const bool heavy = i < c.heavy;
      uint32_t* r = &c.wrec[4 * (size_t)i];
      c.wsv[2 * (size_t)i] = s;
      c.wsv[2 * (size_t)i + 1] = f;
      r[0] = (uint32_t)wo;
      r[1] = len | key(f) << 29;
      r[2] = (uint32_t)(heavy ? eo : eo + (i - lo));
      r[3] = n;
      const uint32_t nb = c.rec[4 * (size_t)s + 3] & 255, nm = (c.rec[4 * (size_t)s + 3] >> 8) & 255;
      for (uint32_t k = 0; k < n; ++k) {
        const EdgeW& e = c.ent[e_cnt[s] + k];
        const uint32_t cls = k < nb ? 0u : k < nb + nm ? 1u : 2u;
        c.went[r[2] + (heavy ? 1 : 32) * (size_t)k] = EdgeW{(int32_t)((uint32_t)e.src | cls << 30), e.w};
      }
      if (heavy) eo += n;
      for (uint32_t k = 0; k + 1 < len; ++k) {
        uint32_t* w = &c.lab[4 * (wo + k / 32)];
        const uint32_t x = key(f + 1 + k), bit = 1u << (k & 31);
        if (x & 1) w[0] |= bit;
        if (x & 2) w[1] |= bit;
        if (x & 4) w[2] |= bit;
      }
      wo += (len - 1 + 31) / 32;
    }
  }
  c.ok = true;
  return c;
}

}  // namespace chsga
