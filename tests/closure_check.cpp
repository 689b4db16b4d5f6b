// Host check of the closure lists (closure.cpp) and of the bit-row word
// operations (row_bits.hpp).
//
//   lists  On generated graphs and random raw scores, every vertex's first
//          score from its list equals the level-by-level sweeps (upward
//          levels rising, downward levels falling, last scores of vertices of
//          two or more chars never refreshed), and the first char's update
//          min(F + 1, min over in-edges of final last + delta) from the
//          merged list equals the one from the in-edges.
//   words  On random rows, lowering under a line and the bit update give the
//          differences of the scalar recurrences, across word boundaries.
// Exit status 0 and "OK" on success.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>

#include "chsga.h"
#include "closure.hpp"
#include "row_bits.hpp"

using namespace chsga;

namespace {

int fails = 0;

void check(bool ok, const std::string& what) {
  if (!ok && fails++ < 20) std::printf("FAIL: %s\n", what.c_str());
}

void check_lists(const HostLayout& L, const HostClosure& c, std::mt19937_64& rng, int range) {
  std::vector<int64_t> bv(2 * (size_t)L.S), raw_f(L.S), raw_l(L.S), fin(L.S);
  for (uint32_t s = 0; s < L.S; ++s) {
    const int64_t len = L.sv_off[s + 1] - L.sv_off[s];
    raw_f[s] = (int64_t)(rng() % range);
    raw_l[s] = len == 1 ? raw_f[s] : std::min<int64_t>(raw_f[s] + len - 1, (int64_t)(rng() % range));
    bv[2 * (size_t)L.sv_dev[s]] = raw_f[s];
    bv[2 * (size_t)L.sv_dev[s] + 1] = raw_l[s];
  }
  for (uint32_t l = 0; l < L.levels; ++l)
    for (uint32_t d = L.lvl_off[l]; d < L.lvl_off[l + 1]; ++d)
      for (uint32_t e = L.up_off[d]; e < L.up_off[d + 1]; ++e)
        bv[2 * (size_t)d] = std::min(bv[2 * (size_t)d], bv[L.up_in[e].src] + L.up_in[e].w);
  for (uint32_t l = L.levels; l-- > 0;)
    for (uint32_t d = L.lvl_off[l]; d < L.lvl_off[l + 1]; ++d)
      for (uint32_t e = L.dn_off[d]; e < L.dn_off[d + 1]; ++e)
        bv[2 * (size_t)d] = std::min(bv[2 * (size_t)d], bv[L.dn_in[e].src] + L.dn_in[e].w);
  for (uint32_t s = 0; s < L.S; ++s) fin[s] = bv[2 * (size_t)L.sv_dev[s]];
  for (uint32_t s = 0; s < L.S; ++s) {
    const uint32_t* r = &c.rec[4 * (size_t)s];
    check((r[1] & 0x1FFFFFFFu) == L.sv_off[s + 1] - L.sv_off[s], "record length");
    int64_t F = raw_f[s], M = 1 << 28;
    const EdgeW* e = &c.ent[r[2]];
    for (uint32_t k = 0; k < (r[3] & 255); ++k, ++e) {
      M = std::min(M, raw_l[e->src] + e->w);
      F = std::min(F, raw_l[e->src] + e->w + 1);
    }
    for (uint32_t k = 0; k < ((r[3] >> 8) & 255); ++k, ++e) M = std::min(M, raw_l[e->src] + e->w);
    for (uint32_t k = 0; k < ((r[3] >> 16) & 255); ++k, ++e) F = std::min(F, raw_l[e->src] + e->w);
    check(F == fin[s], "first score of vertex " + std::to_string(s));
    int64_t want = 1 << 28;
    for (uint32_t k = L.vin_off[s]; k < L.vin_off[s + 1]; ++k) {
      const uint32_t u = L.vin_srcv[k];
      want = std::min(want, std::min(raw_l[u], fin[u] + (int64_t)(L.sv_off[u + 1] - L.sv_off[u]) - 1));
    }
    for (int delta = 0; delta < 2; ++delta)
      check(std::min(F + 1, M + delta) == std::min(fin[s] + 1, want + delta),
            "first char of vertex " + std::to_string(s));
  }
}

// One vertex of `len` chars: scalar recurrences against words.
void check_words(uint32_t len, std::mt19937_64& rng) {
  std::vector<int> raw(len), D(len), T(len), delta(len);
  raw[0] = 500;
  for (uint32_t i = 1; i < len; ++i) raw[i] = raw[i - 1] + (int)(rng() % 3) - 1;
  for (auto& x : delta) x = (int)(rng() % 2);
  const int gap = (int)(rng() % 4) * (int)(rng() % 5), F = raw[0] - gap;
  for (uint32_t i = 0; i < len; ++i) D[i] = std::min(raw[i], F + (int)i);
  T[0] = F + 1 - (int)(rng() % 6);  // also below F - 1
  for (uint32_t i = 1; i < len; ++i) T[i] = std::min(std::min(D[i] + 1, D[i - 1] + delta[i]), T[i - 1] + 1);
  const int Tc = std::max(T[0], F - 1);
  uint32_t g = (uint32_t)gap, low = (uint32_t)(Tc - T[0]);
  int h = Tc - F, cur = T[0];
  for (uint32_t w0 = 1; w0 < len; w0 += 32) {
    const uint32_t n = std::min(32u, len - w0), valid = 0xFFFFFFFFu >> (32 - n);
    bits::PN x{0, 0};
    uint32_t mis = 0;
    for (uint32_t k = 0; k < n; ++k) {
      const int d = raw[w0 + k] - raw[w0 + k - 1];
      if (d > 0) x.p |= 1u << k;
      if (d < 0) x.n |= 1u << k;
      if (delta[w0 + k]) mis |= 1u << k;
    }
    x = bits::under_line(x, valid, g);
    for (uint32_t k = 0; k < n; ++k)
      check((int)((x.p >> k) & 1) - (int)((x.n >> k) & 1) == D[w0 + k] - D[w0 + k - 1], "lowered difference");
    x = bits::step(x, mis, h, n - 1);
    x = bits::under_line(x, valid, low);
    for (uint32_t k = 0; k < n; ++k) {
      cur += (int)((x.p >> k) & 1) - (int)((x.n >> k) & 1);
      check(cur == T[w0 + k], "updated score " + std::to_string(w0 + k) + " of " + std::to_string(len));
    }
  }
  if (len > 1) check(std::min(D[len - 1] + h, T[0] + (int)len - 1) == T[len - 1], "last score");
}

}  // namespace

int main() {
  std::mt19937_64 rng(5);
  for (int i = 0; i < 20000; ++i) check_words(1 + (uint32_t)(rng() % 100), rng);
  uint32_t checked = 0, refused = 0;
  // labels of 1..32, 1..4 and 2..70 chars, dense and sparse bubbles, and
  // one-char vertices only (whose lists are refused)
  const struct {
    uint64_t bb;
    double gap;
    uint32_t lo, hi;
  } cases[] = {{30000, 50, 1, 32}, {200000, 90, 1, 32}, {20000, 20, 1, 4}, {50000, 30, 2, 70}, {300, 20, 1, 1},
               {4000, 50, 1, 1}};
  for (const auto& k : cases) {
    chsga_gen_graph_cfg cfg{k.bb, 7 + k.bb, k.gap, 0.7, 0.2, 0.1, 1, 20, 50, 300, k.lo, k.hi};
    chsga_host_graph* g = nullptr;
    if (chsga_gen_graph(&cfg, &g) != CHSGA_OK) return 2;
    chsga_pch_opts po{500, 1.0, 0, 1, 0x5EED, 0, 0, 0, 0};
    if (chsga_build_pch(g, &po) != CHSGA_OK) return 2;
    chsga_graph_host view{};
    chsga_graph_view(g, &view);
    const HostLayout L = build_layout(view);
    const HostClosure c = build_closure(L);
    if (c.ok)
      for (int range : {3, 40, 2000}) {
        check_lists(L, c, rng, range);
        ++checked;
      }
    else
      ++refused;
    chsga_graph_free(g);
  }
  if (fails || checked < 9 || refused < 1) {
    std::printf("%d failures, %u graphs checked, %u refused\n", fails, checked, refused);
    return 1;
  }
  std::printf("OK: %u list sets checked, %u graphs refused\n", checked, refused);
  return 0;
}
