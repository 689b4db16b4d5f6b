// Host check of what build_closure (closure.cpp) does at its limits, on small
// hand-made layouts and with a counting allocator:
//
//   refused   A graph whose lists would hold 30 times the entries that are
//             allowed is refused before they exist.
//   repeated  A vertex with 100,000 edges from one source with a long list of
//             its own keeps one entry a source on the way, and the result is
//             the list with each source once.
//   memory    std::bad_alloc on any thread comes out of build_closure as
//             itself.
// Exit status 0 and "OK" on success.
#include <malloc.h>
#include <omp.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "closure.hpp"

using namespace chsga;

namespace {
std::atomic<int64_t> live{0}, peak{0}, until_fail{-1};
}

void* operator new(size_t n) {
  // only threads beside the first one run out
  if (until_fail.load() >= 0 && omp_get_thread_num() > 0 && until_fail.fetch_sub(1) <= 0) throw std::bad_alloc();
  void* p = std::malloc(n);
  if (!p) throw std::bad_alloc();
  const int64_t now = live += (int64_t)malloc_usable_size(p);
  int64_t top = peak;
  while (now > top && !peak.compare_exchange_weak(top, now)) {
  }
  return p;
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept {
  if (p) live -= (int64_t)malloc_usable_size(p);
  std::free(p);
}
void operator delete(void* p, size_t) noexcept { operator delete(p); }
void operator delete[](void* p) noexcept { operator delete(p); }
void operator delete[](void* p, size_t) noexcept { operator delete(p); }

namespace {

constexpr uint32_t kSources = 180;

// Vertices: kSources of two chars, `targets` of two chars (level 0) and one of
// one char (level 1) with an upward edge from every source; every target has
// `edges` downward edges from it.
HostLayout layout(uint32_t targets, uint32_t edges) {
  HostLayout L;
  const uint32_t S = L.S = kSources + targets + 1, hub = S - 1;
  L.levels = 2;
  L.lvl_off = {0, hub, S};
  L.sv_off.push_back(0);
  for (uint32_t s = 0; s < S; ++s) {
    L.dv_s.push_back(s);
    L.sv_dev.push_back(s);
    L.dv_len.push_back(s == hub ? 1 : 2);
    L.sv_off.push_back(L.sv_off[s] + L.dv_len[s]);
  }
  L.N = L.sv_off[S];
  L.max_len = 2;
  L.lab4.assign(L.N / 8 + 4, 0);
  L.vin_off.assign(S + 1, 0);
  L.up_off.assign(S + 1, 0);
  L.up_off[S] = kSources;
  for (uint32_t s = 0; s < kSources; ++s) L.up_in.push_back({(int32_t)(2 * s + 1), (int32_t)(1 + s)});
  L.dn_off.assign(S + 1, 0);
  for (uint32_t s = 0; s < S; ++s) {
    if (s >= kSources && s < hub)
      for (uint32_t k = 0; k < edges; ++k) L.dn_in.push_back({(int32_t)(2 * hub), (int32_t)(5 + edges - k)});
    L.dn_off[s + 1] = (uint32_t)L.dn_in.size();
  }
  return L;
}

int fails = 0;
void check(bool ok, const char* what) {
  if (!ok) ++fails, std::printf("FAIL: %s\n", what);
}

}  // namespace

int main() {
  omp_set_num_threads(4);
  {
    const HostLayout L = layout(200'000, 1);
    peak = live.load();
    const int64_t base = live;
    const HostClosure c = build_closure(L);
    check(!c.ok, "lists of 181 entries an edge are refused");
    std::printf("refused: %.1f MB\n", (double)(peak - base) / 1e6);
    check(peak - base < 60'000'000, "a refused graph's lists are never built in full");
  }
  {
    const HostLayout L = layout(1, 100'000);
    peak = live.load();
    const int64_t base = live;
    const HostClosure c = build_closure(L);
    check(c.ok, "repeated edges are one entry");
    std::printf("repeated: %.1f MB\n", (double)(peak - base) / 1e6);
    check(peak - base < 10'000'000, "repeated edges are dropped on the way");
    if (c.ok) {
      const uint32_t* r = &c.rec[4 * kSources];
      check(r[3] == (kSources + 1) << 16, "the target's entries");
      for (uint32_t k = 0; k < kSources + 1; ++k) {
        const EdgeW& e = c.ent[r[2] + k];
        // smallest weight of an edge, 6, and of its source's own edge
        check(e.w == 6 + (e.src < (int32_t)kSources ? 1 + e.src : 0), "the target's weights");
      }
    }
  }
  {
    const HostLayout L = layout(5'000, 1);
    HostLayout M = L;  // accepted: every target's list is its own edge
    M.up_in.resize(3);
    for (uint32_t s = M.S; s <= M.S; ++s) M.up_off[s] = 3;
    check(build_closure(M).ok, "short lists are accepted");
    int thrown = 0;
    for (int64_t n = 0; n < 40; ++n) {
      until_fail = n;
      try {
        build_closure(M);
      } catch (const std::bad_alloc&) {
        ++thrown;
      }
      until_fail = -1;
    }
    check(thrown > 20, "std::bad_alloc of another thread is passed on");
    check(build_closure(M).ok, "and the next build is whole");
  }
  if (fails) return 1;
  std::printf("OK\n");
  return 0;
}
