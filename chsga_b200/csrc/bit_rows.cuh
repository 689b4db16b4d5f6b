// Bit-row kernels: a whole row-step of every slot in one launch.
//
// A row is kept as the raw first and last score of every string vertex (RF,
// RL) and two difference bits per chain char (row_bits.hpp). The hierarchy
// closure is one minimum per vertex over raw last scores (closure.hpp), so
// one pass over the vertices takes a row to the next: for vertex v
//     F = min(RF(v), A(v)),  M = B(v)            closure of the previous row
//     T = min(F + 1, M + delta)                  new raw first score
//     chain: previous differences lowered under the line F + (c - first),
//            then the bit update with the change T - F carried in
//     new RF(v) = T, RL(v) = last chain score
// RF and RL alternate between two buffers (other vertices gather the old
// ones); the bits are the vertex's own and are updated in place, or written
// into the read's matrix (traceback). Nothing orders one vertex after
// another, so the row-step has no phases between blocks, and the block that
// finishes last moves the slots on (bits_advance).
//
// A row's minimum after its closure needs the closure's first scores, which
// the next row-step computes: a read on its last row leaves its slot with its
// raw minimum and "drains" during the next row-step, where the slot may
// already compute row 0 of the next read (two minima per slot, by parity).
//
// If T < F - 1 (the sweeps read last scores they do not refresh, so a first
// score can fall by more than the bits carry) the chain runs from F - 1 and
// the new row is lowered under the line from T: T[c] = min(chain, T + c - f).
#pragma once

#include "kernels.cuh"
#include "row_bits.hpp"

namespace chsga {
namespace dev {

constexpr uint32_t SW_DRAIN = 1u << 13;  // the slot's previous read takes its closure minimum
constexpr uint32_t SW_PAR = 1u << 14;    // which of the slot's two minima its current read uses

// Words of the current row-step for the bit-sliced kernel, written by
// bits_advance: per label key the mismatch bits of 32 slots, and the same per
// slot as 16-bit increments; row-0 (or idle), last-row and draining slots.
struct StepTab {
  uint32_t mis[8][4];
  uint32_t keep[4];   // 0 where the slot is on row 0 or idle
  uint32_t end[4];
  uint32_t drain[4];
  uint32_t any_end, any_drain, pad[2];
  uint16_t mis16[8][128];
  uint16_t init16[128];  // 0xFFFF on row 0 or idle
};

struct BitGraph {
  uint32_t S, n_ent;
  uint64_t words;
  const uint4* rec;       // closure.hpp
  const uint2* ent;
  const uint4* lab;
  const uint8_t* by_list;
  const uint8_t* by_len;  // of the kernel's window
  const uint32_t* sv_off;
  const uint32_t* lab4;
  uint32_t N;
};

// Where a slot's previous and current rows lie in its read's matrix
// (traceback): {bits, RF, F} of a row, row_bits_layout.
struct SlotRows {
  unsigned char* prev;
  unsigned char* cur;
};

struct AdvanceArgs {
  SlotState* slots;
  const ReadDesc* queue;
  const unsigned char* reads;
  int32_t* res_score;
  uint32_t* res_vertex;
  unsigned long long *res_t0, *res_t1;
  CompletionRec* done_ring;
  uint32_t qmask;
  int special, match_n;
  // traceback: matrix of every read id and the slots' row pointers
  unsigned char* const* mats;
  SlotRows* rows;
  size_t pitch;
};

struct BitArgs {
  BitGraph g;
  const void *RFin, *RLin;
  void *RFout, *RLout;
  void* bits;  // uint2 words (one read a word) or bit-sliced char words
  uint32_t* word;
  StepTab* tab;
  unsigned long long* best;  // [2][R]
  StepCtl* ctl;
  AdvanceArgs adv;
};

// Moves every slot to its next row (one block, at least R threads): finishes
// the reads that drained, lets reads past their last row drain, admits queued
// reads and writes the slot words and tables of the next row-step. prime:
// only the first admission (nothing was computed yet).
template <int R>
__device__ void bits_advance(const AdvanceArgs& a, uint32_t* slot_word, StepTab* tab, unsigned long long* best,
                             StepCtl* ctl, bool prime) {
  static_assert(R <= 128, "one thread per slot");
  __shared__ uint32_t s_need[128];
  __shared__ uint32_t s_base, s_take, s_active, s_ending, s_drain;
  const int r = threadIdx.x;
  SlotState st{};
  bool need = false;
  uint32_t drain = 0, par = 0;
  if (r == 0) s_active = s_ending = s_drain = 0;
  SlotRows sr{nullptr, nullptr};
  if (r < R) {
    st = a.slots[r];
    par = st.pad & 1u;
    if (a.mats) sr = a.rows[r];
    sr.prev = sr.cur;
    if (!prime) {
      const int32_t did = (int32_t)(st.pad >> 1) - 1;
      if (did >= 0) {
        const unsigned long long b = __ldcg(best + (par ^ 1u) * R + r);
        const unsigned long long t1 = global_ns();
        a.res_score[did] = (int32_t)(b >> 32);
        a.res_vertex[did] = (uint32_t)(b & 0xffffffffu);
        a.res_t1[did] = t1;
        const uint32_t k = atomicAdd(&ctl->done, 1u);
        if (a.done_ring)
          a.done_ring[k & a.qmask] = CompletionRec{did, (int32_t)(b >> 32), (uint32_t)(b & 0xffffffffu), 0u,
                                                   a.res_t0[did], t1};
      }
      if (st.id >= 0) {
        if (st.row + 1 >= st.len) {
          drain = (uint32_t)st.id + 1;
          st.id = -1;
          par ^= 1u;
        } else {
          st.row += 1;
        }
      }
    }
    need = st.id < 0;
  }
  if (r < 128) s_need[r] = need ? 1u : 0u;
  __syncthreads();
  if (r == 0) {
    uint32_t total = 0;
    for (int i = 0; i < R; ++i) {
      const uint32_t n = s_need[i];
      s_need[i] = total;
      total += n;
    }
    const uint32_t avail = ctl->q_count - ctl->q_head;
    s_take = total < avail ? total : avail;
    s_base = ctl->q_head;
    ctl->q_head += s_take;
  }
  __syncthreads();
  uint32_t w = 0;
  if (r < R) {
    if (need && s_need[r] < s_take) {
      const ReadDesc q = a.queue[(s_base + s_need[r]) & a.qmask];
      st.off = q.off;
      st.len = q.len;
      st.row = 0;
      st.id = q.id;
      best[par * R + r] = ~0ull;
      a.res_t0[q.id] = global_ns();
    }
    if (st.id >= 0) {
      const int byte = a.reads[st.off + st.row];
      w = base_code(byte, a.special) | (mismatch_mask(byte, a.special, a.match_n) << SW_MASK_SHIFT) | SW_ACTIVE;
      w |= st.row == 0 ? SW_INIT : SW_CLOSURE;
      if (st.row + 1 == st.len) w |= SW_ENDING;
      if (a.mats) sr.cur = a.mats[st.id] + (size_t)st.row * a.pitch;
    }
    if (drain) w |= SW_DRAIN;
    if (par) w |= SW_PAR;
    st.pad = drain << 1 | par;
    if (w & (SW_ACTIVE | SW_DRAIN)) atomicOr(&s_active, 1u);
    if (w & SW_ENDING) atomicOr(&s_ending, 1u);
    if (w & SW_DRAIN) atomicOr(&s_drain, 1u);
    a.slots[r] = st;
    slot_word[r] = w;
    if (a.mats) a.rows[r] = sr;
  }
  if constexpr (R >= 32) {
    if (r < R) {
      const bool init = (w & SW_INIT) || !(w & SW_ACTIVE);
      const uint32_t m = (w >> SW_MASK_SHIFT) & SW_MASK;
      const int g = r >> 5;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t bit = (m >> k) & 1u;
        const uint32_t word = __ballot_sync(0xFFFFFFFFu, bit);
        if ((r & 31) == 0) tab->mis[k][g] = word;
        tab->mis16[k][r] = (uint16_t)bit;
      }
      tab->init16[r] = init ? 0xFFFFu : 0u;
      const uint32_t ki = __ballot_sync(0xFFFFFFFFu, !init), ke = __ballot_sync(0xFFFFFFFFu, (w & SW_ENDING) != 0),
                     kd = __ballot_sync(0xFFFFFFFFu, (w & SW_DRAIN) != 0);
      if ((r & 31) == 0) {
        tab->keep[g] = ki;
        tab->end[g] = ke;
        tab->drain[g] = kd;
      }
    }
  }
  __syncthreads();
  if (r == 0) {
    if constexpr (R >= 32) {
      tab->any_end = s_ending;
      tab->any_drain = s_drain;
    }
    ctl->any_active = s_active;
    ctl->any_ending = s_ending | s_drain;
    ctl->arrive = 0;
    if (s_active) ctl->steps += 1;
  }
}

template <int R>
__global__ void __launch_bounds__(128) k_bits_advance(BitArgs a, int prime) {
  pdl_wait();
  bits_advance<R>(a.adv, a.word, a.tab, a.best, a.ctl, prime != 0);
}

// The last block of the launch moves the slots on. Every thread's writes of
// this block are ordered before the arrival (block barrier, then a fence by
// the arriving thread); the last arrival's block sees them all.
template <int R>
__device__ __forceinline__ void bits_finish(const BitArgs& a, uint32_t nblocks) {
  __shared__ uint32_t s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.ctl->arrive, 1u) == nblocks - 1;
    __threadfence();
  }
  __syncthreads();
  if (s_last) bits_advance<R>(a.adv, a.word, a.tab, a.best, a.ctl, false);
}

// Nothing to compute in this launch: true, and when reads wait in the queue
// (published to an idle engine) the launch still ends in their admission.
// Every block takes the same way: only the last arrival changes the words
// this reads.
template <int R>
__device__ __forceinline__ bool bits_idle(const BitArgs& a, uint32_t nblocks) {
  if (a.ctl->any_active) return false;
  if (a.ctl->q_count != a.ctl->q_head) bits_finish<R>(a, nblocks);
  return true;
}

// Row layout of a traceback matrix: bit words, raw first scores, first
// scores after the closure (written by the next row-step).
__host__ __device__ constexpr size_t bits_row_rf(uint64_t words) { return (size_t)words * 8; }
__host__ __device__ constexpr size_t bits_row_f(uint64_t words, uint32_t S) {
  return bits_row_rf(words) + ((size_t)S * 2 + 15) / 16 * 16;
}
__host__ __device__ constexpr size_t bits_row_bytes(uint64_t words, uint32_t S) {
  return (bits_row_f(words, S) + (size_t)S * 2 + 255) / 256 * 256;
}

// ---------------------------------------------------------------------------
// k_row_words: one thread per (string vertex, slot), a vertex's chain in
// words of 32 chars. Slots are interleaved (RF[s * R + r], word w of slot r at
// w * R + r), so the gathers of neighbouring slots share sectors; with MAT
// every slot is blockIdx.y of a one-slot launch with rows in its read's
// matrix. Vertices of a 256-vertex window are taken by list length, so a
// warp's lists end together.
// ---------------------------------------------------------------------------
template <int R, typename ST, bool MAT>
__global__ void __launch_bounds__(256) k_row_words(BitArgs a) {
  static_assert(!MAT || (R == 1 && sizeof(ST) == 2), "matrix rows hold one slot each, 16 bits");
  using bits::PN;
  constexpr int VB = 256 / R;  // vertices per block
  const BitGraph& g = a.g;
  const int r = MAT ? (int)blockIdx.y : (int)(threadIdx.x % R);
  const uint32_t i = blockIdx.x * VB + threadIdx.x / R;  // position in the windows' order
  uint32_t s = 0;
  uint4 rec = make_uint4(0, 1, 0, 0);
  if (i < g.S) {
    s = (i & ~255u) + __ldg(g.by_list + i);
    s = CHSGA_CHK(s, g.S, 20);
    rec = __ldg(g.rec + s);
  }
  pdl_wait();
  if constexpr (MAT) {
    if (!a.ctl->any_active) return;
  } else {
    if (bits_idle<R>(a, gridDim.x)) return;
  }
  const uint32_t w = a.word[r];
  const bool init = (w & SW_INIT) != 0;
  constexpr int NB = R;  // minima per block
  __shared__ unsigned long long s_min[2 * NB];
  const bool ends = a.ctl->any_ending != 0;
  if (ends) {
    if (threadIdx.x < 2 * NB) s_min[threadIdx.x] = ~0ull;
    __syncthreads();
  }
  const ST *RFin, *RLin;
  ST *RFout, *RLout, *Fout = nullptr;
  const uint2* win;
  uint2* wout;
  if constexpr (MAT) {
    const SlotRows sr = a.adv.rows[r];
    const size_t rf = bits_row_rf(g.words);
    RFin = reinterpret_cast<const ST*>(sr.prev + rf);
    RFout = reinterpret_cast<ST*>(sr.cur + rf);
    Fout = reinterpret_cast<ST*>(sr.prev + bits_row_f(g.words, g.S));
    win = reinterpret_cast<const uint2*>(sr.prev);
    wout = reinterpret_cast<uint2*>(sr.cur);
    RLin = static_cast<const ST*>(a.RLin) + (size_t)r * g.S;
    RLout = static_cast<ST*>(a.RLout) + (size_t)r * g.S;
  } else {
    RFin = static_cast<const ST*>(a.RFin) + r;
    RLin = static_cast<const ST*>(a.RLin) + r;
    RFout = static_cast<ST*>(a.RFout) + r;
    RLout = static_cast<ST*>(a.RLout) + r;
    win = static_cast<const uint2*>(a.bits) + r;
    wout = static_cast<uint2*>(a.bits) + r;
  }
  if (i < g.S && (w & (SW_ACTIVE | SW_DRAIN))) {
    const uint32_t len = rec.y & 0x1FFFFFFFu, key = rec.y >> 29, mask = (w >> SW_MASK_SHIFT) & SW_MASK;
    const uint32_t nb = rec.w & 0xFFu, nm = (rec.w >> 8) & 0xFFu, nf = (rec.w >> 16) & 0xFFu;
    const uint32_t nw = (len + 30) / 32;
    const int delta = (int)((mask >> key) & 1u);
    unsigned long long mn = ~0ull;
    // closure of the previous row (a no-op on row 0: its scores are 0 and 1
    // and every weight is at least 1)
    int rf = 0, F = 0, M = 0x3fffffff, dl = 0;
    if (!init || (w & SW_DRAIN)) {
      rf = (int)__ldg(RFin + (size_t)s * R);
      dl = (int)__ldg(RLin + (size_t)s * R);
      uint32_t k0 = rec.z, k1 = k0 + nb + nm + nf;
      CHSGA_CHK_RANGE(k0, k1, g.n_ent, 21);
      const uint32_t kb = k0 + nb, km = kb + nm;
      F = rf;
      constexpr int U = 4;  // gathers in flight
      for (uint32_t k = k0; k < k1; k += U) {
        uint2 e[U];
        int x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < k1) e[u] = __ldg(g.ent + k + u);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < k1) x[u] = (int)__ldg(RLin + (size_t)CHSGA_CHK(e[u].x, g.S, 22) * R) + (int)e[u].y;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < k1) {
            if (k + u < km) M = min(M, x[u]);
            if (k + u < kb || k + u >= km) F = min(F, x[u] + (k + u < kb ? 1 : 0));
          }
      }
      if (MAT && (w & SW_DRAIN || !init)) Fout[s] = (ST)F;
      if (w & SW_DRAIN) mn = pack_min(F, __ldg(g.sv_off + s));
    }
    if (w & SW_DRAIN) atomicMin(&s_min[(((w & SW_PAR) ? 0 : 1)) * NB + (MAT ? 0 : r)], mn);
    if (w & SW_ACTIVE) {
      int T, last;
      if (init) {
        T = delta;
        uint32_t left = (uint32_t)delta;
        for (uint32_t j = 0; j < nw; ++j) {
          const size_t wi = (size_t)CHSGA_CHK(rec.x + j, g.words, 23);
          const uint4 lb = __ldg(g.lab + wi);
          const PN x = bits::first_row(bits::mismatch_word(lb.x, lb.y, lb.z, mask), left, min(31u, len - 2 - 32 * j));
          wout[wi * R] = make_uint2(x.p, x.n);
        }
        last = (int)left;
      } else {
        T = min(F + 1, M + delta);
        const int Tc = max(T, F - 1);
        uint32_t gap = (uint32_t)(rf - F), low = (uint32_t)(Tc - T);
        int h = Tc - F;
        for (uint32_t j = 0; j < nw; ++j) {
          const size_t wi = (size_t)CHSGA_CHK(rec.x + j, g.words, 23);
          const uint4 lb = __ldg(g.lab + wi);
          const uint2 old = win[wi * R];
          const uint32_t top = min(31u, len - 2 - 32 * j), valid = 0xFFFFFFFFu >> (31 - top);
          PN x = bits::under_line(PN{old.x, old.y}, valid, gap);
          x = bits::step(x, bits::mismatch_word(lb.x, lb.y, lb.z, mask), h, top);
          x = bits::under_line(x, valid, low);
          wout[wi * R] = make_uint2(x.p, x.n);
        }
        last = len > 1 ? min(min(dl, F + (int)(len - 1)) + h, T + (int)(len - 1)) : T;
      }
      RFout[(size_t)s * R] = (ST)T;
      RLout[(size_t)s * R] = (ST)last;
      if (w & SW_ENDING) {
        // the raw row's minimum and its first char
        const uint32_t f = __ldg(g.sv_off + s);
        int cur = T, bm = T;
        uint32_t bc = f;
        for (uint32_t j = 0; j < nw; ++j) {
          const uint2 x = wout[((size_t)rec.x + j) * R];
          const uint32_t n = min(32u, len - 1 - 32 * j);
          for (uint32_t k = 0; k < n; ++k) {
            cur += (int)((x.x >> k) & 1u) - (int)((x.y >> k) & 1u);
            if (cur < bm) {
              bm = cur;
              bc = f + 1 + 32 * j + k;
            }
          }
        }
        atomicMin(&s_min[((w & SW_PAR) ? 1 : 0) * NB + (MAT ? 0 : r)], pack_min(bm, bc));
      }
    }
  }
  if (ends) {
    __syncthreads();
    // the minima's array is [parity][slot]
    const int slots = MAT ? (int)gridDim.y : R;
    if (threadIdx.x < 2 * NB && s_min[threadIdx.x] != ~0ull) {
      const int p = threadIdx.x / NB, q = MAT ? r : (int)(threadIdx.x % NB);
      atomicMin(a.best + (MAT ? p * slots : p * NB) + q, s_min[threadIdx.x]);
    }
  }
  if constexpr (!MAT) bits_finish<R>(a, gridDim.x);
}

// ---------------------------------------------------------------------------
// k_row_sliced: 32 to 128 slots, 16-bit scores, bits sliced over the slots:
// word pair {P, N} g of char c (slots 32g .. 32g+31) at c * R/32 + g. Each
// char of 32 slots is a handful of logic operations, where the packed 16-bit
// update spends tens of instructions.
//
// A block takes a window of 8192 / R vertices in three passes:
//   1  thread = (vertex, 8 slots): closure and first char in 16-bit pairs;
//      the gap RF - F, the change T - F and rare cases leave as bytes
//   2  thread = (vertex, 32 slots), vertices by length: the chain
//   3  thread = (vertex, 8 slots): last scores
// The gap of a vertex that the line lowers is a two-bit counter per slot; a
// larger gap (none was seen on variation graphs; gaps of 1 and 2 are common)
// and a chain to be lowered under its own first score take a scalar pass
// over that slot's chars.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 min4(const uint4& a, const uint4& b) {
  return make_uint4(__vminu2(a.x, b.x), __vminu2(a.y, b.y), __vminu2(a.z, b.z), __vminu2(a.w, b.w));
}
__device__ __forceinline__ uint4 max4(const uint4& a, const uint4& b) {
  return make_uint4(__vmaxu2(a.x, b.x), __vmaxu2(a.y, b.y), __vmaxu2(a.z, b.z), __vmaxu2(a.w, b.w));
}
__device__ __forceinline__ uint4 addw4(const uint4& a, uint32_t w) {  // saturating, the same w for every slot
  return make_uint4(__vaddus2(a.x, w), __vaddus2(a.y, w), __vaddus2(a.z, w), __vaddus2(a.w, w));
}
__device__ __forceinline__ uint4 add4(const uint4& a, const uint4& b) {
  return make_uint4(__vaddus2(a.x, b.x), __vaddus2(a.y, b.y), __vaddus2(a.z, b.z), __vaddus2(a.w, b.w));
}
__device__ __forceinline__ uint4 sub4(const uint4& a, const uint4& b) {  // no half borrows
  return make_uint4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
}
__device__ __forceinline__ uint4 sel4(const uint4& a, const uint4& b, const uint4& m) {
  return make_uint4(sel(a.x, b.x, m.x), sel(a.y, b.y, m.y), sel(a.z, b.z, m.z), sel(a.w, b.w, m.w));
}
// Values 0..3 of 8 slots to their two bit planes (bit j = slot j of the 8).
__device__ __forceinline__ void planes2(const uint4& x, uint32_t& lo, uint32_t& hi) {
  const uint32_t y = x.x + (x.y << 2) + (x.z << 4) + (x.w << 6);
  const uint32_t a = y & 0x00550055u, b = (y >> 1) & 0x00550055u;
  lo = (a | (a >> 15)) & 0xFFu;
  hi = (b | (b >> 15)) & 0xFFu;
}
// One bit of 8 slots to 16-bit values.
__device__ __forceinline__ uint4 unplane(uint32_t byte) {
  const uint32_t y = byte | (byte << 15);
  return make_uint4(y & 0x00010001u, (y >> 2) & 0x00010001u, (y >> 4) & 0x00010001u, (y >> 6) & 0x00010001u);
}
// 8 slots: bit j set where value j is not 0.
__device__ __forceinline__ uint32_t nonzero8(const uint4& x) {
  const uint32_t v[4] = {x.x, x.y, x.z, x.w};
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) m |= ((v[j] & 0xFFFFu) ? 1u : 0u) << (2 * j) | ((v[j] >> 16) ? 1u : 0u) << (2 * j + 1);
  return m;
}

// Lowers slot bit `bit` of the n chars at p (stride W word pairs) under a
// line that starts `gap` below their left neighbour.
__device__ __noinline__ void line_slot(uint2* p, int W, uint32_t n, uint32_t bit, uint32_t gap) {
  for (uint32_t k = 0; k < n && gap; ++k, p += W) {
    uint2 x = *p;
    if (x.x & bit) continue;
    const bool down = (x.y & bit) != 0;
    x.y &= ~bit;
    if (down && gap == 1) {
      gap = 0;
    } else {
      x.x |= bit;
      gap -= down ? 2u : 1u;
    }
    *p = x;
  }
}

#ifndef CHSGA_SLICED_BLOCKS
#define CHSGA_SLICED_BLOCKS 4  // blocks per SM the register budget is sized for (build-time tuning)
#endif
template <int R>
__global__ void __launch_bounds__(256, CHSGA_SLICED_BLOCKS) k_row_sliced(BitArgs a) {
  constexpr int C = R / 8, W = R / 32, VB = 8192 / R, NT = 256;
  constexpr uint32_t ONES = 0x00010001u;
  const BitGraph& g = a.g;
  __shared__ __align__(16) uint16_t sF[VB * R];
  enum { G0, G1, VP, VN, GBIG, LOW, NPL };
  __shared__ __align__(4) uint8_t sP[NPL][VB * C];
  __shared__ __align__(16) uint4 sMis16[8 * C], sInit[C];
  __shared__ uint32_t sMis[8 * W], sKeep[W], sEnd[W];
  __shared__ unsigned long long sMin[2 * R];
  const uint32_t v0 = blockIdx.x * VB;
  const uint32_t nv = min((uint32_t)VB, g.S - v0);
  pdl_wait();
  if (bits_idle<R>(a, gridDim.x)) return;
  const StepTab* tab = a.tab;
  const bool ends = a.ctl->any_ending != 0;
  for (int i = threadIdx.x; i < 8 * C; i += NT)
    sMis16[i] = *(reinterpret_cast<const uint4*>(tab->mis16[i / C]) + i % C);
  if (threadIdx.x < C) sInit[threadIdx.x] = *(reinterpret_cast<const uint4*>(tab->init16) + threadIdx.x);
  if (threadIdx.x < 8 * W) sMis[threadIdx.x] = tab->mis[threadIdx.x / W][threadIdx.x % W];
  if (threadIdx.x < W) {
    sKeep[threadIdx.x] = tab->keep[threadIdx.x];
    sEnd[threadIdx.x] = tab->end[threadIdx.x];
  }
  if (ends)
    for (int i = threadIdx.x; i < 2 * R; i += NT) sMin[i] = ~0ull;
  __syncthreads();
  const uint16_t* RFin = static_cast<const uint16_t*>(a.RFin);
  const uint16_t* RLin = static_cast<const uint16_t*>(a.RLin);
  uint16_t* RFout = static_cast<uint16_t*>(a.RFout);
  uint16_t* RLout = static_cast<uint16_t*>(a.RLout);
  const bool drains = ends && tab->any_drain != 0;
  // ---- pass 1
  for (uint32_t it = threadIdx.x; it < nv * C; it += NT) {
    const uint32_t vl = it / C, q = it % C, s = v0 + vl;
    const uint4 rec = __ldg(g.rec + s);
    const uint32_t key = rec.y >> 29;
    const size_t so = (size_t)s * R + 8 * q;
    const uint4 rf = __ldg(reinterpret_cast<const uint4*>(RFin + so));
    const uint32_t nb = rec.w & 0xFFu, nm = (rec.w >> 8) & 0xFFu, nf = (rec.w >> 16) & 0xFFu;
    uint32_t k0 = rec.z, k1 = k0 + nb + nm + nf;
    CHSGA_CHK_RANGE(k0, k1, g.n_ent, 21);
    const uint32_t kb = k0 + nb, km = kb + nm;
    uint4 F = rf, M = make_uint4(~0u, ~0u, ~0u, ~0u);
    constexpr int U = 4;
    for (uint32_t k = k0; k < k1; k += U) {
      uint2 e[U];
      uint4 x[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + u < k1) e[u] = __ldg(g.ent + k + u);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + u < k1)
          x[u] = __ldg(reinterpret_cast<const uint4*>(RLin + (size_t)CHSGA_CHK(e[u].x, g.S, 22) * R + 8 * q));
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + u < k1) {
          const uint4 y = addw4(x[u], min(e[u].y, 0xFFFFu) * ONES);
          if (k + u < km) M = min4(M, y);
          if (k + u < kb)
            F = min4(F, addw4(y, ONES));
          else if (k + u >= km)
            F = min4(F, y);
        }
    }
    const uint4 d = sMis16[key * C + q], in = sInit[q];
    const uint4 one = make_uint4(ONES, ONES, ONES, ONES);
    uint4 T = min4(addw4(F, ONES), add4(M, d));
    T = sel4(d, T, in);
    *reinterpret_cast<uint4*>(RFout + so) = T;
    *reinterpret_cast<uint4*>(sF + vl * R + 8 * q) = F;
    if (drains) {
      const uint32_t f = __ldg(g.sv_off + s), fw[4] = {F.x, F.y, F.z, F.w};
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const uint32_t w = a.word[8 * q + v];
        if (w & SW_DRAIN)
          atomicMin(&sMin[((w & SW_PAR) ? 0 : R) + 8 * q + v],
                    pack_min((int)((fw[v >> 1] >> (16 * (v & 1))) & 0xFFFFu), f));
      }
    }
    // F - 1 never drops below 0 where it matters: T >= 0
    const uint4 Fm = make_uint4(__vsubus2(F.x, ONES), __vsubus2(F.y, ONES), __vsubus2(F.z, ONES), __vsubus2(F.w, ONES));
    const uint4 Tc = max4(T, Fm);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const uint4 gap = sel4(zero, sub4(rf, F), in), low = sel4(zero, sub4(Tc, T), in);
    // change of the first score + 1: 0..2 (row 0: its mismatch + 1)
    const uint4 ch = sel4(add4(d, one), sub4(add4(Tc, one), F), in);
    uint32_t g0, g1, c0, c1, big = 0;
    uint4 gl = gap;
    if ((gap.x | gap.y | gap.z | gap.w) & 0xFFFCFFFCu) {
      big = nonzero8(make_uint4(gap.x & 0xFFFCFFFCu, gap.y & 0xFFFCFFFCu, gap.z & 0xFFFCFFFCu, gap.w & 0xFFFCFFFCu));
      const uint4 b16 = unplane(big);
      const uint4 keepm = make_uint4(b16.x * 0xFFFFu, b16.y * 0xFFFFu, b16.z * 0xFFFFu, b16.w * 0xFFFFu);
      gl = sel4(zero, gap, keepm);
    }
    planes2(gl, g0, g1);
    planes2(ch, c0, c1);
    const uint32_t at = vl * C + q;
    sP[G0][at] = (uint8_t)g0;
    sP[G1][at] = (uint8_t)g1;
    sP[VP][at] = (uint8_t)c1;
    sP[VN][at] = (uint8_t)(~(c0 | c1));
    sP[GBIG][at] = (uint8_t)big;
    sP[LOW][at] = (low.x | low.y | low.z | low.w) ? (uint8_t)nonzero8(low) : (uint8_t)0;
  }
  __syncthreads();
  // ---- pass 2
  {
    const uint32_t vi = threadIdx.x / W, w = threadIdx.x % W;
    if (vi < nv) {
      const uint32_t vl = CHSGA_CHK((uint32_t)__ldg(g.by_len + v0 + vi), nv, 24);
      const uint32_t s = v0 + vl;
      uint32_t f = __ldg(g.sv_off + s), e = __ldg(g.sv_off + s + 1);
      CHSGA_CHK_CHARS(f, e, g.N, 1);
      const uint32_t n = e - f - 1;  // chain chars
      uint2* z = static_cast<uint2*>(a.bits) + (size_t)(f + 1) * W + w;
      auto plane = [&](int p) { return reinterpret_cast<const uint32_t*>(sP[p])[vl * W + w]; };
      uint32_t vp = plane(VP), vn = plane(VN);
      const uint32_t keep = sKeep[w], low = plane(LOW);
      if (n) {
        uint32_t g0 = plane(G0), g1 = plane(G1);
        for (uint32_t big = plane(GBIG); big; big &= big - 1) {
          const uint32_t b = __ffs(big) - 1, r = 32 * w + b;
          line_slot(z, W, n, 1u << b, (uint32_t)RFin[(size_t)s * R + r] - sF[vl * R + r]);
        }
        // label keys, 8 chars a word
        const uint32_t* kp = g.lab4 + ((f + 1) >> 3);
        const uint32_t ks = ((f + 1) & 7u) * 4u;
        uint32_t klo = __ldg(kp);
        constexpr int U = 8;
        for (uint32_t c = 0; c < n; c += U) {
          const uint32_t khi = __ldg(++kp);
          const uint32_t keys = __funnelshift_r(klo, khi, ks);
          klo = khi;
          uint2 x[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c + u < n) x[u] = z[u * W];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (c + u < n) {
              const uint32_t d = sMis[((keys >> (4 * u)) & 7u) * W + w];
              const uint32_t p = x[u].x, m = x[u].y;
              // the previous row under its line (row 0 slots have none)
              const uint32_t t0 = g0 & ~m;
              const uint32_t hp = (p & keep) | g1 | t0;
              const uint32_t hn = m & keep & ~(g1 | g0);
              const uint32_t b = g1 & ~(g0 ^ m);
              g1 &= p | t0;
              g0 = (p & g0) | (~p & b);
              // new score is 1 above the char's left neighbour of the
              // previous row, else level with it
              const uint32_t t = d & ~(vn | hn);
              const uint32_t op = vn | (t & ~vp), om = vp & ~t;
              vp = hn | (t & ~hp);
              vn = hp & ~t;
              z[u * W] = make_uint2(op, om);
            }
          z += U * W;
        }
        z = static_cast<uint2*>(a.bits) + (size_t)(f + 1) * W + w;
        for (uint32_t lb = low; lb; lb &= lb - 1) {
          const uint32_t b = __ffs(lb) - 1, r = 32 * w + b;
          line_slot(z, W, n, 1u << b, (uint32_t)sF[vl * R + r] - 1u - RFout[(size_t)s * R + r]);
        }
        reinterpret_cast<uint32_t*>(sP[VP])[vl * W + w] = vp;
        reinterpret_cast<uint32_t*>(sP[VN])[vl * W + w] = vn;
      }
      if (ends) {
        for (uint32_t eb = sEnd[w]; eb; eb &= eb - 1) {
          const uint32_t b = __ffs(eb) - 1, r = 32 * w + b;
          int cur = RFout[(size_t)s * R + r], bm = cur;
          uint32_t bc = f;
          for (uint32_t c = 0; c < n; ++c) {
            const uint2 x = z[(size_t)c * W];
            cur += (int)((x.x >> b) & 1u) - (int)((x.y >> b) & 1u);
            if (cur < bm) {
              bm = cur;
              bc = f + 1 + c;
            }
          }
          atomicMin(&sMin[((a.word[r] & SW_PAR) ? R : 0) + r], pack_min(bm, bc));
        }
      }
    }
  }
  __syncthreads();
  // ---- pass 3
  for (uint32_t it = threadIdx.x; it < nv * C; it += NT) {
    const uint32_t vl = it / C, q = it % C, s = v0 + vl;
    const uint32_t len = __ldg(&g.rec[s].y) & 0x1FFFFFFFu;
    const size_t so = (size_t)s * R + 8 * q;
    uint4 o;
    if (len == 1) {
      o = *reinterpret_cast<const uint4*>(RFout + so);
    } else {
      const uint32_t lw = min(len - 1, 0xFFFFu) * ONES, at = vl * C + q;
      const uint4 F = *reinterpret_cast<const uint4*>(sF + vl * R + 8 * q);
      o = min4(__ldg(reinterpret_cast<const uint4*>(RLin + so)), addw4(F, lw));
      o = sel4(make_uint4(0, 0, 0, 0), o, sInit[q]);
      const uint4 p = unplane(sP[VP][at]), m = unplane(sP[VN][at]);
      o = make_uint4(o.x + p.x - m.x, o.y + p.y - m.y, o.z + p.z - m.z, o.w + p.w - m.w);
      if (sP[LOW][at]) o = min4(o, addw4(*reinterpret_cast<const uint4*>(RFout + so), lw));
    }
    *reinterpret_cast<uint4*>(RLout + so) = o;
  }
  if (ends) {
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * R; i += NT)
      if (sMin[i] != ~0ull) atomicMin(a.best + i, sMin[i]);
  }
  bits_finish<R>(a, gridDim.x);
}

}  // namespace dev
}  // namespace chsga
