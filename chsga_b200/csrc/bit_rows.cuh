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
// another, so the row-step has no phases between blocks; every block moves
// the slots on for itself at its start (bits_head).
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

constexpr uint32_t SW_DRAIN = 1u << 13;     // the slot's previous read takes its closure minimum
constexpr uint32_t SW_PAR_SHIFT = 14;       // bits 14..15: which of the slot's four minima its read uses
constexpr uint32_t kBitsNarrowMax = 32767;  // longest read whose sums need no saturation

struct BitGraph {  // closure.hpp, k_closure_arrays
  uint32_t S, N, n_ent, n_went, heavy;
  uint64_t words;
  const uint4* rec;
  const uint2* ent16;
  const uint8_t* by_len;  // of the kernel's window
  const uint32_t* sv_off;
  const uint32_t* lab4;
  const uint32_t* pos;
  const uint2* wsv;
  const uint4* wrec;
  const uint2* went;
  const uint4* lab;
};

// Where a slot's previous and current rows lie in its read's matrix
// (traceback): {bits, RF, F} of a row, row_bits_layout.
struct SlotRows {
  unsigned char* prev;
  unsigned char* cur;
};

// The slots before a row-step; every launch reads one and writes the other.
// SlotState::pad: (id of the draining read + 1) << 2 | minimum of the slot.
struct BitState {
  SlotState s[128];
  SlotRows rows[128];  // traceback
  uint32_t next[128];  // the slot's read base after the row's, when there is one
  uint32_t q_head, pad[3];
};

struct BitArgs {
  BitGraph g;
  const void *RFin, *RLin;
  void *RFout, *RLout;
  void* bits;  // uint2 words (one read a word) or bit-sliced char words
  const BitState* st_in;
  BitState* st_out;
  unsigned long long* best;  // [4][R]
  StepCtl* ctl;
  const ReadDesc* queue;
  const unsigned char* reads;
  int32_t* res_score;
  uint32_t* res_vertex;
  unsigned long long *res_t0, *res_t1;
  CompletionRec* done_ring;
  uint32_t qmask;
  int special, match_n;
  unsigned char* const* mats;  // traceback: matrix of every read id
  size_t pitch;
};

// ---------------------------------------------------------------------------
// k_closure_arrays, k_by_len: the arrays of the bit-row kernels from the lists
// of build_closure, once a graph is loaded (they took a third of the list
// build's time on the host and twice the bytes to upload).
//   ent    in {source, weight}; out for 16-bit rows: {source, weight for M |
//          weight for F << 16}, 0xFFFF = no such entry (or a weight no 16-bit
//          score can win with)
//   wrec   in HostClosure::order; out {first bit word, length | key << 29,
//          first entry, entries}
//   wsv    {string vertex, first char} by position; pos the position by vertex
//   went   {source | class << 30 (0 both, 1 M only, 2 F only), weight}
//   lab    per bit word the label planes of its 32 chain chars (bit k of word j
//          = char first + 1 + 32 j + k): {code bit 0, code bit 1, special, 0}
// Eight lanes a position.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_closure_arrays(uint32_t S, uint32_t heavy, const uint4* __restrict__ rec,
                                                        uint2* ent, uint4* wrec, uint2* wsv, uint32_t* pos,
                                                        uint2* went, uint4* lab, const uint32_t* __restrict__ lab4) {
  const uint64_t t = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  const uint32_t i = (uint32_t)(t / 8), l = (uint32_t)(t % 8);
  const bool live = i < S;
  const uint4 in = live ? wrec[i] : make_uint4(0, 0, 0, 0);
  __syncwarp();  // all lanes of a position have read its record
  if (!live) return;
  const uint4 r = rec[in.y];
  const uint32_t nb = r.w & 255u, nm = (r.w >> 8) & 255u, n = nb + nm + (r.w >> 16), len = r.y & 0x1FFFFFFFu;
  if (l == 0) {
    wrec[i] = make_uint4(in.x, r.y, in.z, n);
    wsv[i] = make_uint2(in.y, r.x);
    pos[in.y] = i;
  }
  for (uint32_t k = l; k < n; k += 8) {
    const uint2 e = ent[r.z + k];
    const uint32_t cls = k < nb ? 0u : k < nb + nm ? 1u : 2u, w = min(e.y, 0xFFFEu);
    went[in.z + (size_t)(i < heavy ? 1 : 32) * k] = make_uint2(e.x | cls << 30, e.y);
    ent[r.z + k] = make_uint2(e.x, (cls == 2 ? 0xFFFFu : w) | (cls == 0 ? w + 1 : cls == 2 ? w : 0xFFFFu) << 16);
  }
  for (uint32_t j = l; j < (len + 30) / 32; j += 8) {
    const uint32_t c0 = r.x + 1 + 32 * j, m = min(32u, len - 1 - 32 * j);
    uint4 p = make_uint4(0, 0, 0, 0);
    for (uint32_t k = 0; k < m; ++k) {
      const uint32_t key = lab4[(c0 + k) >> 3] >> ((c0 + k) & 7u) * 4u;
      p.x |= (key & 1u) << k;
      p.y |= ((key >> 1) & 1u) << k;
      p.z |= ((key >> 2) & 1u) << k;
    }
    lab[in.x + j] = p;
  }
}

// Order of the vertices inside every window of 32, 64 and 128 by falling label
// length (local indexes), ties in their order: a thread counts the vertices
// before its own. Blocks of 128 threads.
__global__ void __launch_bounds__(128) k_by_len(uint32_t S, const uint32_t* __restrict__ sv_off, uint8_t* by32,
                                                uint8_t* by64, uint8_t* by128) {
  __shared__ uint32_t s_len[128];
  const uint32_t t = threadIdx.x, base = blockIdx.x * 128, s = base + t;
  const uint32_t len = s < S ? sv_off[s + 1] - sv_off[s] : 0;  // none has length 0: past the end goes last
  s_len[t] = len;
  __syncthreads();
  if (s >= S) return;
  auto place = [&](uint32_t W, uint8_t* out) {
    const uint32_t w0 = t / W * W;
    uint32_t r = 0;
    for (uint32_t u = w0; u < w0 + W; ++u) r += s_len[u] > len || (s_len[u] == len && u < t) ? 1u : 0u;
    out[base + w0 + r] = (uint8_t)(t - w0);
  };
  place(32, by32);
  place(64, by64);
  place(128, by128);
}

// What a row-step has to do, the same in every block.
struct HeadFlags {
  bool work, end, drain, init, wide;
};

// Moves the slots to the row-step about to run. Every block does it for
// itself from the state the launch before left (a few hundred bytes), so no
// block waits for one that advances the slots after all others are done;
// block 0 also finishes the reads that drained, writes the new state and
// counts the step. Admission is by slot order from the queue's head, so the
// blocks agree. word: the slots' words (shared memory, R entries); rows: the
// slots' row pointers (traceback, else null).
//
// A read's minimum is reset when it is read out, by block 0 of the step
// after its drain, while other blocks may already take minima of the slot's
// next but one read: with four minima a slot that is another one.
template <int R>
__device__ __forceinline__ HeadFlags bits_head(const BitArgs& a, uint32_t* word, SlotRows* rows) {
  static_assert(R <= 128, "one thread per slot");
  __shared__ uint32_t s_cnt[4], s_flag[4];
  const int r = threadIdx.x, lane = r & 31, wp = r >> 5;
  constexpr int NW = R < 32 ? 1 : R / 32;
  const bool first = blockIdx.x == 0 && blockIdx.y == 0;
  SlotState st{};
  SlotRows sr{nullptr, nullptr};
  bool need = false, wide = false;
  uint32_t drain = 0, par = 0, q_head = 0, avail = 0, byte = 0;
  unsigned before = 0;
  if (wp < NW) {
    if (r < R) {
      st = a.st_in->s[r];
      byte = a.st_in->next[r];
      q_head = a.st_in->q_head;
      avail = a.ctl->q_count - q_head;
      par = st.pad & 3u;
      if (a.mats) {
        sr = a.st_in->rows[r];
        sr.prev = sr.cur;
      }
      const int32_t did = (int32_t)(st.pad >> 2) - 1;
      if (did >= 0 && first) {
        unsigned long long* bp = a.best + ((par + 3u) & 3u) * R + r;
        const unsigned long long b = __ldcg(bp), t1 = global_ns();
        *bp = ~0ull;
        a.res_score[did] = (int32_t)(b >> 32);
        a.res_vertex[did] = (uint32_t)(b & 0xffffffffu);
        a.res_t1[did] = t1;
        const uint32_t k = atomicAdd(&a.ctl->done, 1u);
        if (a.done_ring)
          a.done_ring[k & a.qmask] = CompletionRec{did, (int32_t)(b >> 32), (uint32_t)(b & 0xffffffffu), 0u,
                                                   a.res_t0[did], t1};
      }
      wide = st.id >= 0 && st.len > kBitsNarrowMax;  // also while it drains
      if (st.id >= 0) {
        if (st.row + 1 >= st.len) {
          drain = (uint32_t)st.id + 1;
          st.id = -1;
          par = (par + 1u) & 3u;
        } else {
          st.row += 1;
        }
      }
      need = st.id < 0;
    }
    const unsigned nb = __ballot_sync(0xFFFFFFFFu, need);
    before = __popc(nb & ((1u << lane) - 1u));
    if (lane == 0) s_cnt[wp] = __popc(nb);
  }
  if constexpr (NW > 1)
    __syncthreads();
  else
    __syncwarp();
  if (wp < NW) {
    uint32_t total = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      if (i < wp) before += s_cnt[i];
      total += s_cnt[i];
    }
    uint32_t w = 0;
    if (r < R) {
      if (need && before < avail) {
        const ReadDesc q = a.queue[(q_head + before) & a.qmask];
        st.off = q.off;
        st.len = q.len;
        st.row = 0;
        st.id = q.id;
        byte = a.reads[q.off];
        if (first) a.res_t0[q.id] = global_ns();
      }
      if (st.id >= 0) {
        w = base_code((int)byte, a.special) | (mismatch_mask((int)byte, a.special, a.match_n) << SW_MASK_SHIFT) |
            SW_ACTIVE;
        w |= st.row == 0 ? SW_INIT : SW_CLOSURE;
        if (st.row + 1 == st.len) w |= SW_ENDING;
        if (a.mats) sr.cur = a.mats[st.id] + (size_t)st.row * a.pitch;
      }
      if (drain) w |= SW_DRAIN;
      w |= par << SW_PAR_SHIFT;
      word[r] = w;
      if (rows) rows[r] = sr;
      if (first) {
        st.pad = drain << 2 | par;
        a.st_out->s[r] = st;
        // fetched here, where nothing waits for it, the base is part of the
        // state the next launch starts from
        if (st.id >= 0 && st.row + 1 < st.len) a.st_out->next[r] = a.reads[st.off + st.row + 1];
        if (a.mats) a.st_out->rows[r] = sr;
        if (r == 0) a.st_out->q_head = q_head + (total < avail ? total : avail);
      }
    }
    const bool act = (w & SW_ACTIVE) != 0;
    const uint32_t f = (__any_sync(0xFFFFFFFFu, (w & (SW_ACTIVE | SW_DRAIN)) != 0) ? 1u : 0u) |
                       (__any_sync(0xFFFFFFFFu, (w & SW_ENDING) != 0) ? 2u : 0u) |
                       (__any_sync(0xFFFFFFFFu, (w & SW_DRAIN) != 0) ? 4u : 0u) |
                       (__any_sync(0xFFFFFFFFu, r < R && (!act || (w & SW_INIT))) ? 8u : 0u) |
                       (__any_sync(0xFFFFFFFFu, wide) ? 16u : 0u);
    if (lane == 0) s_flag[wp] = f;
  }
  __syncthreads();
  uint32_t f = 0;
#pragma unroll
  for (int i = 0; i < NW; ++i) f |= s_flag[i];
  if (first && threadIdx.x == 0 && (f & 1u)) a.ctl->steps += 1;
  return HeadFlags{(f & 1u) != 0, (f & 2u) != 0, (f & 4u) != 0, (f & 8u) != 0, (f & 16u) != 0};
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
// What bounds it: at one slot the chain of dependent loads of a vertex (state
// of the launch before, record and entries, gathers, stores) on a small graph
// (5.4 us a row-step at 100 kbp, of which about 3 us are launch and state), and
// the number of loads in flight on a large one (17.5 us at 5 Mbp; the level
// sweeps and their row kernel took 24.6 and 85 us in 12 and 18 launches). The
// longest lists set the chain: four dependent rounds less for lists of up to
// 60 entries took the 5 Mbp graph from 21.8 to 17.5 us.
//
// k_row_words: one thread per (string vertex, slot), a vertex's chain in
// words of 32 chars. Slots are interleaved (RF[s * R + r], word w of slot r at
// w * R + r), so the gathers of neighbouring slots share sectors; with MAT
// every slot is blockIdx.y of a one-slot launch with rows in its read's
// matrix. Vertices are in the order of closure.hpp (windows by list length),
// so a warp's lists end together and its loads of records, entries, labels
// and bits lie side by side.
// ---------------------------------------------------------------------------
#ifndef CHSGA_WORDS_THREADS
#define CHSGA_WORDS_THREADS 1024  // threads per SM the register budget is sized for (build-time tuning)
#endif
// P = lanes that share a long list (for every slot).
template <int R, typename ST, int H, int NT, int P>
__global__ void __launch_bounds__(NT, CHSGA_WORDS_THREADS / NT) k_row_words(BitArgs a) {
  constexpr bool MAT = H > 0;
  constexpr int SLOTS = MAT ? H : R;
  static_assert(!MAT || (R == 1 && sizeof(ST) == 2), "matrix rows hold one slot each, 16 bits");
  static_assert(NT >= (SLOTS < 32 ? 32 : SLOTS), "the head needs a thread per slot");
  static_assert(P == 1 || R * P <= 32, "a list's lanes lie in one warp");
  using bits::PN;
  constexpr int VB = NT / R;  // vertices per block and turn
  const BitGraph& g = a.g;
  __shared__ uint32_t s_word[SLOTS];
  __shared__ SlotRows s_rows[MAT ? SLOTS : 1];
  __shared__ unsigned long long s_min[4 * R];
  const int r = (int)(threadIdx.x % R);  // of this block's slots
  constexpr int U = R == 1 ? 8 : 4;  // entries and gathers in flight: a short list in one go
  // items: P parts of every long list, rounded up to whole blocks, then the
  // vertices with short lists
  const uint32_t hparts = (g.heavy * P + VB - 1) / VB * VB, items = hparts + (g.S - g.heavy);
  uint32_t i = 0, part = 0, n = 0, stride = 32;  // position of the vertex; this lane's entries
  uint2 sv = make_uint2(0, 0);                   // the vertex, its first char
  bool mine = false;
  uint4 rec = make_uint4(0, 1, 0, 0);
  uint2 e[U];
  auto entries = [&](uint32_t k) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u < n) e[u] = __ldg(g.went + CHSGA_CHK(rec.z + part + stride * (k + u), g.n_went, 21));
  };
  auto fetch = [&](uint32_t item) {
    const bool long_list = item < hparts;
    i = long_list ? item / P : item - hparts + g.heavy;
    part = long_list ? item % P : 0;
    mine = item < items && (!long_list || i < g.heavy);
    n = 0;
    if (mine) {
      rec = __ldg(g.wrec + i);
      sv = __ldg(g.wsv + i);
      sv.x = CHSGA_CHK(sv.x, g.S, 20);
      stride = long_list ? P : 32;
      n = long_list ? (rec.w > part ? (rec.w - part + P - 1) / P : 0) : rec.w;
      entries(0);
    }
  };
  fetch(blockIdx.x * VB + threadIdx.x / R);
  pdl_wait();
  for (int k = threadIdx.x; k < 4 * R; k += NT) s_min[k] = ~0ull;
  const HeadFlags hf = bits_head<SLOTS>(a, s_word, MAT ? s_rows : nullptr);
  if (!hf.work) return;
  if (hf.drain) {
    // a draining read's raw minimum is known: only scores that reach it count
    if (threadIdx.x < R) {
      const uint32_t q = MAT ? blockIdx.y : threadIdx.x, p = ((s_word[q] >> SW_PAR_SHIFT) + 3u) & 3u;
      if (s_word[q] & SW_DRAIN) s_min[p * R + threadIdx.x] = __ldcg(a.best + p * SLOTS + q);
    }
    __syncthreads();
  }
  const uint32_t w = s_word[MAT ? blockIdx.y : r];
  const bool init = (w & SW_INIT) != 0;
  const uint32_t par = (w >> SW_PAR_SHIFT) & 3u;
  const ST *RFin, *RLin;
  ST *RFout, *RLout, *Fout = nullptr;
  const uint2* win;
  uint2* wout;
  if constexpr (MAT) {
    const SlotRows sr = s_rows[blockIdx.y];
    const size_t rf = bits_row_rf(g.words);
    RFin = reinterpret_cast<const ST*>(sr.prev + rf);
    RFout = reinterpret_cast<ST*>(sr.cur + rf);
    Fout = reinterpret_cast<ST*>(sr.prev + bits_row_f(g.words, g.S));
    win = reinterpret_cast<const uint2*>(sr.prev);
    wout = reinterpret_cast<uint2*>(sr.cur);
    RLin = static_cast<const ST*>(a.RLin) + (size_t)blockIdx.y * g.S;
    RLout = static_cast<ST*>(a.RLout) + (size_t)blockIdx.y * g.S;
  } else {
    RFin = static_cast<const ST*>(a.RFin) + r;
    RLin = static_cast<const ST*>(a.RLin) + r;
    RFout = static_cast<ST*>(a.RFout) + r;
    RLout = static_cast<ST*>(a.RLout) + r;
    win = static_cast<const uint2*>(a.bits) + r;
    wout = static_cast<uint2*>(a.bits) + r;
  }
  const uint32_t mask = (w >> SW_MASK_SHIFT) & SW_MASK;
  // turn t of block b: group (b + t) mod n of the turn's n groups (a window's
  // groups go from long to short lists)
  uint32_t gb = blockIdx.x;
  for (uint32_t turn0 = 0; turn0 < items && (w & (SW_ACTIVE | SW_DRAIN)); turn0 += gridDim.x * VB) {
    if (turn0) {
      gb = gb + 1 < gridDim.x ? gb + 1 : 0;
      fetch(turn0 + gb * VB + threadIdx.x / R);
    }
    const bool long_list = turn0 + gb * VB < hparts;  // the same for the whole block
    if (!long_list && !mine) continue;
    const uint32_t len = rec.y & 0x1FFFFFFFu, key = rec.y >> 29;
    const uint32_t nw = (len + 30) / 32;
    const int delta = (int)((mask >> key) & 1u);
    // the first word's labels and bits load beside the gathers
    uint4 lb = make_uint4(0, 0, 0, 0);
    uint2 old = make_uint2(0, 0);
    if (mine && part == 0 && nw) {
      const size_t wi = (size_t)CHSGA_CHK(rec.x, g.words, 23);
      lb = __ldg(g.lab + wi);
      if (!init) old = win[wi * R];
    }
    // closure of the previous row (a no-op on row 0: its scores are 0 and 1
    // and every weight is at least 1)
    int rf = 0, F = 0, M = 0x3fffffff, dl = 0;
    if (!init || (w & SW_DRAIN)) {
      if (mine) {
        rf = (int)__ldg(RFin + (size_t)sv.x * R);
        dl = (int)__ldg(RLin + (size_t)sv.x * R);
      }
      F = rf;
      for (uint32_t k = 0; k < n; k += U) {
        if (k) entries(k);
        int x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < n) x[u] = (int)__ldg(RLin + (size_t)CHSGA_CHK(e[u].x & 0x3FFFFFFFu, g.S, 22) * R) + (int)e[u].y;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < n) {
            const uint32_t cls = e[u].x >> 30;  // 0 both, 1 M only, 2 F only
            if (cls != 2) M = min(M, x[u]);
            if (cls != 1) F = min(F, x[u] + (cls ? 0 : 1));
          }
      }
      if (P > 1 && long_list) {
        // a list's lanes for one slot lie R apart and take the same way here
        // (other slots' lanes may not)
        const uint32_t lane = threadIdx.x & 31u;
        unsigned lanes = 0;
#pragma unroll
        for (int p = 0; p < P; ++p) lanes |= 1u << (p * R);
        lanes <<= lane / (R * P) * (R * P) + lane % R;
#pragma unroll
        for (int o = R; o < R * P; o <<= 1) {
          F = min(F, __shfl_xor_sync(lanes, F, o));
          M = min(M, __shfl_xor_sync(lanes, M, o));
        }
      }
      if (!mine || part) continue;
      if constexpr (MAT) Fout[sv.x] = (ST)F;
      if (w & SW_DRAIN) {
        const unsigned long long b = pack_min(F, sv.y);
        if (b < s_min[((par + 3u) & 3u) * R + r]) atomicMin(&s_min[((par + 3u) & 3u) * R + r], b);
      }
    }
    if ((w & SW_ACTIVE) && mine && part == 0) {
      int T, last;
      if (init) {
        T = delta;
        uint32_t left = (uint32_t)delta;
        for (uint32_t j = 0; j < nw; ++j) {
          const size_t wi = (size_t)CHSGA_CHK(rec.x + j, g.words, 23);
          if (j) lb = __ldg(g.lab + wi);
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
          if (j) {
            lb = __ldg(g.lab + wi);
            old = win[wi * R];
          }
          const uint32_t top = min(31u, len - 2 - 32 * j), valid = 0xFFFFFFFFu >> (31 - top);
          PN x = bits::under_line(PN{old.x, old.y}, valid, gap);
          x = bits::step(x, bits::mismatch_word(lb.x, lb.y, lb.z, mask), h, top);
          x = bits::under_line(x, valid, low);
          wout[wi * R] = make_uint2(x.p, x.n);
        }
        last = len > 1 ? min(min(dl, F + (int)(len - 1)) + h, T + (int)(len - 1)) : T;
      }
      RFout[(size_t)sv.x * R] = (ST)T;
      RLout[(size_t)sv.x * R] = (ST)last;
      // the raw row's minimum and its first char; a chain falls by at most
      // one a char, so most vertices cannot reach the block's best so far
      // (which other warps lower meanwhile: an old value only prunes less)
      if ((w & SW_ENDING) &&
          max(T - (int)(len - 1), 0) <= (int)min(s_min[par * R + r] >> 32, 0x7FFFFFFFull)) {
        const uint32_t f = sv.y;
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
        atomicMin(&s_min[par * R + r], pack_min(bm, bc));
      }
    }
  }
  if (hf.end || hf.drain) {
    __syncthreads();
    for (int k = threadIdx.x; k < 4 * R; k += NT)
      if (s_min[k] != ~0ull) atomicMin(a.best + (MAT ? k * SLOTS + (int)blockIdx.y : k), s_min[k]);
  }
}

// ---------------------------------------------------------------------------
// k_close_row: the final row (after its closure) of a row-step state, as the
// 32-bit scores of every char: one thread per string vertex (checkpoint
// files).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_close_row(BitGraph g, const uint2* __restrict__ bits,
                                                   const uint16_t* __restrict__ RF,
                                                   const uint16_t* __restrict__ RL, int* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.S) return;
  const uint4 rec = __ldg(g.wrec + i);
  const uint2 sv = __ldg(g.wsv + i);
  int F = RF[sv.x], cur = F;
  for (uint32_t k = 0; k < rec.w; ++k) {
    const uint2 e = __ldg(g.went + rec.z + (i < g.heavy ? 1 : 32) * k);
    if (e.x >> 30 != 1) F = min(F, (int)RL[e.x & 0x3FFFFFFFu] + (int)e.y + (e.x >> 30 ? 0 : 1));
  }
  const uint32_t f = sv.y, len = rec.y & 0x1FFFFFFFu;
  out[f] = F;
  for (uint32_t k = 0; k + 1 < len; ++k) {
    const uint2 x = bits[rec.x + (k >> 5)];
    cur += (int)((x.x >> (k & 31u)) & 1u) - (int)((x.y >> (k & 31u)) & 1u);
    out[f + 1 + k] = min(cur, F + (int)(k + 1));
  }
}

// ---------------------------------------------------------------------------
// k_walk_bits: k_walk over a matrix of bit rows (row i at M + (i - row_lo) *
// pitch), one warp. The path stays in a vertex for about as many rows as the
// vertex has chars, so on entering one every lane loads that vertex's words
// of one row (31 rows ahead) and the steps inside it only shuffle; at a first
// char every lane takes one in-edge. One thread reading the rows one after
// another pays a memory round trip a row. Same tie order as k_walk.
// ---------------------------------------------------------------------------
struct BitRowView {
  const unsigned char* M;
  size_t pitch, rf, f;
  __device__ __forceinline__ int first_raw(long long i, uint32_t s) const {
    return reinterpret_cast<const uint16_t*>(M + (size_t)i * pitch + rf)[s];
  }
  __device__ __forceinline__ int first_final(long long i, uint32_t s) const {
    return reinterpret_cast<const uint16_t*>(M + (size_t)i * pitch + f)[s];
  }
  __device__ __forceinline__ uint2 word(long long i, uint32_t w) const {
    return reinterpret_cast<const uint2*>(M + (size_t)i * pitch)[w];
  }
  // final score of char k of vertex s, its words from wo on
  __device__ __forceinline__ int score(long long i, uint32_t s, uint32_t wo, uint32_t k) const {
    int cur = first_raw(i, s);
    const int F = first_final(i, s);
    for (uint32_t j = 0; 32 * j < k; ++j) {
      const uint2 x = word(i, wo + j);
      const uint32_t m = k - 32 * j >= 32 ? 0xFFFFFFFFu : (1u << (k - 32 * j)) - 1u;
      cur += __popc(x.x & m) - __popc(x.y & m);
    }
    return min(cur, F + (int)k);
  }
};

// One walk: rows [row_lo, row_hi] of the matrix at M, from char `start`.
struct WalkJob {
  const unsigned char* M;
  const unsigned char* read;
  long long row_lo, row_hi;
  uint32_t start, pad;
};

// Block j takes jobs[j] (null: the one job given by value) and writes out[j]
// and at most max_ops ops from ops + j * max_ops on. A walk is a chain of
// round trips, so the reads that finish together walk together.
__global__ void __launch_bounds__(32) k_walk_bits(GraphPtrs g, BitGraph bg, size_t pitch,
                                                  const WalkJob* __restrict__ jobs, WalkJob one,
                                                  WalkOp* __restrict__ ops, uint32_t max_ops,
                                                  WalkOut* __restrict__ out, int match_n) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  const WalkJob job = jobs ? jobs[blockIdx.x] : one;
  const unsigned char* const M = job.M;
  const unsigned char* const read = job.read;
  const long long row_lo = job.row_lo, row_hi = job.row_hi;
  const uint32_t start = job.start;
  ops += (size_t)blockIdx.x * max_ops;
  out += blockIdx.x;
  const int lane = threadIdx.x;
  const BitRowView v{M, pitch, bits_row_rf(bg.words), bits_row_f(bg.words, bg.S)};
  uint32_t lo = 0, hi = g.S;
  while (hi - lo > 1) {
    const uint32_t m = (lo + hi) / 2;
    if (g.sv_off[m] <= start) lo = m; else hi = m;
  }
  uint32_t sv = lo, n = 0;
  long long row = row_hi;
  int status = 0, fail_row = 0;
  uint32_t first = g.sv_off[sv], k = start - first;  // char k of vertex sv
  uint32_t wo = bg.wrec[bg.pos[sv]].x;  // first word
  // lane j: vertex sv in row held - j (its first word, enough up to char 32)
  long long held = -1;
  int h_rf = 0, h_f = 0;
  uint2 h_w = make_uint2(0, 0);
  uint32_t h_key = 0, h_byte = 0;
  auto hold = [&] {
    held = row;
    const long long i = row - lane;
    if (i >= row_lo) {
      h_rf = v.first_raw(i - row_lo, sv);
      h_f = v.first_final(i - row_lo, sv);
      if (k > 0) h_w = v.word(i - row_lo, wo);
      h_byte = read[i];
    }
    // label keys of the chars k, k - 1, ... of the vertex
    h_key = (uint32_t)lane <= k ? label_key(g, first + k - (uint32_t)lane) : 0u;
  };
  uint32_t held_k = 0;
  auto at = [&](long long i, uint32_t kk) -> int {  // final score of char kk in row i (held or held - 1 .. - 31)
    if (kk > 32) return v.score(i - row_lo, sv, wo, kk);
    const int j = (int)(held - i);
    const int rf = __shfl_sync(FULL, h_rf, j), f = __shfl_sync(FULL, h_f, j);
    const uint32_t p = __shfl_sync(FULL, h_w.x, j), m = __shfl_sync(FULL, h_w.y, j);
    const uint32_t mask = kk >= 32 ? 0xFFFFFFFFu : (1u << kk) - 1u;
    return min(rf + __popc(p & mask) - __popc(m & mask), f + (int)kk);
  };
  hold();
  held_k = k;
  int s = at(row, k);
  while (row > row_lo) {
    if (n >= max_ops) {
      status = 8;
      fail_row = (int)row;
      break;
    }
    if (held - row >= 31 || held_k - k >= 31) {
      hold();
      held_k = k;
    }
    uint32_t op = 255, src_sv = sv, src_k = k;
    int src_s = 0;
    // scores of up to 32 in-neighbours' last chars in row i: the first (in
    // list order) with value + add == s
    auto from_edges = [&](const uint32_t* list, uint32_t e0, uint32_t e1, long long i, int add, bool& found) {
      for (uint32_t b = e0; b < e1 && !found; b += 32) {
        uint32_t u = 0, kl = 0;
        int x = 0x3fffffff;
        if (b + lane < e1) {
          u = list[b + lane];
          const uint4 rec = bg.wrec[bg.pos[u]];
          kl = (rec.y & 0x1FFFFFFFu) - 1;
          x = v.score(i - row_lo, u, rec.x, kl);
        }
        const unsigned hit = __ballot_sync(FULL, x + add == s);
        if (hit) {
          const int l = __ffs(hit) - 1;
          src_sv = __shfl_sync(FULL, u, l);
          src_k = __shfl_sync(FULL, kl, l);
          src_s = __shfl_sync(FULL, x, l);
          found = true;
        }
      }
    };
    bool found = false;
    if (k > 0) {
      const int x = at(row, k - 1);
      if (x + 1 == s) {
        op = 2;
        src_k = k - 1;
        src_s = x;
      }
    } else {
      from_edges(g.istr_src, g.istr_off[sv], g.istr_off[sv + 1], row, 1, found);
      if (found) op = 2;
    }
    if (op == 255) {
      const int x = at(row - 1, k);
      if (x + 1 == s) {
        op = 0;
        src_s = x;
      }
    }
    if (op == 255) {
      const uint32_t key = __shfl_sync(FULL, h_key, (int)(held_k - k));
      const int byte = (int)__shfl_sync(FULL, h_byte, (int)(held - row));
      const int delta = (int)((mismatch_mask(byte, g.special, match_n) >> key) & 1u);
      if (k > 0) {
        const int x = at(row - 1, k - 1);
        if (x + delta == s) {
          op = 1;
          src_k = k - 1;
          src_s = x;
        }
      } else {
        from_edges(g.vin_srcv, g.vin_off[sv], g.vin_off[sv + 1], row - 1, delta, found);
        if (found) op = 1;
      }
    }
    if (op == 255) {
      status = 7;
      fail_row = (int)row;
      break;
    }
    if (lane == 0) ops[n] = WalkOp{row, first + k, op};
    ++n;
    if (op != 2) --row;
    s = src_s;
    k = src_k;
    if (src_sv != sv || found) {  // an in-edge may lead back to the same vertex (cycles)
      sv = src_sv;
      first = g.sv_off[sv];
      wo = bg.wrec[bg.pos[sv]].x;
      if (row > row_lo) hold();
      held_k = k;
    }
  }
  if (lane == 0) *out = WalkOut{first + k, n, status, fail_row};
}

// ---------------------------------------------------------------------------
// k_row_sliced: 32 to 128 slots, 16-bit scores, bits sliced over the slots:
// word pair {P, N} g of char c (slots 32g .. 32g+31) at c * R/32 + g. Each
// char of 32 slots is a handful of logic operations, where the packed 16-bit
// update spends tens of instructions.
//
// What bounds it: load latency at the 32 warps an SM that 64 registers allow.
// 5 Mbp graph, 128 slots, 305 us a row-step (the sweeps' chain: 771). On the
// 2 Mbp graph ncu counts 145 us, 0.35 GB from and to HBM (54 us at the copy
// peak), 62 M warp-instructions (54 us of issue) and 9.2 of 15.3 cycles between
// a warp's instructions waiting for loads. At 5 Mbp it takes 100 us less
// without the gathers, 150 without the chain. Blocks of 128 threads with barriers
// between the passes took 353, five or six gathers in flight 316-357 (spills
// past 64 registers), prefetches to L2 or shared memory 374-440.
//
// A warp takes a group of vertices in three passes:
//   1  lane = (vertex, 8 slots): closure and first char in 16-bit pairs; the
//      gap RF - F, the change T - F and rare cases leave as bytes
//   2  lane = (vertex, 32 slots): the chain
//   3  lane = (vertex, 8 slots): last scores
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
__device__ __forceinline__ void line_slot(uint2* p, int W, uint32_t n, uint32_t bit, uint32_t gap) {
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

#ifndef CHSGA_SLICED_WARPS
#define CHSGA_SLICED_WARPS 32  // warps per SM the register budget is sized for (build-time tuning)
#endif
#ifndef CHSGA_SLICED_U
#define CHSGA_SLICED_U 3  // gathers in flight (build-time tuning)
#endif
constexpr int kSlicedThreads = 128;

__device__ __forceinline__ uint4 viaddmin4(const uint4& a, uint32_t w, const uint4& c) {  // min(a + w, c), no half wraps
  return make_uint4(__viaddmin_u16x2(a.x, w, c.x), __viaddmin_u16x2(a.y, w, c.y), __viaddmin_u16x2(a.z, w, c.z),
                    __viaddmin_u16x2(a.w, w, c.w));
}
enum { G0, G1, VP, VN, GBIG, LOW, ENDC, NPL };

// Shared memory of a k_row_sliced block. Every warp works for itself on VB
// vertices at a time: K (vertex, 8 slots) items a lane.
template <int R, int K>
struct SlicedShared {
  static constexpr int C = R / 8, W = R / 32, NT = kSlicedThreads, NW = NT / 32, VB = K * 32 / C;
  uint16_t F[NW][VB * R];
  uint16_t mis16[5][R];
  uint16_t init[R];
  uint16_t lim[2][R];  // scores to reach: last row, drain
  unsigned long long best[2][R];
  uint8_t P[NW][NPL][VB * C];
  uint32_t mis[8 * W], keep[W], end[W], drain[W], word[R];
};

// bit j of the result: value j of x (8 slots) is at most that of y
__device__ __forceinline__ uint32_t at_most8(const uint4& x, const uint4& y) {
  const uint4 m = min4(x, y);
  return ~nonzero8(make_uint4(x.x ^ m.x, x.y ^ m.y, x.z ^ m.z, x.w ^ m.w)) & 0xFFu;
}

// The vertices of one warp. WIDE: some read is so long that a sum of a score
// and a weight may leave 16 bits (saturating sums).
template <int R, int K, bool WIDE>
__device__ __forceinline__ void sliced_warp(const BitArgs& a, const HeadFlags& hf, SlicedShared<R, K>& sh) {
  using Shared = SlicedShared<R, K>;
  constexpr int C = Shared::C, W = Shared::W, NW = Shared::NW, VB = Shared::VB;
  constexpr uint32_t ONES = 0x00010001u;
  const BitGraph& g = a.g;
  const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  uint16_t* const sF = sh.F[wp];
  uint8_t(*const sP)[VB * C] = sh.P[wp];
  const uint16_t* RFin = static_cast<const uint16_t*>(a.RFin);
  const uint16_t* RLin = static_cast<const uint16_t*>(a.RLin);
  uint16_t* RFout = static_cast<uint16_t*>(a.RFout);
  uint16_t* RLout = static_cast<uint16_t*>(a.RLout);
  const uint4 zero = make_uint4(0, 0, 0, 0), one = make_uint4(ONES, ONES, ONES, ONES);
  // A block's warps share a window of NW * VB consecutive vertices (their
  // lists and in-edges mostly stay near, so the warps meet in L1) and take
  // its groups by label length, another one each turn.
  constexpr uint32_t WIN = NW * VB;
  uint32_t turn = 0;
  for (uint32_t w0 = blockIdx.x * WIN; w0 < g.S; w0 += gridDim.x * WIN, ++turn) {
    const uint32_t v0 = w0 + ((wp + turn) % NW) * VB;
    if (v0 >= g.S) continue;
    // lane v holds vertex v of the warp's group
    const uint32_t nv = min((uint32_t)VB, g.S - v0);
    uint32_t my_s = 0;
    if (lane < nv) my_s = K == 4 ? CHSGA_CHK(w0 + __ldg(g.by_len + v0 + lane), g.S, 24) : v0 + lane;
    // ---- pass 1
    constexpr int U = CHSGA_SLICED_U;  // gathers in flight
#pragma unroll 1
    for (int j = 0; j < K; ++j) {
      const uint32_t it = lane + 32 * j, vl = it / C, q = it % C;
      const uint32_t s = __shfl_sync(0xFFFFFFFFu, my_s, vl);
      if (vl >= nv) continue;
      const uint4 rec = __ldg(g.rec + s);
      const uint32_t ry = rec.y;
      uint32_t k0 = rec.z, k1 = k0 + (rec.w & 0xFFu) + ((rec.w >> 8) & 0xFFu) + ((rec.w >> 16) & 0xFFu);
      CHSGA_CHK_RANGE(k0, k1, g.n_ent, 21);
      const uint32_t key = ry >> 29;
      const size_t so = (size_t)s * R + 8 * q;
      const uint4 rf = __ldg(reinterpret_cast<const uint4*>(RFin + so));
      const uint4 d = *reinterpret_cast<const uint4*>(&sh.mis16[key][8 * q]);
      const uint16_t* rl = RLin + 8 * q;
      uint4 F = rf;
      // no source: above every score, and one more does not wrap
      const uint32_t none = WIDE ? 0xFFFFFFFFu : 0x80008000u;
      uint4 M = make_uint4(none, none, none, none), T;
      for (uint32_t k = k0; k < k1; k += U) {
        uint2 e[U];
        uint4 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < k1) e[u] = __ldg(g.ent16 + k + u);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < k1) x[u] = __ldg(reinterpret_cast<const uint4*>(rl + (size_t)CHSGA_CHK(e[u].x, g.S, 22) * R));
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u < k1) {
            const uint32_t ww = WIDE ? e[u].y : __vminu2(e[u].y, 0x80008000u);
            const uint32_t wm = __byte_perm(ww, 0, 0x1010), wf = __byte_perm(ww, 0, 0x3232);
            if (WIDE) {
              M = min4(M, addw4(x[u], wm));
              F = min4(F, addw4(x[u], wf));
            } else {
              M = viaddmin4(x[u], wm, M);
              F = viaddmin4(x[u], wf, F);
            }
          }
      }
      const uint4 F1 = make_uint4(F.x + ONES, F.y + ONES, F.z + ONES, F.w + ONES);
      if (WIDE)
        T = min4(F1, add4(M, d));
      else
        T = make_uint4(__viaddmin_u16x2(M.x, d.x, F1.x), __viaddmin_u16x2(M.y, d.y, F1.y),
                       __viaddmin_u16x2(M.z, d.z, F1.z), __viaddmin_u16x2(M.w, d.w, F1.w));
      uint4 in = zero;
      if (hf.init) {
        in = *reinterpret_cast<const uint4*>(sh.init + 8 * q);
        T = sel4(d, T, in);
      }
      *reinterpret_cast<uint4*>(RFout + so) = T;
      *reinterpret_cast<uint4*>(sF + vl * R + 8 * q) = F;
      if (hf.drain) {
        uint32_t m = at_most8(F, *reinterpret_cast<const uint4*>(&sh.lim[1][8 * q]));
        m &= sh.drain[q >> 2] >> (8 * (q & 3));
        if (m) {
          const uint32_t f = __ldg(g.sv_off + s);
          for (; m; m &= m - 1) {
            const int v = __ffs(m) - 1;
            atomicMin(&sh.best[1][8 * q + v], pack_min(sF[vl * R + 8 * q + v], f));
          }
        }
      }
      if (hf.end) {
        // a chain falls by at most one a char: most vertices stay above the best so far
        const uint32_t n = ((ry & 0x1FFFFFFFu) - 1) * ONES;
        const uint4 lo = make_uint4(__vsubus2(T.x, n), __vsubus2(T.y, n), __vsubus2(T.z, n), __vsubus2(T.w, n));
        sP[ENDC][it] = (uint8_t)(at_most8(lo, *reinterpret_cast<const uint4*>(&sh.lim[0][8 * q])) &
                                 (sh.end[q >> 2] >> (8 * (q & 3))));
      }
      // chain start: not below F - 1 (max(T + 1, F) - 1; no half wraps)
      const uint4 T1 = max4(make_uint4(T.x + ONES, T.y + ONES, T.z + ONES, T.w + ONES), F);  // + 1
      uint4 low = sub4(sub4(T1, one), T), gap = sub4(rf, F);
      uint4 ch = sub4(T1, F);  // change of the first score + 1: 0..2
      if (hf.init) {  // row 0: its mismatch + 1
        low = sel4(zero, low, in);
        gap = sel4(zero, gap, in);
        ch = sel4(make_uint4(d.x + ONES, d.y + ONES, d.z + ONES, d.w + ONES), ch, in);
      }
      uint32_t g0, g1, c0, c1, big = 0;
      if ((gap.x | gap.y | gap.z | gap.w) & 0xFFFCFFFCu) {
        big = nonzero8(make_uint4(gap.x & 0xFFFCFFFCu, gap.y & 0xFFFCFFFCu, gap.z & 0xFFFCFFFCu, gap.w & 0xFFFCFFFCu));
        const uint4 b16 = unplane(big);
        gap = sel4(zero, gap, make_uint4(b16.x * 0xFFFFu, b16.y * 0xFFFFu, b16.z * 0xFFFFu, b16.w * 0xFFFFu));
      }
      planes2(gap, g0, g1);
      planes2(ch, c0, c1);
      sP[G0][it] = (uint8_t)g0;
      sP[G1][it] = (uint8_t)g1;
      sP[VP][it] = (uint8_t)c1;
      sP[VN][it] = (uint8_t)(~(c0 | c1));
      sP[GBIG][it] = (uint8_t)big;
      sP[LOW][it] = (low.x | low.y | low.z | low.w) ? (uint8_t)nonzero8(low) : (uint8_t)0;
    }
    __syncwarp();
    // ---- pass 2
    {
      const uint32_t vl = lane / W, w = lane % W;
      const uint32_t s = __shfl_sync(0xFFFFFFFFu, my_s, vl % VB);
      if (vl < nv) {
        uint32_t f = __ldg(g.sv_off + s), e = __ldg(g.sv_off + s + 1);
        CHSGA_CHK_CHARS(f, e, g.N, 1);
        const uint32_t n = e - f - 1;  // chain chars
        uint2* const z0 = static_cast<uint2*>(a.bits) + (size_t)(f + 1) * W + w;
        auto plane = [&](int p) { return reinterpret_cast<const uint32_t*>(sP[p])[vl * W + w]; };
        if (n) {
          uint32_t vp = plane(VP), vn = plane(VN);
          const uint32_t keep = sh.keep[w];
          uint32_t g0 = plane(G0), g1 = plane(G1);
          for (uint32_t big = plane(GBIG); big; big &= big - 1) {
            const uint32_t b = __ffs(big) - 1, r = 32 * w + b;
            line_slot(z0, W, n, 1u << b, (uint32_t)RFin[(size_t)s * R + r] - sF[vl * R + r]);
          }
          const uint32_t* kp = g.lab4 + ((f + 1) >> 3);  // label keys, 8 chars a word
          const uint32_t ks = ((f + 1) & 7u) * 4u;
          uint32_t klo = __ldg(kp);
          // chars whose words load together: a lone group of vertices waits for
          // each load, many groups lose more to the chars past the last
          constexpr int U2 = K == 1 ? 8 : 4;
          uint32_t keys = 0, c = 0;
          uint2* z = z0;
          auto one = [&](uint2* at, const uint2& x, uint32_t key) {
            const uint32_t d = sh.mis[key * W + w];
            const uint32_t p = x.x, m = x.y;
            // the previous row under its line (row 0 slots have none)
            const uint32_t t0 = g0 & ~m;
            const uint32_t hp = (p & keep) | g1 | t0;
            const uint32_t hn = m & keep & ~(g1 | g0);
            const uint32_t b = g1 & ~(g0 ^ m);
            g1 &= p | t0;
            g0 = (p & g0) | (~p & b);
            // the new score is 1 above the previous row's left neighbour, else level with it
            const uint32_t t1 = d & ~(vn | hn);
            const uint32_t op = vn | (t1 & ~vp), om = vp & ~t1;
            vp = hn | (t1 & ~hp);
            vn = hp & ~t1;
            *at = make_uint2(op, om);
          };
          auto next_keys = [&] {  // of the chars c .. c + 7, when c is a multiple of 8
            const uint32_t khi = __ldg(++kp);
            keys = __funnelshift_r(klo, khi, ks);
            klo = khi;
          };
          for (; c < n; c += U2, z += U2 * W) {
            uint2 x[U2];
#pragma unroll
            for (int u = 0; u < U2; ++u)
              if (c + u < n) x[u] = z[u * W];
            if (U2 == 4 && (c & 4u))
              keys >>= 16;
            else
              next_keys();
#pragma unroll
            for (int u = 0; u < U2; ++u)
              if (c + u < n) one(z + u * W, x[u], (keys >> (4 * u)) & 7u);
          }
          for (uint32_t lb = plane(LOW); lb; lb &= lb - 1) {
            const uint32_t b = __ffs(lb) - 1, r = 32 * w + b;
            line_slot(z0, W, n, 1u << b, (uint32_t)sF[vl * R + r] - 1u - RFout[(size_t)s * R + r]);
          }
          reinterpret_cast<uint32_t*>(sP[VP])[vl * W + w] = vp;
          reinterpret_cast<uint32_t*>(sP[VN])[vl * W + w] = vn;
        }
        if (hf.end) {
          for (uint32_t eb = plane(ENDC); eb; eb &= eb - 1) {
            const uint32_t b = __ffs(eb) - 1, r = 32 * w + b;
            int cur = RFout[(size_t)s * R + r], bm = cur;
            uint32_t bc = f;
            for (uint32_t c = 0; c < n; ++c) {
              const uint2 x = z0[(size_t)c * W];
              cur += (int)((x.x >> b) & 1u) - (int)((x.y >> b) & 1u);
              if (cur < bm) {
                bm = cur;
                bc = f + 1 + c;
              }
            }
            atomicMin(&sh.best[0][r], pack_min(bm, bc));
          }
        }
      }
    }
    __syncwarp();
    // ---- pass 3 (first + len - 1 stays below 2^16: the kernel runs up to 512 chars)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t it = lane + 32 * j, vl = it / C, q = it % C;
      const uint32_t s = __shfl_sync(0xFFFFFFFFu, my_s, vl);
      if (vl >= nv) continue;
      const uint32_t len = __ldg(&g.rec[s].y) & 0x1FFFFFFFu;
      const size_t so = (size_t)s * R + 8 * q;
      uint4 o;
      if (len == 1) {
        o = *reinterpret_cast<const uint4*>(RFout + so);
      } else {
        const uint32_t lw = (len - 1) * ONES;
        o = viaddmin4(*reinterpret_cast<const uint4*>(sF + vl * R + 8 * q), lw,
                      __ldg(reinterpret_cast<const uint4*>(RLin + so)));
        if (hf.init) o = sel4(zero, o, *reinterpret_cast<const uint4*>(sh.init + 8 * q));
        const uint4 p = unplane(sP[VP][it]), m = unplane(sP[VN][it]);
        o = make_uint4(o.x + p.x - m.x, o.y + p.y - m.y, o.z + p.z - m.z, o.w + p.w - m.w);
        if (sP[LOW][it]) o = viaddmin4(*reinterpret_cast<const uint4*>(RFout + so), lw, o);
      }
      *reinterpret_cast<uint4*>(RLout + so) = o;
    }
    if (hf.end) {
      // hand the best so far to the other blocks and take theirs. Warps read
      // lim and best while others write them: values only fall, and an old one
      // only prunes less
      for (int r = (int)lane; r < R; r += 32) {
        const unsigned long long b = *(volatile unsigned long long*)&sh.best[0][r];
        if (b == ~0ull) continue;
        unsigned long long* gb = a.best + ((sh.word[r] >> SW_PAR_SHIFT) & 3u) * R + r;
        const unsigned long long o = __ldcg(gb);
        if (b < o) atomicMin(gb, b);
        sh.lim[0][r] = (uint16_t)min((unsigned long long)0xFFFFu, min(b, o) >> 32);
      }
    }
    __syncwarp();  // the next vertices reuse the warp's arrays
  }
}

template <int R, int K>
__global__ void __launch_bounds__(kSlicedThreads, CHSGA_SLICED_WARPS * 32 / kSlicedThreads) k_row_sliced(BitArgs a) {
  using Shared = SlicedShared<R, K>;
  constexpr int NT = Shared::NT, W = Shared::W;
  static_assert(R <= NT, "a thread per slot");
  __shared__ __align__(16) Shared sh;
  pdl_wait();
  const HeadFlags hf = bits_head<R>(a, sh.word, nullptr);
  if (!hf.work) return;
  // the step's words: per label key the mismatches of 32 slots, and as 16-bit increments
  if (threadIdx.x < R) {
    const int i = threadIdx.x;
    const uint32_t w = sh.word[i], m = (w >> SW_MASK_SHIFT) & SW_MASK;
    const bool init = (w & SW_INIT) || !(w & SW_ACTIVE);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < 5) sh.mis16[k][i] = (uint16_t)((m >> k) & 1u);
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, (m >> k) & 1u);
      if ((i & 31) == 0) sh.mis[k * W + (i >> 5)] = b;
    }
    sh.init[i] = init ? 0xFFFFu : 0u;
    const uint32_t bk = __ballot_sync(0xFFFFFFFFu, !init), be = __ballot_sync(0xFFFFFFFFu, (w & SW_ENDING) != 0),
                   bd = __ballot_sync(0xFFFFFFFFu, (w & SW_DRAIN) != 0);
    if ((i & 31) == 0) {
      sh.keep[i >> 5] = bk;
      sh.end[i >> 5] = be;
      sh.drain[i >> 5] = bd;
    }
    sh.best[0][i] = sh.best[1][i] = ~0ull;
    sh.lim[0][i] = 0xFFFFu;
    // a draining read's raw minimum is known: only scores that reach it count
    if (hf.drain)
      sh.lim[1][i] = (uint16_t)min((unsigned long long)0xFFFFu,
                                   __ldcg(a.best + (((w >> SW_PAR_SHIFT) + 3u) & 3u) * R + i) >> 32);
  }
  __syncthreads();
  if (hf.wide)
    sliced_warp<R, K, true>(a, hf, sh);
  else
    sliced_warp<R, K, false>(a, hf, sh);
  if (hf.end || hf.drain) {
    __syncthreads();
    if (threadIdx.x < R) {
      const int i = threadIdx.x;
      const uint32_t par = (sh.word[i] >> SW_PAR_SHIFT) & 3u;
      if (sh.best[0][i] != ~0ull) atomicMin(a.best + par * R + i, sh.best[0][i]);
      if (sh.best[1][i] != ~0ull) atomicMin(a.best + ((par + 3u) & 3u) * R + i, sh.best[1][i]);
    }
  }
}

}  // namespace dev
}  // namespace chsga
