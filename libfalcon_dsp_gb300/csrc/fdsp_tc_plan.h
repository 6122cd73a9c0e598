// Launch planning of the tensor-core filter-bank kernel (host only).
//
// One launch covers every decimation group computed on the tensor cores.
// Per group the output rows (windows ending D apart) become 128-row tiles of
// a matrix product Y = A B:
//
//   A[j][k]  input sample  j D' + a + k  of [history | block], split into
//            16-bit {hi, lo} parts: 4 K elements per sample
//            (re_hi, im_hi, re_lo, im_lo), a Hankel matrix that TMA loads
//            16 samples (128 bytes) at a time through a tensor map whose
//            row stride is D' samples;
//   B[k][n]  the NCO-modulated taps of each output stream ("slot") at its
//            offset inside the merged window, hi taps in columns [0, 2 NS),
//            lo taps in [2 NS, 4 NS) (Re, Im per slot): the epilogue adds
//            the two halves, so each output is (x_hi + x_lo)(g_hi + g_lo)
//            with FP32 accumulation.
//
// A slot is one output class of one channel: output m = r + U j of channel
// c uses tap phase phi and the window ending at delta + j D (block relative).
// A row split S (rows j = S i + b become S slots whose rows are S D apart)
// widens groups with few slots, and makes an odd D even (TMA strides are
// multiples of 16 bytes = 2 samples).  Slots sorted by window start are
// kept together per channel (a bundle, in output order) and partitioned into
// merge sets ("msets") of <= 64 slots (N <= 256) by the fewest K chunks; an
// mset's window starts on an even sample (TMA x coordinates are multiples of
// 16 bytes) and is chunked in 16 taps.
//
// Kept apart from the kernel so that its bounds can be checked on the CPU
// (tests/cpp/tc_plan_check.cc).
#pragma once

#include <stdint.h>

#include <algorithm>
#include <climits>
#include <cstddef>
#include <vector>

#if defined(__CUDACC__)
#define FDSP_HD __host__ __device__
#else
#define FDSP_HD
#endif

namespace fdsp {

constexpr int kTcMaxGroups = 16;
constexpr int kTcSideStreams = 3;  // streams of launch packs 1.. (pack 0 runs on the caller's)
constexpr int kTcMaxMsets = 64;
constexpr int kTcMaxSlots = 512;
constexpr int kTcRows = 128;           // rows per tile (MMA M)
constexpr int kTcChunkTaps = 16;       // taps per K chunk: 128 bytes of A per row
constexpr int kTcTileBytes = kTcRows * 128;
constexpr int kTcMsetSlots = 64;       // slots per merge set (N = 4 NS <= 256)
constexpr int kTcStageMaxBytes = 49152;
constexpr int kTcSmemDyn = 223 * 1024; // dynamic shared memory ceiling (227 KB minus static and alignment)
constexpr int kTcMaxStages = 6;
constexpr int kTcEpiSlotBytes = 48;    // per-slot epilogue constants staged in shared memory
constexpr int kTcEpiWarps = 16;        // epilogue warps, each with its own scratch:
constexpr int kTcEpiRows = 32 * 8 * 8; // 32 rows of 8 outputs (launches with runs)
constexpr int kTcEpiRecs = 16 * 48;    // and a record per slot of two chunks

// ---- launch records (kernel parameters; shared with the device code) -----
struct TcGroup {
  int32_t D;        // row stride D' = S D (samples, even)
  int32_t S;        // row split
  int32_t pad_[2];
};

struct TcMset {
  uint64_t b;       // device address of its B image: [nchunks][N][128 B]
  int32_t a;        // window start of row 0 in [history | block] samples (even)
  int32_t items;    // work items (R tiles each)
  int16_t group, slot0, NS, nchunks, R, pad_;
  int32_t ntiles;   // 128-row tiles with an output
};

struct TcSlot {
  uint64_t out;     // float2*: output of row 0 (channel output + r)
  int32_t w0;       // window start of row 0, block relative (delta - T + 1)
  int32_t J;        // rows with an output (0: padding slot)
  uint16_t ch;      // channel
  uint16_t T;       // taps per phase
  uint16_t U;       // output stride (up rate x row split)
  uint16_t o;       // window start inside the merge set's window (taps)
  uint16_t phi;     // tap phase
  uint16_t flags;   // kTcPair .. kTcRun
  uint16_t D;       // row stride D' (samples)
  uint16_t pad_;
};

// Slot flags: how the epilogue stores a slot's outputs (8 slots, a column
// chunk, are one warp's).
constexpr int kTcPair = 1;      // the next slot holds the same channel's next output (16-byte store)
constexpr int kTcQuad = 2;      // and the two after it, rows multiples of 32 bytes (32-byte store)
constexpr int kTcRun = 4;       // one of a row's outputs, all of them in this chunk: bits 4-7 their number (3-8),
                                // bits 8-11 this one's place (rows follow one another without gaps)
FDSP_HD constexpr int tc_run_len(int flags) { return (flags >> 4) & 15; }
FDSP_HD constexpr int tc_run_pos(int flags) { return (flags >> 8) & 15; }
static_assert(sizeof(TcSlot) == 32, "slot record");
static_assert(sizeof(TcMset) == 32, "merge-set record");

// ---- planner input ----------------------------------------------------------
struct TcSlotIn {
  int ch, T, U, r, phi;
  int64_t delta;    // window end of row 0 (block relative)
  int64_t J;        // rows with an output this apply
};
struct TcGroupIn {
  int D;
  int max_split;    // largest row split allowed (power of two, 1..32)
  std::vector<TcSlotIn> slots;
};

struct TcPlanGroup {
  int D, S;
  int64_t Wx;       // samples a row of its tensor map spans (max over its msets of (a mod D') + Kw)
};

struct TcPlan {
  std::vector<TcPlanGroup> groups;
  std::vector<TcMset> ms;         // b = byte offset into the B buffer (the engine adds the base)
  std::vector<TcSlot> slots;      // out = 0 (the engine fills it)
  std::vector<int> slot_r;        // output offset r of each slot (for the out pointer)
  size_t b_bytes = 0;
  int64_t xhl_samples = 0;        // [history | block | zero pad] samples the split writes
  int stages = 0, stage_bytes = 0, smem = 0;  // smem: stages, the epilogue slot table, the epilogue warps' scratch
  int table_off = 0, scratch_off = 0;         // (from the 1 KB aligned start)
  int scratch_warp = 0;                       // bytes of a warp's scratch
  int G = 0;                      // grid (CTAs)
  int64_t Lc = 0;                 // samples a CTA has on average (the cut by input range, tc_item_range)
  int64_t items = 0;
  uint32_t ctotal = 0;            // cost of all items, each at least 1 and scaled by 2^-cost_shift
  int cost_shift = 0;
};

inline int64_t tc_round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// A slot of a split group: output m = r + U j, window ending at delta + j D'.
struct TcSlotX {
  TcSlotIn s;
  int64_t start;  // window start of row 0 (block relative)
};

// A bundle: every slot of one channel under row split S, in output order
// (offset r + b U = 0 .. U S - 1), so that row j of the bundle holds the
// channel's consecutive outputs U S j .. U S j + U S - 1 and the epilogue
// writes them as contiguous pairs (a slot at an even position of its merge
// set and the next one of the same bundle).  Its width is its slot count:
// bundles sit back to back, a one-slot bundle takes one column pair.
struct TcBundle {
  int first, last;  // the channel's slots [first, last) of the sorted group (in output order, before the split)
  int64_t start;    // earliest window start of its slots
  int64_t end;      // latest window end
  int width;
};

// The group's slots by channel and output offset: a bundle's slots are then
// one range, whatever the split.
inline std::vector<TcSlotIn> tc_sorted(const TcGroupIn& g) {
  std::vector<TcSlotIn> xs = g.slots;
  std::stable_sort(xs.begin(), xs.end(),
                   [](const TcSlotIn& a, const TcSlotIn& b) { return a.ch != b.ch ? a.ch < b.ch : a.r < b.r; });
  return xs;
}

// Calls fn(slot) for the slots of xs[first, last) under row split S, in output
// order: rows j = S i + b become slot b, whose rows are S D apart.
template <class Fn>
inline void tc_split_slots(const std::vector<TcSlotIn>& xs, int first, int last, int D, int S, Fn&& fn) {
  for (int b = 0; b < S; ++b)
    for (int i = first; i < last; ++i) {
      const TcSlotIn& s = xs[i];
      if (s.J <= b) continue;
      TcSlotX x;
      x.s = s;
      x.s.delta = s.delta + (int64_t)b * D;
      x.s.J = (s.J - b + S - 1) / S;
      x.s.U = s.U * S;
      x.s.r = s.r + b * s.U;
      x.start = x.s.delta - s.T + 1;
      fn(x);
    }
}

// Bundles of the sorted slots under row split S, by window start.
inline void tc_bundles(const std::vector<TcSlotIn>& xs, int D, int S, std::vector<TcBundle>& bs) {
  bs.clear();
  for (int i = 0; i < (int)xs.size();) {
    TcBundle b;
    b.first = i;
    b.start = INT64_MAX;
    b.end = INT64_MIN;
    b.width = 0;
    for (; i < (int)xs.size() && xs[i].ch == xs[b.first].ch; ++i) {
      const int n = (int)std::min<int64_t>(S, xs[i].J);  // slots of this output class
      if (n <= 0) continue;
      b.start = std::min(b.start, xs[i].delta - xs[i].T + 1);
      b.end = std::max(b.end, xs[i].delta + (int64_t)(n - 1) * D);
      b.width += n;
    }
    b.last = i;
    if (b.width > 0) bs.push_back(b);
  }
  std::stable_sort(bs.begin(), bs.end(), [](const TcBundle& a, const TcBundle& b) {
    return a.start != b.start ? a.start < b.start : a.end < b.end;
  });
}

// Merge-set window of bundles [i, j) (sorted by start): its start in
// [history | block] samples rounded down to even, and its K chunks.
inline void tc_window(const std::vector<TcBundle>& bs, size_t i, size_t j, int H, int64_t* a, int64_t* chunks) {
  int64_t st = bs[i].start + H;
  if (st & 1) st -= 1;
  int64_t end = bs[i].end;
  for (size_t q = i + 1; q < j; ++q) end = std::max(end, bs[q].end);
  *a = st;
  *chunks = (end + H - st + 1 + kTcChunkTaps - 1) / kTcChunkTaps;
}

// Partition of the sorted bundles into merge sets of at most kTcMsetSlots
// slots minimising the total K chunks: one MMA of M = 128, K = 16 costs the
// same for any N up to 256, so the work of a tile is its merge sets' chunks
// (dynamic programming over the split points).  Returns the cut points and
// the chunks per tile row; -1 when a bundle alone exceeds a merge set.
inline int64_t tc_partition(const std::vector<TcBundle>& bs, int H, std::vector<size_t>& cuts) {
  const size_t n = bs.size();
  std::vector<int64_t> best(n + 1, INT64_MAX);
  std::vector<size_t> from(n + 1, 0);
  best[0] = 0;
  for (size_t i = 0; i < n; ++i) {
    if (best[i] == INT64_MAX) continue;
    int64_t st = bs[i].start + H;
    if (st & 1) st -= 1;
    int64_t end = bs[i].end;
    int width = 0;
    for (size_t j = i + 1; j <= n; ++j) {
      width += bs[j - 1].width;
      if (width > kTcMsetSlots) break;
      end = std::max(end, bs[j - 1].end);
      const int64_t c = best[i] + (end + H - st + 1 + kTcChunkTaps - 1) / kTcChunkTaps;
      if (c < best[j]) {
        best[j] = c;
        from[j] = i;
      }
    }
  }
  cuts.clear();
  if (best[n] == INT64_MAX) return -1;
  for (size_t j = n; j > 0; j = from[j]) cuts.push_back(j);
  cuts.push_back(0);
  std::reverse(cuts.begin(), cuts.end());
  return best[n];
}

// Row split of a group: the power of two up to max_split (S even for odd D,
// so that rows start 16 bytes apart) with the fewest K chunks over all its
// tiles (chunks per tile row x rows / S); ties keep the smaller split.  A
// channel's bundle (U S slots) fits one merge set, and the group's slots
// stay within four full merge sets.
inline int tc_choose_split(const std::vector<TcSlotIn>& xs, int D, int max_split, int H) {
  int64_t J = 0;
  int Umax = 1;
  for (const TcSlotIn& s : xs) {
    J = std::max(J, s.J);
    Umax = std::max(Umax, s.U);
  }
  int bestS = 0;
  double bestc = 0;
  std::vector<TcBundle> bs;
  std::vector<size_t> cuts;
  for (int S = 1; S <= std::max((D & 1) ? 2 : 1, max_split); S *= 2) {
    if ((D & 1) && (S & 1)) continue;
    if ((int64_t)Umax * S > kTcMsetSlots) break;
    if (S > 2 && (int64_t)xs.size() * S > 4 * kTcMsetSlots) break;
    tc_bundles(xs, D, S, bs);
    if (bs.empty()) continue;
    const int64_t ch = tc_partition(bs, H, cuts);
    if (ch < 0) continue;
    const double c = (double)ch * (double)((J + (int64_t)S * kTcRows - 1) / ((int64_t)S * kTcRows));
    if (bestS == 0 || c < bestc) {
      bestS = S;
      bestc = c;
    }
  }
  return bestS;
}

// Positions of bundles [i, j) in a merge set of NS slots.  The epilogue's warps
// take 8 slots each, so bundles are packed into runs of 8 where they fit
// (widest first, first fit: 6 + 2, 3 + 3 + 1 + 1, 4 + 4), which keeps a row's
// outputs in one warp; where that would need more columns they sit back to
// back.  Position b of `order` starts at at[b].
inline void tc_arrange(const std::vector<TcBundle>& bs, size_t i, size_t j, int NS, std::vector<int>& order,
                       std::vector<int>& at) {
  order.clear();
  at.clear();
  for (size_t b = i; b < j; ++b) order.push_back((int)b);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return bs[a].width > bs[b].width; });
  int used[kTcMsetSlots / 8] = {0};
  const int bins = NS / 8;
  bool fits = true;
  for (int b : order) {
    const int w = bs[b].width, whole = w / 8, rest = w % 8;
    int p = -1;
    for (int c = 0; c + whole + (rest ? 1 : 0) <= bins && p < 0; ++c) {
      if (whole == 0) {
        if (used[c] + rest <= 8) p = c * 8 + used[c];
        continue;
      }
      bool free = true;
      for (int k = 0; k < whole + (rest ? 1 : 0); ++k) free = free && used[c + k] == 0;
      if (free) p = c * 8;
    }
    if (p < 0) {
      fits = false;
      break;
    }
    at.push_back(p);
    for (int k = 0; k < whole; ++k) used[p / 8 + k] = 8;
    if (rest) used[p / 8 + whole] += rest;
  }
  if (fits) return;
  at.clear();
  int p = 0;
  for (int b : order) {
    at.push_back(p);
    p += bs[b].width;
  }
}

// One group planned by itself: its merge sets (group 0, slots and B image
// counted from 0), to be placed into a launch by tc_append.
struct TcGroupPlan {
  TcPlanGroup g;
  std::vector<TcMset> ms;
  std::vector<TcSlot> slots;
  std::vector<int> slot_r;
  size_t b_bytes = 0;
};

// Plans a group; S: its row split, or 0 to choose one.  Returns 0, or -1 when
// the group exceeds a launch's record limits by itself.  A group without
// outputs gives a plan without merge sets.
inline int tc_plan_group(const TcGroupIn& g, int H, int S, TcGroupPlan& q) {
  q = TcGroupPlan();
  const std::vector<TcSlotIn> xs = tc_sorted(g);
  if (S == 0) S = tc_choose_split(xs, g.D, g.max_split, H);
  if (S == 0) return -1;
  const int64_t Dp = (int64_t)S * g.D;
  if (Dp > 65535) return -1;  // record field range
  q.g.D = (int)Dp;
  q.g.S = S;
  q.g.Wx = 0;
  std::vector<TcBundle> bs;
  std::vector<size_t> cuts;
  tc_bundles(xs, g.D, S, bs);
  if (bs.empty()) return 0;
  if (tc_partition(bs, H, cuts) < 0) return -1;
  for (size_t ci = 0; ci + 1 < cuts.size(); ++ci) {
    const size_t i = cuts[ci], j = cuts[ci + 1];
    int64_t a, nchunks;
    tc_window(bs, i, j, H, &a, &nchunks);
    int width = 0;
    for (size_t b = i; b < j; ++b) width += bs[b].width;
    if (nchunks * kTcChunkTaps > 65535) return -1;  // record field ranges (16-bit taps, strides and offsets)
    const int NS = (int)tc_round_up(width, 8);
    if ((int)q.ms.size() >= kTcMaxMsets || (int)q.slots.size() + NS > kTcMaxSlots) return -1;
    TcMset m{};
    m.a = (int32_t)a;
    m.slot0 = (int16_t)q.slots.size();
    m.NS = (int16_t)NS;
    m.nchunks = (int16_t)nchunks;
    int64_t Jmax = 0;
    bool range = true;
    std::vector<int> order, at;
    tc_arrange(bs, i, j, NS, order, at);
    q.slots.resize((size_t)m.slot0 + NS, TcSlot{});
    q.slot_r.resize((size_t)m.slot0 + NS, 0);
    for (size_t b = 0; b < order.size(); ++b) {
      const TcBundle& bd = bs[order[b]];
      const int n0 = at[b];  // the bundle's first position in the merge set
      int n = n0;
      tc_split_slots(xs, bd.first, bd.last, g.D, S, [&](const TcSlotX& x) {
        if (x.s.T > 65535 || x.s.U > 65535 || x.s.phi > 65535 || x.s.J > INT32_MAX) range = false;
        TcSlot& s = q.slots[(size_t)m.slot0 + n];
        s.w0 = (int32_t)x.start;
        s.J = (int32_t)x.s.J;
        s.ch = (uint16_t)x.s.ch;
        s.T = (uint16_t)x.s.T;
        s.U = (uint16_t)x.s.U;
        s.o = (uint16_t)(x.start + H - a);
        s.phi = (uint16_t)x.s.phi;
        s.D = (uint16_t)Dp;
        q.slot_r[(size_t)m.slot0 + n] = x.s.r;
        Jmax = std::max(Jmax, x.s.J);
        ++n;
      });
      // how each position is stored: whole rows of 3, 5, 6 or 7 outputs in one
      // chunk go through shared memory, else the widest aligned pieces
      const TcSlot* sl = &q.slots[(size_t)m.slot0];
      const int* r = &q.slot_r[(size_t)m.slot0];
      const int W = sl[n0].U;
      const bool run = n - n0 == W && W >= 3 && W <= 7 && W != 4 && n0 / 8 == (n - 1) / 8;
      for (int k = n0; k < n; ++k) {
        int f = 0;
        if (k % 2 == 0 && k + 1 < n && r[k + 1] == r[k] + 1) f |= kTcPair;
        if (k % 4 == 0 && k + 3 < n && W % 4 == 0 && r[k] % 4 == 0 && r[k + 3] == r[k] + 3) f |= kTcQuad;
        if (run) f |= kTcRun | (W << 4) | ((k - n0) << 8);
        q.slots[(size_t)m.slot0 + k].flags = (uint16_t)f;
      }
    }
    if (!range) return -1;
    m.ntiles = (int32_t)((Jmax + kTcRows - 1) / kTcRows);
    m.R = (int16_t)(4 * NS <= 128 ? 2 : 1);  // two narrow tiles an item share each B chunk
    m.items = (m.ntiles + m.R - 1) / m.R;
    m.b = q.b_bytes;
    q.b_bytes += (size_t)tc_round_up((int64_t)m.nchunks * 4 * NS * 128, 1024);
    q.g.Wx = std::max<int64_t>(q.g.Wx, a % Dp + (int64_t)m.nchunks * kTcChunkTaps);
    q.ms.push_back(m);
  }
  return 0;
}

// Adds a planned group to launch p; false when the launch's records are full.
inline bool tc_append(TcPlan& p, const TcGroupPlan& q) {
  if (p.groups.size() >= (size_t)kTcMaxGroups || p.ms.size() + q.ms.size() > (size_t)kTcMaxMsets ||
      p.slots.size() + q.slots.size() > (size_t)kTcMaxSlots)
    return false;
  for (TcMset m : q.ms) {
    m.group = (int16_t)p.groups.size();
    m.slot0 = (int16_t)(m.slot0 + p.slots.size());
    m.b += p.b_bytes;
    p.ms.push_back(m);
  }
  p.groups.push_back(q.g);
  p.slots.insert(p.slots.end(), q.slots.begin(), q.slots.end());
  p.slot_r.insert(p.slot_r.end(), q.slot_r.begin(), q.slot_r.end());
  p.b_bytes += q.b_bytes;
  return true;
}

// Items of a merge set (first start a, step P) that start before sample lim:
// summed over the merge sets, an item's place in the launch's item list.
FDSP_HD inline uint32_t tc_items_before(uint32_t a, uint32_t P, uint32_t items, uint32_t lim) {
  if (lim <= a) return 0;
  const uint32_t n = (lim - a + P - 1u) / P;
  return n < items ? n : items;
}

// Cost of an item in units of 32 cycles: 4 MMAs a chunk and tile, which took
// 96 cycles at N = 128 and 168 at N = 256, and about 2000 cycles to start,
// drain and store it; in units of 2^shift as much for launches of more work.
// Never 0, so costs grow along the item list.
FDSP_HD inline uint32_t tc_item_cost(const TcMset& m, int shift = 0) {
  const uint32_t c = (((uint32_t)m.R * (uint32_t)m.nchunks * (96u + 9u * (uint32_t)m.NS) + 2000u) / 32u) >> shift;
  return c > 0u ? c : 1u;
}

// Input samples between the starts of a merge set's items.
template <class Group>
FDSP_HD inline uint32_t tc_item_step(const TcMset& m, const Group* groups) {
  return (uint32_t)m.R * (uint32_t)kTcRows * (uint32_t)groups[m.group].D;
}

// Where item t of merge set m stands in the list of all items, ordered by
// first input sample (ties: the lower merge set), and the cost of the items
// before it: a division per merge set gives both.
template <class Group>
FDSP_HD inline void tc_item_place(const TcMset* ms, int nmsets, const Group* groups, int m, int t, int shift,
                                  uint32_t* place, uint32_t* cost) {
  const uint32_t u = (uint32_t)ms[m].a + (uint32_t)t * tc_item_step(ms[m], groups);
  *place = *cost = 0;
  for (int k = 0; k < nmsets; ++k) {
    const uint32_t before =
        tc_items_before((uint32_t)ms[k].a, tc_item_step(ms[k], groups), (uint32_t)ms[k].items, u + (k < m ? 1u : 0u));
    *place += before;
    *cost += before * tc_item_cost(ms[k], shift);
  }
}

// The items of CTA b of G are those whose cost before them lies in
// [tc_cost_bound(b), tc_cost_bound(b + 1)).
FDSP_HD inline uint32_t tc_cost_bound(uint32_t total, int b, int G) {
  return (uint32_t)(((uint64_t)total * (uint64_t)b + (uint64_t)G - 1u) / (uint64_t)G);
}

// Sizes and schedule of a launch whose groups are all added.  Returns 0, or
// -1 when its stages do not fit shared memory.
inline int tc_finish(TcPlan& p, int64_t N, int H, int num_sms) {
  if (p.ms.empty()) return 0;
  int64_t wx_max = 0;
  for (const TcPlanGroup& g : p.groups) wx_max = std::max(wx_max, g.Wx);
  // the split writes [history | block] and a zero tail: every row a tensor
  // map can address ((rows - 1) D' + Wx samples) stays inside it
  p.xhl_samples = tc_round_up(N + H + wx_max + 16, 16);
  // pipeline stages: R A tiles + one B chunk each
  int sb = 0;
  for (const TcMset& m : p.ms)
    sb = std::max<int>(sb, m.R * kTcTileBytes + (int)tc_round_up((int64_t)4 * m.NS * 128, 1024));
  if (sb > kTcStageMaxBytes) return -1;
  p.stage_bytes = sb;
  const int table = (int)tc_round_up((int64_t)p.slots.size() * kTcEpiSlotBytes, 1024);
  bool runs = false;
  for (const TcSlot& x : p.slots) runs = runs || (x.flags & kTcRun) != 0;
  p.scratch_warp = kTcEpiRecs + (runs ? kTcEpiRows : 0);  // (without runs: one more stage for narrow tiles)
  const int scratch = kTcEpiWarps * p.scratch_warp;
  p.stages = std::min(kTcMaxStages, (kTcSmemDyn - 1024 - table - scratch) / sb);
  if (p.stages < 2) return -1;
  p.table_off = p.stages * sb;
  p.scratch_off = p.table_off + table;
  p.smem = p.scratch_off + scratch + 1024;
  // schedule: a CTA an SM at most, each running a stretch of the item list
  // (tc_cost_bound) in input order
  int64_t umax = 0;
  for (const TcMset& m : p.ms) {
    const int64_t P = (int64_t)m.R * kTcRows * p.groups[m.group].D;
    umax = std::max<int64_t>(umax, m.a + (int64_t)m.items * P);
    p.items += m.items;
  }
  p.G = (int)std::max<int64_t>(1, std::min<int64_t>(num_sms, p.items));
  p.Lc = (umax + p.G - 1) / p.G;
  // The CTAs' cuts and the costs in the item list are 32-bit: the unit of cost
  // doubles until the total stays below 2^31 (only calls of half a second of
  // work and more, such as 4095 taps of 32 channels over 2^31 samples, need it).
  uint64_t total = 0;
  for (p.cost_shift = 0;; ++p.cost_shift) {
    total = 0;
    for (const TcMset& m : p.ms) total += (uint64_t)m.items * tc_item_cost(m, p.cost_shift);
    if (total < (1ull << 31) || p.cost_shift == 31) break;
  }
  if (total >= (1ull << 31)) return -1;
  p.ctotal = (uint32_t)total;
  return 0;
}

// Scratch of an apply: the split input (samples), the B images (bytes, a 1 KB
// aligned region per launch) and the item lists (items, one after another).
// Between blocks of equal size the windows' offsets move; the slack covers a
// period of the largest row stride and two chunks, two chunks of taps per
// merge set and an eighth for merge sets that fall another way, and twice the
// items, so that few streams' buffers grow after their first block.
struct TcScratch {
  size_t xhl = 0, b = 0, items = 0;
  size_t xhl_slack = 0, b_slack = 0, items_slack = 0;
  std::vector<size_t> b_off, item_off;  // each launch's parts
};
inline TcScratch tc_scratch(const std::vector<TcPlan>& plans) {
  TcScratch s;
  for (const TcPlan& p : plans) {
    s.b_off.push_back(s.b);
    s.item_off.push_back(s.items);
    s.b += (p.b_bytes + 1023u) & ~(size_t)1023u;
    s.items += (size_t)p.items;
    s.xhl = std::max(s.xhl, (size_t)p.xhl_samples);
    for (const TcPlanGroup& g : p.groups) s.xhl_slack = std::max(s.xhl_slack, (size_t)g.D + 2 * kTcChunkTaps);
    for (const TcMset& m : p.ms) s.b_slack += 2 * (size_t)tc_round_up((int64_t)4 * m.NS * 128, 1024);
  }
  s.b_slack += s.b / 8;
  s.items_slack = s.items;
  return s;
}

// Every group in one launch.  Returns 0 on success, -1 when they exceed a
// launch's record limits.
inline int tc_plan(const std::vector<TcGroupIn>& gin, int64_t N, int H, int num_sms, TcPlan& p) {
  p = TcPlan();
  TcGroupPlan q;
  for (const TcGroupIn& g : gin) {
    if (g.slots.empty()) continue;
    if (tc_plan_group(g, H, 0, q) != 0) return -1;
    if (!q.ms.empty() && !tc_append(p, q)) return -1;
  }
  return tc_finish(p, N, H, num_sms);
}

// Item range [first, last) of merge set m were each CTA to own an equal range of
// input samples (the kernel cuts the item list by cost instead).
FDSP_HD inline void tc_item_range(int64_t a, int64_t P, int64_t items, int64_t Lc, int b, int G, int64_t* first,
                          int64_t* last) {
  const int64_t v0 = (int64_t)b * Lc - a, v1 = (int64_t)(b + 1) * Lc - a;
  int64_t f = v0 <= 0 ? 0 : (v0 + P - 1) / P;
  int64_t l = v1 <= 0 ? 0 : (v1 + P - 1) / P;
  *first = f < items ? f : items;
  *last = (b == G - 1) ? items : (l < items ? l : items);
}

}  // namespace fdsp
