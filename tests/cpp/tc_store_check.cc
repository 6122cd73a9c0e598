// How the tensor-core planner's slots are stored, on random channel sets: the
// epilogue derives every address of a 32-row block from a slot's flags, and
// the check restates them.
//
//   * a run (kTcRun): its members sit side by side inside one chunk of 8
//     slots, are all the outputs of a row (place = output offset, number =
//     output stride), so rows follow one another without gaps in the warp's
//     scratch, inside its bounds, and the members' row counts never grow;
//   * a quad (kTcQuad): four slots at a multiple of 4 of the same channel with
//     consecutive outputs and rows a multiple of 32 bytes long;
//   * a pair (kTcPair): an even position followed by the next output;
//   * the scratch and the slot table inside the launch's shared memory;
//   * the item list: every item has a place of its own, sorted by first input
//     sample, and the CTAs' cuts by cost partition it, each within an item's
//     cost of the mean.
//
// Usage: tc_store_check <cases>; prints "ok <runs> <quads> <pairs> <singles>".
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <random>
#include <utility>
#include <vector>

#include "fdsp_tc_plan.h"

using namespace fdsp;

#define CHECK(c)                                              \
  do {                                                        \
    if (!(c)) {                                               \
      std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #c); \
      return 1;                                               \
    }                                                         \
  } while (0)

int main(int argc, char** argv) {
  const int cases = argc > 1 ? std::atoi(argv[1]) : 2000;
  std::mt19937_64 rng(99);
  auto U = [&](int64_t lo, int64_t hi) { return (int64_t)(lo + (int64_t)(rng() % (uint64_t)(hi - lo + 1))); };
  long runs = 0, quads = 0, pairs = 0, singles = 0;
  for (int cs = 0; cs < cases; ++cs) {
    TcGroupIn in;
    in.D = (int)U(1, 200);
    in.max_split = 1 << U(0, 5);
    const int64_t N = U(1, 4) == 1 ? U(1, 3000) : U(20000, 2000000);
    int ch = 0, Tmax = 1;
    for (int k = (int)U(1, 3); k > 0; --k) {
      const int up = (int)U(1, 9), phase = (int)U(0, up - 1), xoff = (int)U(0, in.D);
      if (xoff >= N) continue;
      const int64_t M = (int64_t)(((unsigned __int128)up * (uint64_t)(N - xoff) - phase + in.D - 1) / in.D);
      for (int c = (int)U(1, 12); c > 0; --c, ++ch) {
        const int T = (int)U(1, 70);
        Tmax = std::max(Tmax, T);
        for (int r = 0; r < up && r < M; ++r) {
          const int64_t t = phase + (int64_t)r * in.D;
          in.slots.push_back(TcSlotIn{ch, T, up, r, (int)(t % up), xoff + t / up, (M - r + up - 1) / up});
        }
      }
    }
    TcPlan p;
    if (in.slots.empty() || tc_plan({in}, N, Tmax - 1, 152, p) != 0) continue;
    CHECK(p.table_off >= p.stages * p.stage_bytes && p.table_off % 1024 == 0);
    CHECK(p.scratch_off >= p.table_off + (int)p.slots.size() * kTcEpiSlotBytes && p.scratch_off % 1024 == 0);
    CHECK(p.scratch_off + kTcEpiWarps * p.scratch_warp + 1024 <= p.smem && p.smem <= kTcSmemDyn);
    CHECK(p.scratch_warp % 16 == 0 && p.scratch_warp >= kTcEpiRecs);
    std::vector<std::pair<int64_t, int>> list((size_t)p.items, {-1, -1});
    std::vector<uint32_t> before((size_t)p.items, 0);
    uint32_t total = 0, most = 0;
    auto step = [&](const TcMset& m) { return (uint32_t)m.R * (uint32_t)kTcRows * (uint32_t)p.groups[m.group].D; };
    for (int mi = 0; mi < (int)p.ms.size(); ++mi) {
      total += (uint32_t)p.ms[mi].items * tc_item_cost(p.ms[mi]);
      most = std::max(most, tc_item_cost(p.ms[mi]));
      for (int t = 0; t < p.ms[mi].items; ++t) {
        const uint32_t u = (uint32_t)p.ms[mi].a + (uint32_t)t * step(p.ms[mi]);
        uint32_t place = 0, cost = 0;
        for (int k = 0; k < (int)p.ms.size(); ++k) {
          const uint32_t n =
              tc_items_before((uint32_t)p.ms[k].a, step(p.ms[k]), (uint32_t)p.ms[k].items, u + (k < mi ? 1u : 0u));
          place += n;
          cost += n * tc_item_cost(p.ms[k]);
        }
        CHECK(place < list.size() && list[place].second < 0);
        list[place] = {u, mi};
        before[place] = cost;
      }
    }
    for (size_t i = 1; i < list.size(); ++i) CHECK(list[i - 1] < list[i] && before[i - 1] < before[i]);
    size_t next = 0;
    for (int b = 0; b < p.G; ++b) {
      auto cut = [&](int c) {
        return (size_t)(std::lower_bound(before.begin(), before.end(), tc_cost_bound(total, c, p.G)) - before.begin());
      };
      CHECK(cut(b) == next && cut(b + 1) >= next);
      next = cut(b + 1);
      const uint32_t end = next < before.size() ? before[next] : total;
      CHECK(cut(b) == next || end - before[cut(b)] <= total / (uint32_t)p.G + most + 1);
    }
    CHECK(next == list.size());
    for (const TcMset& m : p.ms) {
      const TcSlot* s = &p.slots[m.slot0];
      const int* r = &p.slot_r[m.slot0];
      for (int i = 0; i < m.NS; ++i) {
        if (s[i].J == 0) {
          CHECK(s[i].flags == 0);
          continue;
        }
        if (s[i].flags & kTcRun) {
          const int len = tc_run_len(s[i].flags), pos = tc_run_pos(s[i].flags), first = i - pos;
          CHECK(len >= 3 && len <= 7 && pos < len && first >= 0 && first / 8 == (first + len - 1) / 8);
          CHECK(s[i].U == len && r[i] == pos && s[i].ch == s[first].ch && (s[first].flags & kTcRun));
          CHECK(pos == 0 || (s[i].J <= s[i - 1].J && s[i].J + 1 >= s[i - 1].J));
          CHECK((first % 8) * 256 + (31 * len + len) * 8 <= p.scratch_warp - kTcEpiRecs);
          runs += pos == 0;
        }
        if (s[i].flags & kTcQuad) {
          CHECK(i % 4 == 0 && i + 3 < m.NS && s[i].U % 4 == 0 && r[i] % 4 == 0 && !(s[i].flags & kTcRun));
          for (int k = 1; k < 4; ++k) CHECK(s[i + k].ch == s[i].ch && r[i + k] == r[i] + k && s[i + k].U == s[i].U);
          CHECK(s[i + 3].J <= s[i + 2].J && s[i + 2].J <= s[i + 1].J && s[i + 1].J <= s[i].J);
          ++quads;
        }
        if (s[i].flags & kTcPair) {
          CHECK(i % 2 == 0 && s[i + 1].ch == s[i].ch && r[i + 1] == r[i] + 1 && s[i + 1].J <= s[i].J);
          ++pairs;
        }
        singles += s[i].flags == 0;
      }
    }
  }
  CHECK(runs > 0 && quads > 0 && pairs > 0);
  std::printf("ok %ld %ld %ld %ld\n", runs, quads, pairs, singles);
  return 0;
}
