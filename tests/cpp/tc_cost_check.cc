// The tensor-core launch's cut of its item list by cost, for calls up to the
// largest block (2^31 - 1 samples), with every sum restated in 64 bits:
//
//   * the launch's total is the sum over all items and stays below 2^31;
//   * walking the list in order of first input sample (ties: the lower merge
//     set), each item has the place it stands at and the cost of all items
//     before it, which grows from item to item;
//   * the CTAs' cuts start at 0, never go back and end at the last item, and
//     no CTA has more than an item's cost above the mean.
//
// Usage: tc_cost_check <channels> <decimation> <taps> <up> <samples>; prints
// "ok <items> <unit> <cost of the work in units of 32 cycles>".
#include <algorithm>
#include <cstdio>
#include <cstdlib>
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
  if (argc != 6) return 2;
  const int nch = std::atoi(argv[1]), D = std::atoi(argv[2]), T = std::atoi(argv[3]), up = std::atoi(argv[4]);
  const int64_t N = std::atoll(argv[5]);
  TcGroupIn in;
  in.D = D;
  in.max_split = 32;
  const int64_t M = (N * up + D - 1) / D;
  for (int r = 0; r < up; ++r)
    for (int c = 0; c < nch; ++c) {
      const int64_t t = (int64_t)r * D;
      in.slots.push_back(TcSlotIn{c, T, up, r, (int)(t % up), t / up, (M - r + up - 1) / up});
    }
  TcPlan p;
  CHECK(tc_plan({in}, N, T - 1, 152, p) == 0);
  uint64_t total = 0, work = 0, most = 0;
  int64_t items = 0;
  for (const TcMset& m : p.ms) {
    const uint64_t c = tc_item_cost(m, p.cost_shift);
    CHECK(c >= 1);
    total += (uint64_t)m.items * c;
    work += (uint64_t)m.items * tc_item_cost(m);
    most = std::max(most, c);
    items += m.items;
  }
  CHECK(items == p.items && total == p.ctotal && total < (1ull << 31));
  // the list, merged from the merge sets' items
  std::vector<uint32_t> before((size_t)items);
  std::vector<int> next(p.ms.size(), 0);
  uint64_t cost = 0;
  for (size_t at = 0; at < before.size(); ++at) {
    int best = -1;
    uint64_t bu = 0;
    for (int m = 0; m < (int)p.ms.size(); ++m) {
      if (next[m] >= p.ms[m].items) continue;
      const uint64_t u = (uint64_t)p.ms[m].a +
                         (uint64_t)next[m] * (uint64_t)p.ms[m].R * kTcRows * (uint64_t)p.groups[p.ms[m].group].D;
      if (best < 0 || u < bu) {
        best = m;
        bu = u;
      }
    }
    uint32_t place = 0;
    tc_item_place(p.ms.data(), (int)p.ms.size(), p.groups.data(), best, next[best], p.cost_shift, &place, &before[at]);
    CHECK(place == at && before[at] == cost);
    cost += tc_item_cost(p.ms[best], p.cost_shift);
    ++next[best];
  }
  CHECK(cost == total);
  size_t done = 0;
  for (int b = 0; b < p.G; ++b) {
    auto cut = [&](int c) {
      return (size_t)(std::lower_bound(before.begin(), before.end(), tc_cost_bound(p.ctotal, c, p.G)) - before.begin());
    };
    CHECK(cut(b) == done && cut(b + 1) >= done);
    const uint64_t lo = done < before.size() ? before[done] : total;
    done = cut(b + 1);
    const uint64_t hi = done < before.size() ? before[done] : total;
    CHECK(hi - lo <= total / (uint64_t)p.G + most + 1);
  }
  CHECK(done == before.size());
  std::printf("ok %lld %d %llu\n", (long long)items, p.cost_shift, (unsigned long long)work);
  return 0;
}
