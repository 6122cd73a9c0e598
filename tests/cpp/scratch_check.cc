// Scratch buffers that grow (fdsp_pool.h: grow_scratch) and their sizes
// (fdsp_tc_plan.h: tc_scratch).
//
//   * a buffer that grows waits for the work queued so far before its range
//     goes back to the pool, keeps the range when the wait fails, waits for
//     nothing on its first allocation, and takes the exact size where the
//     slack does not fit;
//   * two owners in one pool: work of one queued on its old range is done
//     before the other can be given any byte of it;
//   * a stream of equal blocks of random channel sets keeps its first block's
//     buffers.
//
// Usage: scratch_check <sets>; prints "ok <streams> <blocks> <streams that grew>".
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "fdsp_pool.h"
#include "fdsp_tc_plan.h"

using namespace fdsp;

#define CHECK(c)                                              \
  do {                                                        \
    if (!(c)) {                                               \
      std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #c); \
      return 1;                                               \
    }                                                         \
  } while (0)

// An owner in the pool: pending is the range that queued work still reads.
struct Owner {
  RangePool* pool;
  char* p = nullptr;
  size_t cap = 0, pending = RangePool::kNone, pending_bytes = 0;
  int waits = 0, wait_status = 0;
  int grow(size_t need, size_t slack) {
    return grow_scratch(
        &p, &cap, need, slack,
        [&]() {
          ++waits;
          if (wait_status == 0) pending = RangePool::kNone;
          return wait_status;
        },
        [&](char* q) { pool->release((size_t)(q - static_cast<char*>(nullptr)) - 4096); },
        [&](char** q, size_t n) {
          const size_t off = pool->alloc(n);
          if (off == RangePool::kNone) return -3;
          *q = static_cast<char*>(nullptr) + 4096 + off;  // (never read: offsets stand for addresses)
          return 0;
        });
  }
  size_t off() const { return (size_t)(p - static_cast<char*>(nullptr)) - 4096; }
};

int main(int argc, char** argv) {
  const int sets = argc > 1 ? std::atoi(argv[1]) : 300;
  {
    RangePool pool;
    pool.init(1 << 20);
    Owner a{&pool}, b{&pool};
    CHECK(a.grow(1000, 24) == 0 && a.cap == 1024 && a.waits == 0);
    CHECK(a.grow(1024, 500) == 0 && a.cap == 1024 && a.waits == 0);
    a.pending = a.off();
    a.pending_bytes = a.cap;
    a.wait_status = -4;
    const char* old = a.p;
    CHECK(a.grow(5000, 0) == -4 && a.p == old && a.cap == 1024 && a.waits == 1);  // nothing was released
    a.wait_status = 0;
    CHECK(a.grow(5000, 0) == 0 && a.cap == 5000 && a.waits == 2 && a.pending == RangePool::kNone);
    CHECK(a.grow((1 << 20) - 4096, 1 << 20) == 0 && a.cap == (1 << 20) - 4096);  // without the slack
    CHECK(a.grow(1 << 21, 1 << 20) == -3 && a.p == nullptr && a.cap == 0);
    CHECK(a.grow(256, 0) == 0);
    // owners in turn: no range is given out while queued work reads it
    std::mt19937 rng(7);
    for (int i = 0; i < 20000; ++i) {
      Owner& o = (rng() & 1) ? a : b;
      Owner& other = &o == &a ? b : a;
      if (o.cap > (1 << 18)) {  // closed and opened again (after a wait)
        o.pending = RangePool::kNone;
        pool.release(o.off());
        o.p = nullptr;
        o.cap = 0;
      }
      CHECK(o.grow(o.cap + rng() % 3000, rng() % 300) == 0);
      if (other.pending != RangePool::kNone && o.cap > 0)
        CHECK(o.off() + o.cap <= other.pending || o.off() >= other.pending + other.pending_bytes);
      if (o.cap > 0) {
        o.pending = o.off();
        o.pending_bytes = o.cap;
      }
    }
  }
  std::mt19937_64 rng(5);
  auto U = [&](int64_t lo, int64_t hi) { return (int64_t)(lo + (int64_t)(rng() % (uint64_t)(hi - lo + 1))); };
  int streams = 0, blocks = 0, grew = 0;
  for (int s = 0; s < sets; ++s) {
    struct Class {
      int up, T, nch;
      uint64_t phase, xoff;
    };
    const int D = (int)U(1, 320), max_split = 32;
    const int64_t N = U(4096, 400000);
    std::vector<Class> cls;
    int H = 0;
    for (int k = (int)U(1, 3); k > 0; --k) {
      cls.push_back({(int)U(1, 5), (int)U(1, 70), (int)U(1, 12), 0, 0});
      H = std::max(H, cls.back().T - 1);
    }
    size_t xhl = 0, b = 0, items = 0;
    bool any = false;
    int split = 0;
    for (int blk = 0; blk < 12; ++blk) {
      TcGroupIn in;
      in.D = D;
      in.max_split = max_split;
      int ch = 0;
      for (Class& c : cls) {
        if ((int64_t)c.xoff >= N) continue;
        const uint64_t M = ((uint64_t)c.up * (uint64_t)(N - (int64_t)c.xoff) - c.phase + (uint64_t)D - 1) / (uint64_t)D;
        for (int i = 0; i < c.nch; ++i, ++ch)
          for (uint64_t r = 0; r < (uint64_t)c.up && r < M; ++r) {
            const uint64_t t = c.phase + r * (uint64_t)D;
            in.slots.push_back(TcSlotIn{ch, c.T, c.up, (int)r, (int)(t % (uint64_t)c.up),
                                        (int64_t)(c.xoff + t / (uint64_t)c.up), (int64_t)((M - r + c.up - 1) / c.up)});
          }
        const uint64_t t = c.phase + M * (uint64_t)D;
        c.phase = t % (uint64_t)c.up;
        c.xoff = c.xoff + t / (uint64_t)c.up - (uint64_t)N;
      }
      TcGroupPlan gp;
      std::vector<TcPlan> plans(1);
      if (in.slots.empty() || tc_plan_group(in, H, split, gp) != 0 || gp.ms.empty() || !tc_append(plans[0], gp) ||
          tc_finish(plans[0], N, H, 152) != 0)
        continue;
      split = gp.g.S;
      const TcScratch sc = tc_scratch(plans);
      CHECK(sc.b_off.size() == 1 && sc.b_off[0] == 0 && sc.item_off[0] == 0);
      CHECK(sc.xhl == (size_t)plans[0].xhl_samples && sc.b >= plans[0].b_bytes && sc.items == (size_t)plans[0].items);
      ++blocks;
      if (!any) {
        ++streams;
        xhl = sc.xhl + sc.xhl_slack;
        b = sc.b + sc.b_slack;
        items = sc.items + sc.items_slack;
        any = true;
      } else if (sc.xhl > xhl || sc.b > b || sc.items > items) {
        ++grew;
        break;
      }
    }
  }
  std::printf("ok %d %d %d\n", streams, blocks, grew);
  return 0;
}
