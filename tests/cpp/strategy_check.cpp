// Host checks of strategy.h: the untuned rule over commands on standard input,
// and the growth of the split-K partial buffer with an allocator that counts
// and can fail.  "rule SMS N K BATCH FUSED SPLIT" answers "MODE SPLITS BYTES",
// "bound N K BATCH" the bytes that cover every shape up to that one, "fp4 PAIRS N
// KBLOCKS BATCH SPLIT" the NVFP4 kernel's store mode.
#include <cstdio>
#include <cstring>
#include <map>

#include "strategy.h"

using namespace ftdx;

#define CHECK(x)                                               \
  do {                                                         \
    if (!(x)) {                                                \
      std::printf("line %d: %s\n", __LINE__, #x);              \
      return 1;                                                \
    }                                                          \
  } while (0)

namespace {
struct Heap {
  std::map<uint8_t*, size_t> live;
  size_t limit = ~size_t(0), used = 0, next = 4096;
  int allocs = 0;
  uint8_t* alloc(size_t n) {
    ++allocs;
    if (used + n > limit) return nullptr;
    uint8_t* p = reinterpret_cast<uint8_t*>(next);
    next += n;
    live[p] = n;
    used += n;
    return p;
  }
  void free(uint8_t* p) {
    used -= live.at(p);
    live.erase(p);
  }
};

int partials() {
  Heap heap;
  auto alloc = [&](size_t n) { return heap.alloc(n); };
  auto drop = [&](uint8_t* p) { heap.free(p); };
  Partials p;
  CHECK(p.grow(1000, alloc, drop) && p.cap == 1000);
  uint8_t* first = p.ptr;
  CHECK(p.grow(900, alloc, drop) && p.ptr == first && heap.allocs == 1);
  // not captured: replaced and freed
  CHECK(p.grow(2000, alloc, drop) && heap.live.size() == 1 && p.cap == 2000);
  // captured: the buffer outlives its replacement
  uint8_t* in_graph = p.ptr;
  p.captured = true;
  CHECK(p.grow(2100, alloc, drop) && p.ptr != in_graph && heap.live.count(in_graph));
  CHECK(!p.captured && p.cap == 3000 && p.held.size() == 1);
  // captured again and again: what is held stays below twice the last buffer
  for (int i = 0; i < 20; ++i) {
    p.captured = true;
    CHECK(p.grow(p.cap + 1, alloc, drop));
    CHECK(heap.used <= 3 * p.cap);
  }
  CHECK(heap.live.count(in_graph));
  // no room for the larger one: a captured buffer stays
  uint8_t* last = p.ptr;
  const size_t cap = p.cap;
  p.captured = true;
  heap.limit = heap.used + cap / 2;
  CHECK(!p.grow(cap + 1, alloc, drop));
  CHECK(p.ptr == last && p.cap == cap && p.captured && heap.live.count(last));
  // room for what is needed, not for half as much again
  heap.limit = heap.used + cap + 8;
  CHECK(p.grow(cap + 8, alloc, drop) && p.cap == cap + 8 && heap.live.count(last));
  // what was refused is remembered, and more than it; less is not, nor what fits
  heap.limit = heap.used;
  const size_t now = p.cap;
  CHECK(!p.grow(3 * now, alloc, drop) && p.cap == now && p.ptr);
  const int tries = heap.allocs;
  CHECK(p.hopeless(3 * now) && p.hopeless(4 * now) && !p.hopeless(2 * now) && !p.hopeless(now));
  CHECK(heap.allocs == tries);
  // a smaller one that fits does not make it forget, a larger one does
  heap.limit = ~size_t(0);
  CHECK(p.grow(2 * now, alloc, drop) && p.hopeless(3 * now));
  CHECK(p.grow(3 * now, alloc, drop) && !p.hopeless(4 * now));
  p.release(drop);
  CHECK(heap.live.empty() && heap.used == 0 && !p.ptr && p.cap == 0 && p.held.empty());
  return 0;
}

// 512 x 8192 x 4 and x 2: split by the rule, unsplit where the partials cannot be had
int fallback() {
  int asked = 0;
  auto yes = [&](int sp) { return asked = sp, true; };
  auto no = [&](int sp) { return asked = sp, false; };
  for (int b : {4, 2})
    for (bool fused : {false, true}) {
      const Strategy s = untuned_choice(148, 512, 8192, b, fused, true, yes);
      CHECK(s.splits > 1 && s.splits == asked);
      CHECK(s == auto_strategy(148, 512, 8192, b, fused, true));
      const Strategy u = untuned_choice(148, 512, 8192, b, fused, true, no);
      CHECK(u == auto_strategy(148, 512, 8192, b, fused, false) && u.splits == 1);
    }
  asked = 0;  // nothing is asked for where the rule does not split
  CHECK(untuned_choice(148, 2048, 1024, 16, true, true, no).splits == 1 && asked == 0);
  return 0;
}

// a promotion's blocks are all resident at once unless 32 pieces per thread are not enough
int promotion() {
  for (int chunks : {8, 16, 24, 64, 128, 250, 256, 512, 8192, 10000})
    for (int64_t rows = 1; rows < 3000000; rows += 1 + rows / 7) {
      const int64_t r = promotion_rows_per_block(rows, chunks), blocks = (rows + r - 1) / r;
      CHECK(r >= 1 && (r == 1 || r * chunks <= 8192));
      CHECK(blocks <= kPromotionBlocks || (r + 1) * chunks > 8192);
      CHECK(r * chunks >= 256 || chunks > 8192);
      CHECK((r - 1) * chunks < 256 || (rows + r - 2) / (r - 1) > kPromotionBlocks);  // no larger than it must
    }
  return 0;
}
}  // namespace

int main() {
  if (partials() || fallback() || promotion()) return 1;
  char cmd[16];
  while (std::scanf("%15s", cmd) == 1) {
    if (!std::strcmp(cmd, "rule")) {
      int sms, n, k, b, f, s;
      if (std::scanf("%d %d %d %d %d %d", &sms, &n, &k, &b, &f, &s) != 6) return 2;
      const Strategy st = auto_strategy(sms, n, k, b, f != 0, s != 0);
      std::printf("%d %d %zu\n", st.store_mode, st.splits,
                  st.splits > 1 ? split_bytes(n, b, st.splits) : size_t(0));
    } else if (!std::strcmp(cmd, "bound")) {
      int n, k, b;
      if (std::scanf("%d %d %d", &n, &k, &b) != 3) return 2;
      std::printf("%zu\n", most_split_bytes(n, k, b));
    } else if (!std::strcmp(cmd, "fp4")) {
      int pairs, n, kb, b, s;
      if (std::scanf("%d %d %d %d %d", &pairs, &n, &kb, &b, &s) != 5) return 2;
      std::printf("%d\n", fp4_strategy(pairs, n, kb, b, s != 0).store_mode);
    }
  }
  return 0;
}
