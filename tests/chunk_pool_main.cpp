// The pool of kept outputs (eddy_pool.h) over a counting allocator: prints one
// line per check, "ok <what>" or "FAILED <what>".
#include <stdio.h>
#include <string.h>

#include <map>

#include "eddy_pool.h"

namespace {
size_t limit = ~(size_t)0, held = 0, most = 0;  // page-locked bytes
std::map<void *, size_t> blocks;
struct Counting {
  static void *alloc(size_t n) {
    if (held + n > limit) return nullptr;
    void *p = malloc(n);
    blocks[p] = n;
    held += n;
    if (held > most) most = held;
    return p;
  }
  static void release(void *p) {
    held -= blocks.at(p);
    blocks.erase(p);
    free(p);
  }
};
using Pool = eddy::ChunkPool<Counting>;
void check(bool ok, const char *what) { printf("%s %s\n", ok ? "ok" : "FAILED", what); }
constexpr size_t MB = (size_t)1 << 20;
}  // namespace

int main() {
  {
    // outputs of one call after the other, given back each time: what is held
    // does not grow with the calls, whatever their sizes and retries
    Pool p;
    size_t after = 0;
    for (int k = 0; k < 200; k++) {
      const Pool::Mark m = p.mark();
      memset(p.take(300000 + 1000 * (k % 7)), 1, 300000);
      if (k % 3 == 0) p.take(400000);
      p.rewind(m);
      if (k == 20) after = held;
    }
    check(held <= after && held <= 3 * MB, "repeated calls hold a bounded amount");
  }
  check(held == 0, "all given back");
  {
    // the same behind a run's results, which stay as they were
    Pool p;
    uint8_t *kept = p.take(100000);
    memset(kept, 7, 100000);
    for (int k = 0; k < 50; k++) {
      const Pool::Mark m = p.mark();
      memset(p.take(20000 + 30000 * k), 1, 20000 + 30000 * k);
      p.rewind(m);
    }
    uint8_t *more = p.take(500);
    memset(more, 2, 500);
    bool same = true;
    for (int i = 0; i < 100000; i++) same = same && kept[i] == 7;
    check(same, "results outlive the calls after them");
    check(held <= 100000 + 20000 + 30000 * 50 + 2 * Pool::kMinChunk, "one chunk behind them");
  }
  {
    // a large run: page-locked memory up to the bound, ordinary memory past it
    Pool p;
    most = 0;
    std::map<uint8_t *, int> got;
    for (int k = 0; k < 40; k++) {
      uint8_t *x = p.take(10 * MB);
      memset(x, k, 64);
      got[x] = k;
    }
    bool own = got.size() == 40;
    for (auto &x : got) own = own && x.first[0] == x.second && x.first[63] == x.second;
    check(own, "every result has its own room");
    check(most <= Pool::kPinnedBytes && most >= 200 * MB, "page-locked up to the bound");
    p.clear();
    check(held == 0, "a large run is given back");
    p.take(10 * MB);
    check(held >= 200 * MB && held <= Pool::kPinnedBytes, "the next run's room at once");
    p.clear();
    check(held >= 200 * MB && held <= Pool::kPinnedBytes, "one chunk kept");
    const size_t one = held;
    for (int k = 0; k < 20; k++) p.take(10 * MB);
    check(held == one, "and used again");
  }
  {
    // no page-locked memory: ordinary memory, as much as is asked for
    limit = 0;
    Pool p;
    bool all = true;
    for (int k = 0; k < 10; k++) all = all && p.take(MB) != nullptr;
    check(all && held == 0, "ordinary memory where none can be page-locked");
    p.clear();
    check(p.take(1) != nullptr, "after clear");
    limit = ~(size_t)0;
  }
  return 0;
}
