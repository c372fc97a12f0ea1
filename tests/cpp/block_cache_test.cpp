// Host check of the kept device blocks (birp_cpp_gb300/csrc/block_cache.h) with
// a release function that only notes what it is given. Exit code: 1 if a check
// failed.
#include <cstdio>
#include <map>
#include <random>
#include <thread>
#include <vector>

#include "../../birp_cpp_gb300/csrc/block_cache.h"

using birp::BlockCache;

static std::mutex g_mu;
static std::map<void*, int> g_freed;
static void note(void* p) {
  std::lock_guard<std::mutex> lk(g_mu);
  ++g_freed[p];
}
static int fails = 0;
#define CHECK(c)                                          \
  do {                                                    \
    if (!(c)) {                                           \
      ++fails;                                            \
      std::printf("line %d: %s\n", __LINE__, #c);         \
    }                                                     \
  } while (0)

static void* ptr(size_t i) { return reinterpret_cast<void*>((i + 1) << 8); }
static bool freed(size_t i) { return g_freed.count(ptr(i)) != 0; }
constexpr size_t MB = (size_t)1 << 20, MAX = BlockCache::kKeepMax, MIN = BlockCache::kKeepMin;

int main() {
  {  // what is kept at all
    g_freed.clear();
    BlockCache c(note);
    c.give(ptr(0), 16 * MB, 0, true);  // not open
    CHECK(freed(0));
    c.open(1);
    c.give(ptr(1), MIN - 1, 1, true);    // too small
    c.give(ptr(2), MAX + 1, 1, true);    // too large
    c.give(ptr(3), 16 * MB, 1, false);   // still in use
    c.give(ptr(4), 16 * MB, 0, true);    // another device's
    c.give(ptr(5), 16 * MB, -1, true);   // of no device
    c.give(nullptr, 16 * MB, 1, true);
    for (size_t i = 1; i <= 5; ++i) CHECK(freed(i));
    CHECK(g_freed.size() == 6 && c.held() == 0);
    c.give(ptr(6), MIN, 1, true);
    CHECK(!freed(6) && c.held() == MIN);
    c.close();
    CHECK(freed(6) && c.held() == 0);
    c.give(ptr(7), 16 * MB, 1, true);
    CHECK(freed(7));
  }
  {  // what a request gets: the smallest that fits, at most an eighth larger, of its device
    g_freed.clear();
    BlockCache c(note);
    c.open(0);
    c.give(ptr(0), 90 * MB, 0, true);
    c.give(ptr(1), 84 * MB, 0, true);
    c.give(ptr(2), 100 * MB, 0, true);
    size_t b = 80 * MB;
    CHECK(c.take(1, &b) == nullptr && b == 80 * MB);
    CHECK(c.take(0, &b) == ptr(1) && b == 84 * MB);
    b = 80 * MB;
    CHECK(c.take(0, &b) == ptr(0) && b == 90 * MB);
    b = 80 * MB;
    CHECK(c.take(0, &b) == nullptr && b == 80 * MB && c.held() == 100 * MB);
    b = MIN - 1;
    CHECK(c.take(0, &b) == nullptr);
    c.release_all();
    CHECK(freed(2) && c.held() == 0);
    c.give(ptr(3), 90 * MB, 0, true);  // still open
    CHECK(c.held() == 90 * MB);
    c.close();
  }
  {  // the bound: distinct sizes past it, oldest first; as many of the smallest as it holds
    g_freed.clear();
    BlockCache c(note);
    c.open(0);
    const size_t sizes[] = {150, 180, 210, 250, 300, 360, 420, 1000, 1024};
    size_t i = 0, sum = 0;
    std::vector<size_t> kept;
    for (size_t s : sizes) {
      c.give(ptr(i), s * MB, 0, true);
      kept.push_back(i);
      sum += s * MB;
      while (sum > MAX) {
        CHECK(freed(kept.front()));
        sum -= sizes[kept.front()] * MB;
        kept.erase(kept.begin());
      }
      for (size_t k : kept) CHECK(!freed(k));
      CHECK(c.held() == sum && sum <= MAX);
      ++i;
    }
    c.release_all();
    g_freed.clear();
    for (size_t k = 0; k < 300; ++k) c.give(ptr(k), MIN, 0, true);
    CHECK(c.held() <= MAX && c.held() + MIN > MAX && g_freed.size() == 300 - MAX / MIN && freed(0) && !freed(299));
    c.close();
    CHECK(g_freed.size() == 300);
  }
  {  // threads: no block twice, none lost
    g_freed.clear();
    BlockCache c(note);
    c.open(0);
    std::vector<std::thread> th;
    for (int t = 0; t < 4; ++t)
      th.emplace_back([&, t] {
        std::mt19937 rng(t);
        std::vector<std::pair<void*, size_t>> mine;
        for (size_t k = 0; k < 20000; ++k) {
          size_t b = MIN + (rng() % 64) * MB;
          if (rng() % 2 || mine.empty()) {
            void* p = c.take(0, &b);
            mine.push_back({p ? p : ptr((size_t)t * 100000 + k), b});
          } else {
            c.give(mine.back().first, mine.back().second, 0, true);
            mine.pop_back();
          }
          if (rng() % 1000 == 0) c.release_all();
        }
        for (auto& m : mine) c.give(m.first, m.second, 0, true);
      });
    for (auto& x : th) x.join();
    CHECK(c.held() <= MAX);
    c.close();
    for (auto& f : g_freed) CHECK(f.second == 1);
  }
  std::printf("%d failures\n", fails);
  return fails != 0;
}
