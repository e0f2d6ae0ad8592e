// Runs the queue of claimed tasks of a CTA pair (csrc/mmoe_pair_queue.h) with a thread per role, on barriers that keep track of what each
// thread knows of the others.  A release or acquire carries knowledge only between threads that are inside its scope, as in the GPU's memory
// model.  A slot that is written while a read of it is not known to be over, or read while the write is not known, counts as a race.
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "../vllm_plugin_b200/csrc/mmoe_pair_queue.h"

using namespace mmoe;

enum Scope { kCta, kCluster };
typedef std::map<int, int> Clock;      // thread -> its latest event that is known
static void join(Clock& a, const Clock& b) {
  for (auto& e : b)
    if (a[e.first] < e.second) a[e.first] = e.second;
}

struct Arrival { int cta; Scope scope; Clock clock; };
struct Barrier {
  uint32_t count = 0, pending = 0, phase = 0;
  int tx = 0;
  std::vector<Arrival> now, last;      // releases of this phase and of the one before
  void settle() {
    if (pending != 0 || tx != 0) return;
    pending = count;
    ++phase;
    last.swap(now);
    now.clear();
  }
};
struct Slot {
  int value = -1, writer = -1, written = 0;
  Clock reads;
};

static std::mutex g_lock;
static std::condition_variable g_changed;
static Barrier g_bar[2][2][kPairQueue];      // [CTA][which][slot]
static Slot g_slot[2][kPairQueue];
static int g_races = 0, g_wrong = 0, g_next_thread = 0;
static Scope g_pair_scope = kCluster;        // kCta: what the checker has to find

struct Port {
  int id, cta;
  Clock clock;
  explicit Port(int cta_) : id(g_next_thread++), cta(cta_) {}
  int tick() { return ++clock[id]; }
  bool wait(PairBarrier which, uint32_t slot, uint32_t parity, Scope scope) {
    std::unique_lock<std::mutex> hold(g_lock);
    Barrier& b = g_bar[cta][which][slot];
    g_changed.wait(hold, [&] { return (b.phase & 1u) != parity; });
    for (const Arrival& a : b.last)
      if (a.cta == cta || (a.scope == kCluster && scope == kCluster)) join(clock, a.clock);
    return true;
  }
  bool wait_own(PairBarrier which, uint32_t slot, uint32_t parity) { return wait(which, slot, parity, kCta); }
  bool wait_pair(PairBarrier which, uint32_t slot, uint32_t parity) { return wait(which, slot, parity, g_pair_scope); }
  void arrive(int at, PairBarrier which, uint32_t slot, Scope scope) {
    std::lock_guard<std::mutex> hold(g_lock);
    tick();
    Barrier& b = g_bar[at][which][slot];
    b.now.push_back(Arrival{cta, scope, clock});
    --b.pending;
    b.settle();
    g_changed.notify_all();
  }
  void arrive_own(PairBarrier which, uint32_t slot) { arrive(cta, which, slot, kCta); }
  void arrive_leader(PairBarrier which, uint32_t slot) { arrive(0, which, slot, g_pair_scope); }
  int read(uint32_t slot) {
    std::lock_guard<std::mutex> hold(g_lock);
    Slot& s = g_slot[cta][slot];
    if (s.writer >= 0 && clock[s.writer] < s.written) ++g_races;
    s.reads[id] = tick();
    return s.value;
  }
  void send(uint32_t slot, int task) {
    for (int to = 0; to < 2; ++to) {
      std::lock_guard<std::mutex> hold(g_lock);
      Barrier& b = g_bar[to][kPairFull][slot];
      tick();
      b.now.push_back(Arrival{cta, g_pair_scope, clock});
      b.tx += 4;
      --b.pending;
      // the asynchronous store: a thread of its own, which knows what the sender knew, and completes the barrier cluster-wide
      Slot& s = g_slot[to][slot];
      Clock store = clock;
      for (auto& r : s.reads)
        if (store[r.first] < r.second) ++g_races;
      if (s.writer >= 0 && store[s.writer] < s.written) ++g_races;
      s.reads.clear();
      s.value = task;
      s.writer = g_next_thread++;
      s.written = 1;
      store[s.writer] = 1;
      b.now.push_back(Arrival{cta, kCluster, store});
      b.tx -= 4;
      b.settle();
      g_changed.notify_all();
    }
  }
};

static void pause_at_random(unsigned* seed) {
  if (rand_r(seed) % 3 == 0) std::this_thread::yield();
  if (rand_r(seed) % 16 == 0) std::this_thread::sleep_for(std::chrono::microseconds(rand_r(seed) % 50));
}

// pair_queue <tasks> <epilogue warps> <seed> <scope of what crosses the pair: cta or cluster>: races, wrong tasks, tasks read
int main(int, char** argv) {
  const int tasks = atoi(argv[1]), epilogue = atoi(argv[2]), seed = atoi(argv[3]);
  g_pair_scope = argv[4][1] == 't' ? kCta : kCluster;
  int taken = 0;
  for (int cta = 0; cta < 2; ++cta)
    for (uint32_t s = 0; s < kPairQueue; ++s) {
      Barrier* b = &g_bar[cta][0][0];
      b[kPairFull * kPairQueue + s].count = b[kPairFull * kPairQueue + s].pending = pair_full_count();
      b[kPairEmpty * kPairQueue + s].count = b[kPairEmpty * kPairQueue + s].pending = pair_empty_count(cta == 0, epilogue + (cta == 0 ? 2 : 1));
    }
  std::vector<std::thread> roles;
  for (int cta = 0; cta < 2; ++cta)
    for (int r = 0; r < epilogue + (cta == 0 ? 2 : 1); ++r)
      roles.emplace_back([&, port = Port(cta), rnd = static_cast<unsigned>(seed * 64 + 32 * cta + r)]() mutable {
        int t = -1;
        for (uint32_t n = 0; t < tasks && pair_take(port, n, &t); ++n) {
          std::unique_lock<std::mutex> hold(g_lock);
          if (t != static_cast<int>(n)) ++g_wrong;
          ++taken;
          hold.unlock();
          pause_at_random(&rnd);
        }
      });
  roles.emplace_back([&, port = Port(0), rnd = static_cast<unsigned>(seed * 64 + 62)]() mutable {
    for (uint32_t n = 0; pair_put(port, n, static_cast<int>(n)) && static_cast<int>(n) < tasks; ++n) pause_at_random(&rnd);
  });
  roles.emplace_back([&, port = Port(1), rnd = static_cast<unsigned>(seed * 64 + 63)]() mutable {
    int t;
    for (uint32_t n = 0; pair_peek(port, n, &t) && t < tasks && pair_forward(port, n); ++n) pause_at_random(&rnd);
  });
  for (auto& r : roles) r.join();
  printf("%d %d %d\n", g_races, g_wrong, taken);
  return 0;
}
