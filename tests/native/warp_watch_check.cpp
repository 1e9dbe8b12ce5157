// Host check that watch_ready (common.cuh) keeps a warp together: 32 threads
// stand for the lanes, and a full-mask operation (any, ballot, sync) completes
// only when all 32 have come to the same one. The word done() reads turns true
// for some lanes a poll before the others, as when another warp stores it
// between two lanes' reads. A loop in which each lane goes by its own value
// must be caught by the check (lanes in a ballot wait for lanes that have
// left); watch_ready must return the same lanes on all 32, and after `limit`
// polls when nothing happens. Built and run by tests/test_host.py.
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

enum Op { ANY, BALLOT, SYNC };

// A full-mask operation of 32 lanes: waits until all have come, fails all if
// one comes to another operation or has left for good.
struct Lanes {
  std::mutex m;
  std::condition_variable cv;
  int count = 0, gone = 0;
  long long gen = 0;
  Op op = SYNC;
  unsigned votes = 0, result = 0;
  bool broken = false;

  unsigned meet(int lane, Op o, bool p) {
    std::unique_lock<std::mutex> l(m);
    if (broken) return 0;
    if (gone || (count && op != o)) return fail();
    op = o;
    votes |= (unsigned)p << lane;
    if (++count == 32) {
      result = votes;
      votes = 0;
      count = 0;
      gen++;
      cv.notify_all();
      return result;
    }
    const long long g = gen;
    cv.wait(l, [&] { return gen != g || broken; });
    return broken ? 0 : result;
  }
  void leave() {
    std::unique_lock<std::mutex> l(m);
    if (count) fail();
    gone++;
  }
  unsigned fail() {
    broken = true;
    cv.notify_all();
    return 0;
  }
};

struct LaneWarp {
  Lanes *w;
  int lane;
  bool any(bool p) const { return w->meet(lane, ANY, p) != 0; }
  unsigned ballot(bool p) const { return w->meet(lane, BALLOT, p); }
  void pause() const {}
};

// done() turns true at poll `at` for the lanes of `early` and a poll later for
// the others; ready() at poll `readyAt` for lane 5 (never: -1).
struct Scenario {
  int at;
  unsigned early;
  int readyAt, limit;
};

template <class Watch>
static bool run(const Scenario &sc, Watch watch, std::vector<unsigned> *out) {
  Lanes lanes;
  out->assign(32, ~0u);
  std::vector<std::thread> th;
  for (int lane = 0; lane < 32; lane++)
    th.emplace_back([&, lane] {
      LaneWarp w{&lanes, lane};
      int reads = 0, asks = 0;
      auto done = [&] { return reads++ >= sc.at + !(sc.early >> lane & 1); };
      auto ready = [&] { return lane == 5 && sc.readyAt >= 0 && asks++ >= sc.readyAt; };
      (*out)[lane] = watch(w, lanes, sc.limit, done, ready);
      lanes.meet(lane, SYNC, false);  // what follows: a full-mask synchronisation
      lanes.leave();
    });
  for (auto &t : th) t.join();
  return !lanes.broken;
}

int main() {
  auto vote = [](LaneWarp &w, Lanes &, int limit, auto done, auto ready) { return watch_ready(w, limit, done, ready); };
  auto own = [](LaneWarp &w, Lanes &lanes, int, auto done, auto ready) -> unsigned {
    while (!done()) {
      unsigned r = w.ballot(ready());
      if (lanes.broken) return 0;
      if (r) return r;
    }
    return 0;
  };
  std::vector<unsigned> got;
  int bad = 0;
  const Scenario split = {3, 0x0000ffffu, -1, 1000};
  if (run(split, own, &got)) {
    printf("the per-lane loop was not caught\n");
    bad++;
  }
  const Scenario all[] = {split, {0, 1u, -1, 1000}, {5, 0x80000000u, -1, 1000}, {7, 0u, 2, 1000}, {2, ~1u, 2, 1000}, {1, ~1u, 2, 1000}, {1000, 0u, -1, 20}};
  for (const Scenario &sc : all) {
    bool ok = run(sc, vote, &got);
    // in the poll in which both come, what is ready is returned
    unsigned want = sc.readyAt >= 0 && sc.readyAt <= sc.at + (sc.early == 0) && sc.readyAt < sc.limit ? 1u << 5 : 0;
    for (unsigned g : got) ok = ok && g == want;
    if (!ok) {
      printf("at %d early %08x ready %d limit %d: lanes apart, or %08x instead of %08x\n", sc.at, sc.early, sc.readyAt, sc.limit,
             got[0], want);
      bad++;
    }
  }
  return bad;
}
