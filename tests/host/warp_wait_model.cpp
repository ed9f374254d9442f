// Host model of a consumer warp of the X-steps' stage rings: 32 threads stand
// for its lanes, each with a bounded wait of its own that succeeds or runs out
// per stage.  A stage ends at the warp's barrier, the loop at the CTA's.  Prints, for the vote of gx_warp_wait.h and for lanes that decide
// alone, how many patterns of waits left a lane at a barrier for good.
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
#include "../../difx_b200/csrc/gx_warp_wait.h"

constexpr int kLanes = 32, kStages = 4;

struct Barrier {   // of all lanes; arrive() is false when the others do not come
  std::mutex m;
  std::condition_variable cv;
  int n = 0, gen = 0;
  bool all = true, last = true;
  bool arrive(bool good, bool *agreed)
  {
    std::unique_lock<std::mutex> l(m);
    const int g = gen;
    all = all && good;
    if (++n == kLanes) {
      last = all;
      all = true;
      n = 0;
      gen++;
      cv.notify_all();
    } else if (!cv.wait_for(l, std::chrono::milliseconds(400), [&] { return gen != g; })) {
      return false;
    }
    if (agreed) *agreed = last;
    return true;
  }
};

// wait_ok[lane][stage], abort_seen[lane][stage]; true if every lane reaches the end
static bool run(const std::vector<std::vector<bool>> &wait_ok, const std::vector<std::vector<bool>> &abort_seen, bool vote)
{
  Barrier ballot, warp, cta;
  std::vector<char> done(kLanes, 0);
  std::vector<std::thread> t;
  for (int lane = 0; lane < kLanes; lane++)
    t.emplace_back([&, lane] {
      for (int st = 0; st < kStages; st++) {
        const bool good = wait_ok[lane][st] && !abort_seen[lane][st];
        bool met = true;
        const bool go = gx::warp_goes_on(
            good,
            [&](bool g) {
              if (!vote) return g;
              bool agreed = false;
              met = ballot.arrive(g, &agreed);
              return met && agreed;
            },
            [&] { met = warp.arrive(true, nullptr) && met; });
        if (!met) return;
        if (!go) break;
      }
      done[lane] = cta.arrive(true, nullptr);
    });
  for (auto &x : t) x.join();
  for (char d : done)
    if (!d) return false;
  return true;
}

int main()
{
  int stuck[2] = {0, 0}, patterns = 0;
  std::srand(3);
  for (int k = 0; k < 6; k++) {
    std::vector<std::vector<bool>> ok(kLanes, std::vector<bool>(kStages, true)), ab(kLanes, std::vector<bool>(kStages, false));
    const int st = std::rand() % (kStages - 1);
    for (int lane = 0; lane < kLanes; lane++) {
      if (k % 2 == 0) ok[lane][st] = std::rand() % 3 != 0;        // some lanes' waits run out
      else ab[lane][st] = std::rand() % 3 == 0;                   // some lanes see the flag earlier
      for (int later = st + 1; later < kStages; later++) ab[lane][later] = true;
    }
    patterns++;
    for (int vote = 0; vote < 2; vote++) stuck[vote] += !run(ok, ab, vote == 1);
  }
  std::printf("%d %d %d\n", patterns, stuck[1], stuck[0]);
  return 0;
}
