// Host check of the warp queue (csrc/warp_queue.cuh): a warp of 32 threads runs the scan
// and batch loop of the direct builds' kernels over tasks of every length, with random
// and extreme survivors.  Prints, per pattern, the tasks, the kets that should survive,
// those taken exactly once, and the faults: kets out of the task's range, slots used
// beyond the queue, lanes that disagree.
#include <array>
#include <atomic>
#include <barrier>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
#define __restrict__

static std::barrier<> warp_bar(32);
static std::array<std::atomic<unsigned>, 2> votes;
static thread_local int my_lane, vote_no;
static void __syncwarp() { warp_bar.arrive_and_wait(); }
static unsigned __ballot_sync(unsigned, bool p) {
  std::atomic<unsigned>& v = votes[vote_no++ & 1];   // the other one is cleared for the next vote
  if (p) v.fetch_or(1u << my_lane);
  warp_bar.arrive_and_wait();
  const unsigned r = v.load();
  if (my_lane == 0) votes[vote_no & 1].store(0);
  warp_bar.arrive_and_wait();
  return r;
}
static int __popc(unsigned x) { return __builtin_popcount(x); }
static int clz(unsigned x) { return x ? __builtin_clz(x) : 32; }
#include "warp_queue.cuh"

int main() {
  using namespace gbhf;
  std::mt19937 rng(3);
  for (int pattern = 0; pattern < 4; ++pattern) {
    constexpr int FIRST = 1000, MOST = 256;
    int q[QUEUE_SLOTS + 32];   // guard slots behind the queue
    std::vector<char> pass(MOST);
    std::vector<std::atomic<int>> taken(MOST);
    std::atomic<int> faults{0};
    long want = 0, once = 0, tasks = 0;
    for (int len = 1; len <= MOST; len += len < 70 ? 1 : 37, ++tasks) {
      for (int i = 0; i < MOST; ++i) {
        pass[i] = i < len && (pattern == 0 || (pattern == 1 && rng() % 2) || (pattern == 2 && rng() % 8 == 0) ||
                              (pattern == 3 && i == len - 1));
        want += pass[i];
        taken[i] = 0;
      }
      for (int& x : q) x = -1;
      votes[0] = votes[1] = 0;
      std::vector<std::thread> lanes;
      for (int t = 0; t < 32; ++t)
        lanes.emplace_back([&, t] {
          my_lane = t;
          vote_no = 0;
          int queued = 0, scanned = 0;
          while (true) {
            while (queued < 32 && scanned < len) {
              const int o = scanned + t;
              queue_push(q, queued, FIRST + o, o < len && pass[o], t);
              scanned += 32;
              if (queued > QUEUE_SLOTS) ++faults;
            }
            if (queued == 0) break;
            const int nk = queued < 32 ? queued : 32, lg = 32 - clz(nk - 1);
            bool keep, bad;
            const int jk = queue_ket(q, nk, lg, t, FIRST, len, keep, bad);
            if (bad || jk < FIRST || jk >= FIRST + len) ++faults;
            if (keep && (t >> lg) == 0 && jk >= FIRST && jk < FIRST + len) ++taken[jk - FIRST];
            queue_pop(q, queued, nk, t);
            if (queued < 0 || queued > 31) ++faults;
          }
        });
      for (auto& l : lanes) l.join();
      for (int i = 0; i < 32; ++i) faults += q[QUEUE_SLOTS + i] != -1;
      for (int i = 0; i < MOST; ++i) {
        once += pass[i] && taken[i] == 1;
        faults += taken[i] != (pass[i] ? 1 : 0);
      }
    }
    std::printf("%d %ld %ld %ld %d\n", pattern, tasks, want, once, faults.load());
  }
  // a ket from outside the task is dropped and reported
  const int q[2] = {1005, 7};
  bool keep, bad;
  const int a = queue_ket(q, 2, 1, 0, 1000, 10, keep, bad);
  std::printf("in %d %d %d\n", a, keep, bad);
  const int b = queue_ket(q, 2, 1, 1, 1000, 10, keep, bad);
  std::printf("out %d %d %d\n", b, keep, bad);
  return 0;
}
