// Model of the warps of a block that take one block-wide maximum after the other with
// one barrier each, under the rules of gpusgdlm_gb300/csrc/max_sets.hpp: every order in
// which the warps' accesses can be served is a sequence of choices "which warp does its
// next access", drawn at random here.
#include <cstdint>
#include <vector>

#include "../gpusgdlm_gb300/csrc/max_sets.hpp"

namespace {
uint64_t next_random(uint64_t &x) {
  x ^= x << 13;
  x ^= x >> 7;
  x ^= x << 17;
  return x;
}
}  // namespace

// `calls` reductions by `warps` warps, warp 0 clears; two_sets: the rule with two sets.
// Warp w's value in reduction c is 1 + (c + w) % warps, so the maximum is `warps`.
// Returns the number of (warp, reduction) pairs that read another value.
extern "C" long max_sets_run(int warps, int calls, int two_sets, uint64_t seed) {
  enum Step { kAdd, kWait, kRead, kClear, kDone };
  struct Warp {
    int call = 0, set = 0;
    Step step = kAdd;
  };
  uint64_t rnd = seed * 0x9E3779B97F4A7C15ull + 1;
  std::vector<int> sets(sgdlm::kMaxSets, 0);
  std::vector<Warp> w(warps);
  int arrived = 0;
  long wrong = 0;
  for (int done = 0; done < warps;) {
    // a warp that runs on for a while is the case that matters: keep it for some steps
    const int q = (int)(next_random(rnd) % (uint64_t)warps);
    for (int burst = (int)(next_random(rnd) % 6); burst >= 0; --burst) {
      Warp &a = w[q];
      if (a.step == kDone || (a.step == kWait)) break;
      if (a.step == kAdd) {
        const int v = 1 + (a.call + q) % warps;
        if (v > sets[a.set]) sets[a.set] = v;
        a.step = kWait;
        if (++arrived == warps) {
          arrived = 0;
          for (Warp &b : w) b.step = kRead;
        }
      } else if (a.step == kRead) {
        if (sets[a.set] != warps) ++wrong;
        a.step = kClear;
      } else {  // kClear
        if (q == 0) sets[two_sets ? a.set ^ 1 : sgdlm::set_to_clear(a.set)] = 0;
        a.set = two_sets ? a.set ^ 1 : sgdlm::set_after(a.set);
        a.step = ++a.call == calls ? kDone : kAdd;
        if (a.step == kDone) ++done;
      }
    }
  }
  return wrong;
}
