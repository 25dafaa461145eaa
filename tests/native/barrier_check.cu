// Host-only check of the cooperative kernels' grid barrier (wotg_barrier.cuh): CTAs that
// arrive and poll in random order, each at its own pace, walk the barriers of the
// streamed solver, of the on-the-fly solver and of the batch's loop, with flags that
// single CTAs raise now and then. Every CTA has to find a flag exactly where one was
// raised, and so to take the same branches. Launches nothing.
#include <cstdio>
#include <random>
#include <vector>

#include "wotg_barrier.cuh"

using namespace wotg;

struct Op {
  bool flag, flag2, take;
};

// A kernel's barriers as one CTA meets them; `chance` decides whether this CTA raises a
// flag at this barrier, a and a2 what it found at the last one.
struct Cta {
  int variant, phase = 0, n = 0;
  bool over = false;
  std::vector<int> found;   // what it decided on, in order

  template <class Chance>
  Op next(bool a, bool a2, const Chance& chance) {
    switch (variant) {
      case 0:   // rows | columns | merge (over) [| absorption] [| test]
        if (phase == 3) {
          found.push_back(a);
          ++n;
          phase = a ? 4 : n % 5 == 0 ? 5 : 0;
        } else if (phase == 4) {
          phase = n % 5 == 0 ? 5 : 0;
        } else if (phase > 4) {
          phase = 0;
        }
        if (phase <= 1) return ++phase, Op{false, false, false};
        if (phase == 2) return ++phase, Op{chance(), false, true};
        if (phase == 5) phase = 6;
        return Op{false, false, false};
      case 1:   // per side: half-step | finish (over, redo) [| redo (over)], then [| absorption]
        if (phase == 2) {
          over = over || a;
          found.push_back(a2);
          phase = a2 ? 3 : 4;
        } else if (phase == 3) {
          over = over || a;
          phase = 4;
        }
        if (phase == 4) {
          if (++n % 2 == 0) {
            found.push_back(over);
            phase = over ? 5 : 0;
            over = false;
          } else {
            phase = 0;
          }
        } else if (phase == 6) {
          phase = 0;
        }
        if (phase == 5) return ++phase, Op{false, false, false};
        if (phase == 0) return ++phase, Op{false, false, false};
        if (phase == 1) return ++phase, Op{chance(), chance(), true};
        return Op{chance(), false, true};   // 3: the recompute
      default:   // rows | columns (wants) [| items | check, active [| check pass | test | apply | active]]
        if (phase == 2) {
          found.push_back(a);
          phase = a ? 2 : 0;
        } else if (phase == 4) {
          found.push_back(a);
          found.push_back(a2);
          phase = a ? 4 : 0;
        } else if (phase == 8) {
          found.push_back(a2);
          phase = 0;
        }
        ++phase;
        if (phase == 2) return Op{chance(), false, true};
        if (phase == 4) return Op{chance(), chance(), true};
        if (phase == 8) return Op{false, chance(), true};
        return Op{false, false, false};
    }
  }
};

static int run(int variant, int n, unsigned seed) {
  std::mt19937 rng(seed);
  const unsigned rare = 2 + seed % 4 * 3;
  const auto chance = [&] { return rng() % (rare * n) == 0; };
  std::vector<Cta> cta(n);
  std::vector<BarrierSeen> seen(n, BarrierSeen{(unsigned)n, 0, 0});
  std::vector<Op> op(n);
  std::vector<bool> waits(n, false);
  std::vector<int> at(n, 0);
  std::vector<char> raised(1, 0), raised2(1, 0);   // by barrier
  unsigned long long word = 0;
  for (auto& c : cta) c.variant = variant;
  for (int k = 0; k < n; ++k) op[k] = cta[k].next(false, false, chance);
  // a CTA's pace changes now and then, so that one may read long after the others went on
  std::vector<int> pace(n, 1);
  for (long step = 0; step < 60000; ++step) {
    if (step % 64 == 0)
      for (auto& p : pace) p = 1 + (int)(rng() % 40);
    const int k = (int)(rng() % n);
    if ((int)(rng() % 40) >= pace[k]) continue;
    if (!waits[k]) {
      word += barrier_arrival(op[k].flag, op[k].flag2);
      if ((int)raised.size() <= at[k]) {
        raised.push_back(0);
        raised2.push_back(0);
      }
      raised[at[k]] |= op[k].flag;
      raised2[at[k]] |= op[k].flag2;
      waits[k] = true;
    } else if (barrier_complete(word, seen[k])) {
      bool a, a2;
      const Op was = op[k];
      barrier_pass(word, n, was.take, seen[k], &a, &a2);
      // a flag of this barrier is always found, unless it was found before it (the recompute's)
      if (was.take && variant != 1 && (a != (raised[at[k]] != 0) || a2 != (raised2[at[k]] != 0))) return 1;
      if (was.take && a2 != (raised2[at[k]] != 0)) return 2;
      waits[k] = false;
      ++at[k];
      op[k] = cta[k].next(a, a2, chance);
    }
  }
  // the same decisions, as far as each has come
  for (int k = 1; k < n; ++k) {
    size_t m = cta[k].found.size() < cta[0].found.size() ? cta[k].found.size() : cta[0].found.size();
    for (size_t t = 0; t < m; ++t)
      if (cta[k].found[t] != cta[0].found[t]) return 3;
  }
  return at[0] < 100 ? 4 : 0;   // a barrier that nobody completes any more
}

int main() {
  int cases = 0;
  for (int variant = 0; variant < 3; ++variant)
    for (int n : {1, 2, 3, 5, 13})
      for (unsigned seed = 1; seed <= 40; ++seed) {
        const int r = run(variant, n, seed);
        ++cases;
        if (r) {
          std::printf("FAIL variant=%d ctas=%d seed=%u code=%d\n", variant, n, seed, r);
          return 1;
        }
      }
  std::printf("ok %d\n", cases);
  return 0;
}
