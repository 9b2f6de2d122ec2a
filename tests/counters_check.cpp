// Check of when a small sort's counters are cleared (gpu-quicksort_gb300/csrc/gqs_counters.h), compiled and run by
// tests/test_counters.py on the CPU: a model of the counters beside the tracker, with launches that succeed, fail before the
// first kernel, or fail with half of the sort enqueued, clearings that fail, captured streams, and new scratch. Every sort that
// was enqueued as a whole must have found the counters zero. Then which scratch is asked for after a refusal. Prints "ok" and exits 0, or the violation and exits 1.
#include <cstdio>
#include <cstdlib>

#include "gqs_counters.h"

int main() {
  gqs::SplitCounters t;
  bool zero = false;  // the counters themselves
  t.spoil();          // as allocated
  std::srand(7);
  long clears = 0, good = 0;
  for (long op = 0; op < 200000; ++op) {
    const int what = std::rand() % 8;
    if (what == 0) {  // new scratch
      zero = false;
      t.spoil();
      continue;
    }
    const bool captured = what == 1;
    const bool clear_fails = what == 2, fails = what == 3, fails_half = what == 4;
    bool graph_clears = false, found_zero = false;
    const bool unclear = t.unclear();
    const int e = t.enqueue<int>(
        [&] { return captured; },
        [&] {
          ++clears;
          if (clear_fails) return 2;
          if (captured) graph_clears = true;
          else zero = true;
          return 0;
        },
        [&] {
          if (fails) return 3;
          found_zero = captured ? graph_clears || zero : zero;
          if (fails_half) {
            zero = false;  // the first kernel has counted, the second, which clears, is missing
            return 4;
          }
          return 0;
        });
    const int want = unclear && clear_fails ? 2 : fails ? 3 : fails_half ? 4 : 0;
    if (e != want) return std::printf("status %d for %d at operation %ld\n", e, want, op), 1;
    if (e == 0 && !found_zero) return std::printf("a sort on counters that are not zero at operation %ld\n", op), 1;
    if (!t.unclear() && !zero) return std::printf("called clear but are not at operation %ld\n", op), 1;
    good += e == 0;
  }
  // a sort that follows a good one clears nothing
  t.enqueue<int>([] { return false; }, [&] { zero = true; return 0; }, [] { return 0; });
  bool again = false;
  t.enqueue<int>([] { return false; }, [&] { again = true; return 0; }, [] { return 0; });
  if (again || !clears || !good) return std::printf("cleared without need\n"), 1;
  // scratch that there was no room for
  gqs::SplitRoom room;
  if (!room.may_hold(0) || !room.may_hold(~(size_t)1)) return std::printf("refused at first\n"), 1;
  room.refuse(1000);
  room.refuse(2000);
  if (room.may_hold(1000) || room.may_hold(2000) || !room.may_hold(999)) return std::printf("refusals not kept\n"), 1;
  room.refuse(1);
  if (room.may_hold(1) || !room.may_hold(0)) return std::printf("a sort without the split was refused\n"), 1;
  room.forget();
  if (!room.may_hold(1000)) return std::printf("a refusal was not forgotten\n"), 1;
  std::printf("ok\n");
  return 0;
}
