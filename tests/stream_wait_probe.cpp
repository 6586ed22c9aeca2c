// The bounded wait of the streaming kernel's claim warp (gv_stream_schedule.h) on a clock of its own.  Prints "ok", or what went wrong.
#include <cstdio>

#include "../gevva_b200/csrc/gv_stream_schedule.h"

namespace {
struct Play {
  long long clock = 0;
  int looks = 0, reports = 0;
  // The clock goes on by `step` a pause; it is ready from `ready_at` on, and somebody else has given up from `stopped_at` on.
  bool wait(long long limit, long long step, long long ready_at, long long stopped_at) {
    return gv::stream_wait(
        limit, [&] { return ++looks, clock >= ready_at; }, [&] { return clock >= stopped_at; }, [&] { return clock; }, [&] { clock += step; },
        [&] { ++reports; });
  }
};
constexpr long long kNever = 1ll << 60;
}  // namespace

int main() {
  Play at_once, soon, asleep, never, stopped, stopped_asleep;
  if (!at_once.wait(100, 10, 0, kNever) || at_once.looks != 1 || at_once.reports) return std::puts("ready at once"), 0;
  if (!soon.wait(100, 10, 50, kNever) || soon.reports) return std::puts("ready within the limit"), 0;
  // one pause lasts longer than the limit (the thread was not running), and what it waits for happened meanwhile
  if (!asleep.wait(100, 5000, 50, kNever) || asleep.reports) return std::puts("gave up what was there"), 0;
  if (never.wait(100, 10, kNever, kNever) || never.reports != 1 || never.clock > 130) return std::puts("gives up, and says so once"), 0;
  if (stopped.wait(100, 10, kNever, 30) || stopped.reports) return std::puts("ends with the others, whose report stands"), 0;
  if (stopped_asleep.wait(100, 5000, kNever, 30) || stopped_asleep.reports) return std::puts("ends with the others, late"), 0;
  std::puts("ok");
  return 0;
}
