// The w2 items of the streaming kernel (gv_stream_schedule.h): shares without their pooled items, and the pool, hold every item once.
// Arguments: chunks, CTAs.  Prints "ok", or what went wrong.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../gevva_b200/csrc/gv_stream_schedule.h"

int main(int, char** argv) {
  const gv::StreamShares shares(std::atoi(argv[1]), std::atoi(argv[2]));
  std::vector<char> done(shares.down);
  int items = 0;
  auto take = [&](int item) {
    if (item < 0 || item >= shares.down || done[item]++) std::exit((std::puts("a w2 item twice or out of range"), 0));
    ++items;
  };
  const int pooled = shares.pooled();
  for (int turn = 0; turn < shares.ctas; ++turn) {
    if (shares.down_count(turn) < pooled) return std::puts("a share shorter than its part of the pool"), 0;
    for (int k = 0; k < shares.down_count(turn) - pooled; ++k) take(shares.down_item(turn, k));
  }
  for (int j = 0; j < pooled * shares.ctas; ++j) take(shares.pool_item(j));
  std::puts(items != shares.down ? "w2 items left over" : "ok");
  return 0;
}
