// The sharing rule of the streaming kernel (gv_stream_schedule.h), played through on the host: some of the grid's
// CTAs run, the others start only when those have ended.  Arguments: chunks, CTAs, running CTAs, seed.  Prints "ok" if
// every wait of a running CTA ends and every item is done once, else what went wrong.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../gevva_b200/csrc/gv_stream_schedule.h"

int main(int, char** argv) {
  const int chunks = std::atoi(argv[1]), ctas = std::atoi(argv[2]), running = std::atoi(argv[3]);
  std::mt19937 rng(static_cast<unsigned>(std::atoi(argv[4])));
  const gv::StreamShares shares(chunks, ctas);
  int counter = 0, ups_done = 0, downs_done = 0;
  std::vector<char> up(shares.up), down(shares.down), first_taken(ctas);
  std::vector<int> turn(ctas, -1);
  auto do_up = [&](int item) {
    if (up[item]++) return false;
    ++ups_done;
    return true;
  };
  auto play = [&](int first, int last) {
    // whoever is ready next goes on; a CTA's first item is its own unless it was taken while the CTA was not running
    std::vector<int> busy;
    for (int c = first; c < last; ++c) {
      if (!first_taken[c] && c < shares.firsts && !do_up(c)) return std::puts("a first item twice"), false;
      first_taken[c] = 1;
      turn[c] = shares.fixed_turn(c);
      busy.push_back(c);
    }
    while (!busy.empty()) {
      const size_t pick = rng() % busy.size();
      const int cta = busy[pick];
      if (shares.up > shares.ctas) {
        const int item = shares.firsts + counter++;
        if (item < shares.up) {
          if (!do_up(item)) return std::puts("a w13 item twice"), false;
          continue;
        }
        turn[cta] = item - shares.up;
      }
      for (int c = 0; c < shares.firsts; ++c)
        if (!first_taken[c]) {
          first_taken[c] = 1;
          if (!do_up(c)) return std::puts("a first item twice"), false;
        }
      busy.erase(busy.begin() + static_cast<long>(pick));
    }
    // the w2 items of these CTAs wait for w13 items that must all be done by now
    if (ups_done != shares.up) return std::puts("a running CTA waits for one that is not"), false;
    for (int c = first; c < last; ++c) {
      for (int k = 0; k < shares.down_count(turn[c]); ++k) {
        const int item = shares.down_item(turn[c], k);
        if (item < 0 || item >= shares.down || down[item]++) return std::puts("a w2 item twice or out of range"), false;
        ++downs_done;
      }
    }
    return true;
  };
  if (!play(0, running) || (running < ctas && !play(running, ctas))) return 0;
  std::puts(downs_done == shares.down ? "ok" : "w2 items left over");
  return 0;
}
