// The sharing rule of the streaming kernel (gv_stream_schedule.h), played through on the host: some of the grid's
// CTAs run, the others start only when those have ended.  Arguments: chunks, CTAs, running CTAs, seed.  Prints "ok" if
// every wait of a running CTA ends and every item is done once, else what went wrong.
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <random>
#include <vector>

#include "../gevva_b200/csrc/gv_stream_schedule.h"

// A claim from the pool: the counter's answer, which the claimer has when it looks at it and not before.
struct Claim {
  int value;
  std::shared_ptr<bool> looked_at;
  Claim(int v) : value(v), looked_at(std::make_shared<bool>(true)) {}
  static Claim issued(int v) {
    Claim c(v);
    *c.looked_at = false;
    return c;
  }
  operator int() const {
    *looked_at = true;
    return value;
  }
};

int main(int, char** argv) {
  const int chunks = std::atoi(argv[1]), ctas = std::atoi(argv[2]), running = std::atoi(argv[3]);
  std::mt19937 rng(static_cast<unsigned>(std::atoi(argv[4])));
  const gv::StreamShares shares(chunks, ctas);
  int counter = 0, pool_counter = 0, ups_done = 0, downs_done = 0;
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
    // the w2 items, as the claim warps walk over them
    std::vector<gv::StreamDownWalk<Claim>> walks;
    std::vector<std::shared_ptr<bool>> claims;
    for (int c = first; c < last; ++c) walks.emplace_back(shares, turn[c]);
    auto claim = [&] {
      const Claim c = Claim::issued(pool_counter++);
      claims.push_back(c.looked_at);
      return c;
    };
    while (!walks.empty()) {
      const size_t pick = rng() % walks.size();
      auto& walk = walks[pick];
      if (walk.asks()) {
        walk.next = claim();
        walk.after = claim();
      }
      const int item = walk.item();
      if (item < 0) {
        if (!walk.answered()) return std::puts("a negative claim"), false;
        walks.erase(walks.begin() + static_cast<long>(pick));
        continue;
      }
      if (item >= shares.down || down[item]++) return std::puts("a w2 item twice or out of range"), false;
      ++downs_done;
      if (walk.advance()) walk.after = claim();
    }
    for (const auto& looked_at : claims)
      if (!*looked_at) return std::puts("a CTA ended with a claim in flight"), false;
    return true;
  };
  if (!play(0, running) || (running < ctas && !play(running, ctas))) return 0;
  std::puts(downs_done == shares.down ? "ok" : "w2 items left over");
  return 0;
}
