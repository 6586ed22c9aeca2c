// How the CTAs of the streaming kernel (experts_stream.cu) share out its items, in a form that also compiles for
// the host (tests/stream_schedule_probe.cpp).
//
// A w2 item has to wait for the w13 items of its expert, so no w13 item may lie with a CTA that is not running:
// another stream's kernels can hold back a part of the grid for as long as they like, and two such grids could
// each hold some SMs and wait for the rest.  Hence every CTA marks its own first w13 item, the one of its number, as
// taken when it starts, and claims further ones one by one from a counter.  When they are exhausted it
// looks at the marks: a first item that is still not taken after a while it takes itself, and when none is left
// it goes on to its share of the w2 items, which nobody waits for.  Then all w13 items lie with CTAs that run, in
// front of any w2 item of theirs, and every wait ends.  (First items by the counter too: 0.8 to 2.2 us a layer, as the
// grid's claims of one address take that long.)
#pragma once

#include "gv_transcendentals.h"

namespace gv {

// Counters of the streaming kernel (RoutePlan::stream_sync), zero on entry and on exit.  The claims lie 128 bytes
// from the others, which are polled.
constexpr int kStreamQuantised = 0;     // CTAs that have quantised their tokens
constexpr int kStreamFinished = 1;      // CTAs at their end
constexpr int kStreamRescued = 2;       // tokens quantised in place of CTAs that are not running
constexpr int kStreamItemClaims = 32;
constexpr int kStreamRescueClaims = 33;
constexpr int kStreamDownClaims = 34;
constexpr int kStreamFirsts = 64;       // per CTA: its first w13 item is taken
constexpr int kStreamMaxCtas = 256;
constexpr int kStreamSyncInts = kStreamFirsts + kStreamMaxCtas;

constexpr int kStreamUpItems = 11;      // w13 items (64 intermediate columns) of a chunk
constexpr int kStreamDownItems = 22;    // w2 items (128 output columns)

// A pool of each share's last three w2 items (ends the launch evenly, see experts_stream.cu), from eight items a share on: with a
// pool of two from six on, 8 tokens took 41.45 us a layer instead of 41.3.
constexpr int kStreamPooled = 3, kStreamLongShare = 8;

struct StreamShares {
  int ctas, up, down, firsts;  // w13 items 0 .. firsts - 1 are CTAs' first ones, firsts .. up - 1 are claimed
  int lacking, pre;            // this many CTAs get one w13 item less than the others; each takes `pre` w2 items first

  GV_HD_MEMBER StreamShares(int chunks, int grid) {
    ctas = grid;
    up = chunks * kStreamUpItems;
    down = chunks * kStreamDownItems;
    firsts = up < ctas ? up : ctas;
    lacking = up % ctas == 0 ? 0 : ctas - up % ctas;
    pre = lacking > 0 && down >= 4 * lacking + 4 * ctas ? 4 : 0;  // a short list is spread evenly instead
  }
  // CTAs are given w2 items by turns, 0 .. ctas - 1, of which the first `lacking` are meant for the CTAs that get a w13
  // item less: where items are claimed, the order in which CTAs find them exhausted (the n-th claim, n >= up - firsts,
  // is turn n - (up - firsts)), else a fixed one.
  GV_HD_MEMBER int fixed_turn(int cta) const { return cta < up ? lacking + cta : cta - up; }
  GV_HD_MEMBER int down_count(int turn) const {
    const int rest = down - pre * lacking;
    return (turn < lacking ? pre : 0) + (rest > turn ? (rest - 1 - turn) / ctas + 1 : 0);
  }
  GV_HD_MEMBER int down_item(int turn, int k) const {
    if (turn < lacking) {
      if (k < pre) return turn + k * lacking;
      k -= pre;
    }
    return pre * lacking + turn + k * ctas;
  }
  // The last w2 items of every share go to whoever comes for them, where the smallest share has some to spare.
  GV_HD_MEMBER int pooled() const { return down - pre * lacking >= kStreamLongShare * ctas ? kStreamPooled : 0; }
  // The j-th of them, one of each share after the other.
  GV_HD_MEMBER int pool_item(int j) const {
    const int turn = j % ctas;
    return down_item(turn, down_count(turn) - kStreamPooled + j / ctas);
  }
};

// A CTA's walk over its w2 items: its share but for the pooled ones, then what it claims from the pool.  A claim takes as long as an
// item, so two are on their way at a time, the first two with the last item of the share.  The walk ends with the first answer that lies
// behind the pool; the other claim's is looked at by `answered`, without which a CTA must not end (a claim in flight could arrive behind the zeros of the
// CTA that finishes last, and the next launch would leave an item out).
// Index: int, or in a test a type that notices when it is looked at.
template <class Index>
struct StreamDownWalk {
  StreamShares shares;
  int turn, pool, share;  // `share`: items of the CTA's own
  int k = 0;
  Index next, after;      // claims

  GV_HD_MEMBER StreamDownWalk(const StreamShares& s, int t) : shares(s), turn(t), pool(s.pooled() * s.ctas), share(s.down_count(t) - s.pooled()), next(pool), after(pool) {}
  GV_HD_MEMBER bool asks() const { return pool > 0 && (k + 1 == share || (k == 0 && share == 0)); }  // for `next` and `after`
  GV_HD_MEMBER int item() const { return k < share ? shares.down_item(turn, k) : next < pool ? shares.pool_item(next) : -1; }
  // To the item behind this one; true where `after` is to be claimed anew.
  GV_HD_MEMBER bool advance() {
    if (k++ < share) return false;
    next = after;
    return after < pool;
  }
  GV_HD_MEMBER bool answered() const { return next >= 0 && after >= 0; }
};

// A bounded wait of a thread that others rely on: until ready(), with pause() between two looks.  It ends early where stopped(): somebody has given up, and
// reported it.  Past the limit it gives up, and calls report(), but not without another look: the thread itself may be what was not running meanwhile.
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class Ready, class Stopped, class Now, class Pause, class Report>
GV_HD bool stream_wait(long long limit, Ready ready, Stopped stopped, Now now, Pause pause, Report report) {
  const long long start = now();
  for (;;) {
    const bool late = now() - start > limit;
    if (ready()) return true;
    if (stopped()) return false;
    if (late) {
      report();
      return false;
    }
    pause();
  }
}

}  // namespace gv
