// The walk's exchange of shares (ShareTurns, waits.cuh) on a model of its mbarriers, with a share that never arrives: every
// CTA's steps come to an end, no barrier is armed that expects no arrival, and none counts more bytes than it can hold.
// With an argument: the codes of an error word.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "waits.cuh"

using namespace alto;

// An mbarrier initialised with a count of 1: a phase completes when its arrival and all its bytes are in.
struct Bar {
  int pending = 1, phase = 0;
  long tx = 0;
  bool bad = false;
  void settle() {
    if (tx <= -(1 << 20) || tx >= (1 << 20)) bad = true;  // the range of the transaction count
    if (!pending && !tx) {
      pending = 1;
      ++phase;
    }
  }
  void arm(long bytes) {  // arrive.expect_tx
    if (!pending) bad = true;  // the phase expects no arrival
    tx += bytes;
    if (pending) --pending;
    settle();
  }
  void receive(long bytes) {
    tx -= bytes;
    settle();
  }
  bool done(uint32_t parity) const { return (uint32_t)(phase & 1) != parity; }
};

struct Rearming : ShareTurns {  // goes on after a wait that ran out
  template <class F> void arm(F f) const { f(buf); }
  template <class F> void send(F f) const { f(buf); }
  template <class F> void wait(F f) {
    if (!f(buf, parity)) live = false;
  }
};

// `steps` steps of C CTAs of W warps in lockstep; CTA `from` loses its copy to CTA `to` of warp `w` in step `at` (at < 0:
// none).  Returns whether the barriers were used as they may be; *live counts the warps still exchanging at the end.
template <class Turns>
bool walk(int C, int W, int steps, int from, int to, int w, int at, int *live) {
  std::vector<std::vector<Bar>> bar(C, std::vector<Bar>(2));
  std::vector<std::vector<Turns>> turn(C, std::vector<Turns>(W));
  for (int s = 0; s < steps; ++s) {
    for (int c = 0; c < C; ++c) turn[c][0].arm([&](int b) { bar[c][b].arm((long)(C - 1) * W * 512); });
    for (int c = 0; c < C; ++c)
      for (int v = 0; v < W; ++v)
        for (int r = 0; r < C; ++r)
          if (r != c) turn[c][v].send([&](int b) {
            if (!(s == at && c == from && r == to && v == w)) bar[r][b].receive(512);
          });
    for (int c = 0; c < C; ++c)
      for (int v = 0; v < W; ++v) {
        turn[c][v].wait([&](int b, uint32_t parity) { return bar[c][b].done(parity); });
        turn[c][v].next();
      }
  }
  bool good = true;
  *live = 0;
  for (int c = 0; c < C; ++c) {
    for (const Bar &b : bar[c]) good = good && !b.bad;
    for (const Turns &t : turn[c]) *live += t.live;
  }
  return good;
}

// Every set of codes, recorded in any order and more than once, is the set that is read.
static int codes() {
  int bad = 0;
  for (uint32_t set = 0; set < 16; ++set)
    for (int last = 0; last < 4; ++last) {
      uint32_t word = 0;
      for (int i = 0; i < 8; ++i) {
        const uint32_t bit = 1u << ((last + 1 + i) % 4);
        if (set & bit) record_error(&word, bit);
      }
      bad += error_codes(word) != set || (set != 0) != (word != 0);
    }
  return bad;
}

int main(int argc, char **) {
  if (argc > 1) {
    const int bad = codes();
    printf("%d\n", bad);
    return bad != 0;
  }
  int bad = 0, live = 0;
  for (int C : {2, 3, 4, 8}) {
    const int W = 16, steps = 1023;
    if (!walk<ShareTurns>(C, W, steps, 0, 0, 0, -1, &live) || live != C * W) ++bad;
    for (int at : {0, 1, 2, 3, 511, steps - 3, steps - 2, steps - 1})
      for (int w : {0, 15}) {
        // the CTA that misses the share stops in that step, the others one step later
        if (!walk<ShareTurns>(C, W, steps, 0, C - 1, w, at, &live)) ++bad;
        if (live != (at == steps - 1 ? (C - 1) * W : 0)) ++bad;
        // the model sees a barrier that is armed again (two steps later)
        if (at + 2 < steps && walk<Rearming>(C, W, steps, 0, C - 1, w, at, &live)) ++bad;
      }
  }
  printf("%d\n", bad);
  return bad != 0;
}
