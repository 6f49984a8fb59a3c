// waits.cuh -- what follows from a bounded wait that ran out, apart from the hardware: compiled for the host too, where the
// tests run it.
#pragma once
#include <cstdint>

#include "modq.cuh"

namespace alto {

// One warp's part, step by step, in an exchange through two buffers with a barrier each, used in turn (the walk of
// offline.cuh): one thread of the CTA arms the step's barrier for the shares of the other CTAs, every warp sends its own,
// and every warp waits for the step's phase.  Once a wait has run out the warp arms, sends and waits for nothing more: the
// phase whose shares are missing stays open, and arming it again two steps later would be an arrival that no phase
// expects.  The other CTAs then miss this one's shares and stop in the same way, each after at most one full wait, so that
// a barrier sees at most the shares of the steps until then.
struct ShareTurns {
  int buf = 0;           // the step's buffer and barrier
  uint32_t parity = 0;   // of the phase that the step waits for: alternates each time a barrier comes round
  bool live = true;

  template <class F> ALTO_HD void arm(F f) const {
    if (live) f(buf);
  }
  template <class F> ALTO_HD void send(F f) const {
    if (live) f(buf);
  }
  // f(buffer, parity) waits: false when the wait ran out
  template <class F> ALTO_HD void wait(F f) {
    if (live) live = f(buf, parity);
  }
  ALTO_HD void next() {
    buf ^= 1;
    parity ^= (uint32_t)(buf ^ 1);
  }
};

}  // namespace alto
