// waits.cuh -- what follows from a bounded wait that ran out, apart from the hardware: compiled for the host too, where the
// tests run it.
#pragma once
#include <cstdint>

#include "modq.cuh"

// What ran out, as recorded in a batch's error word.
enum : uint32_t {
  ALTO_ERR_WAIT_FULL = 1u,    // MMA issuer gave up waiting for a TMA stage
  ALTO_ERR_WAIT_EMPTY = 2u,   // producer gave up waiting for a stage to be released
  ALTO_ERR_WAIT_ACCUM = 4u,   // epilogue gave up waiting for the accumulator
  ALTO_ERR_WAIT_DRAIN = 8u,   // a bail-out drain wait gave up
};

namespace alto {

// The error word is pinned host memory, which the CTAs of a batch write without atomics: every code has a byte of its own,
// so that none hides another.  error_codes: the codes recorded in a word, together.
ALTO_HD void record_error(uint32_t *word, uint32_t code) {
  volatile uint8_t *byte = reinterpret_cast<volatile uint8_t *>(word);
  byte[code == ALTO_ERR_WAIT_FULL ? 0 : code == ALTO_ERR_WAIT_EMPTY ? 1 : code == ALTO_ERR_WAIT_ACCUM ? 2 : 3] = 1;
}
ALTO_HD uint32_t error_codes(uint32_t word) {
  uint32_t codes = 0;
  for (int i = 0; i < 4; ++i) codes |= (uint32_t)((word >> (8 * i) & 0xffu) != 0) << i;
  return codes;
}

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
