// Montgomery products and the sums kept below 2^32 (modq.cuh) against 128-bit arithmetic: every pair of a set of edge
// values, then pseudorandom operands.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "modq.cuh"

using namespace alto;

static int bad = 0;
static void check(uint32_t a, uint32_t w) {  // a any 32-bit value, w in [0, Q)
  const uint32_t want = (uint32_t)((unsigned __int128)a * w % kQ32);
  if (mont_q(a, to_mont(w)) != want) ++bad;
  const uint32_t s = lazy_add(a, w), d = lazy_sub(a, w);
  if ((uint64_t)s % kQ32 != ((uint64_t)a + w) % kQ32) ++bad;
  if ((uint64_t)d % kQ32 != ((uint64_t)a % kQ32 + kQ32 - w) % kQ32) ++bad;
  if (canon_q(s) != s % kQ32 || canon_q(d) != d % kQ32) ++bad;
}

int main() {
  std::vector<uint32_t> edge = {0, 1, 2, 12286, 12287, 12288, 65535, 0x7fffffff, 0x80000000u, kQ32 / 2, kQ32 - 12288,
                                kQ32 - 12287, kQ32 - 2, kQ32 - 1, kQ32, kQ32 + 1, 0xfffffffeu, 0xffffffffu};
  for (uint32_t a : edge)
    for (uint32_t w : edge)
      if (w < kQ32) check(a, w);
  uint64_t x = 1;
  for (int i = 0; i < 20000000; ++i) {
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    check((uint32_t)(x >> 32), (uint32_t)((x ^ (x >> 29)) & 0xffffffffu) % kQ32);
  }
  printf("%d\n", bad);
  return bad != 0;
}
