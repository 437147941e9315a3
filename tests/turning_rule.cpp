// The sizes from which stages turn, on the L2 they were measured with.
#include <cstdio>

#include "bhr_internal.h"

using namespace bhr;

static constexpr size_t states(int n, int N, int M) { return static_cast<size_t>(n) * 32 * N * M; }
static int failures = 0;
static void check(bool ok, const char *what) {
  if (!ok) failures++, std::printf("FAILED: %s\n", what);
}

int main() {
  const size_t l2 = 132644864;
  // measured without a gain, and the smallest with one
  check(states(3, 8192, 96) < turn_bytes(l2) && states(3, 7168, 112) < turn_bytes(l2) &&
            states(4, 4096, 144) < turn_bytes(l2), "grids that stay in L2 walk one way");
  check(states(3, 8192, 112) > turn_bytes(l2) && states(4, 4096, 160) > turn_bytes(l2), "larger ones turn");
  check(states(3, 8192, 128) < turn_mixed_bytes(l2) && states(3, 8192, 144) > turn_mixed_bytes(l2),
        "the FP32 stages turn from 8192 x 144 on");
  check(turn_bytes(2 * l2) >= 2 * turn_bytes(l2) && turn_mixed_bytes(2 * l2) >= 2 * turn_mixed_bytes(l2),
        "the sizes grow with the L2");
  for (int tiling : {kTilingBlock8, kTilingBlock16, kTilingPersistent, kTilingRing})
    check(!batch_turns(tiling, states(3, 16384, 256), l2), "batches whose kernels take no direction keep their graph");
  check(batch_turns(kTilingBlock8n, states(3, 8192, 112), l2) && !batch_turns(kTilingBlock8n, states(3, 8192, 96), l2),
        "batches of block8n tiles turn from the same size on as single solves");
  return failures != 0;
}
