// The launch shape of the kernels whose units take a cluster (split_launch.h):
// what is asked for, and what a CTA accepts.
#include <cstdio>
#include <initializer_list>

#include "split_launch.h"

static int fails = 0;
#define EXPECT(c)                                     \
  do {                                                \
    if (!(c)) {                                       \
      std::printf("line %d: %s\n", __LINE__, #c);     \
      ++fails;                                        \
    }                                                 \
  } while (0)

int main() {
  using namespace mprgp;
  const int qs[] = {1, 2, 4, 8};
  for (int q : qs) {
    SplitLaunch L;
    split_launch(L, q, 6 * q, 128, 4096, nullptr);
    EXPECT(L.cfg.gridDim.x == (unsigned)(6 * q) && L.cfg.blockDim.x == 128);
    EXPECT(L.cfg.dynamicSmemBytes == 4096 && L.cfg.attrs == L.at);
    bool cluster = false, coop = false;
    for (unsigned i = 0; i < L.cfg.numAttrs; ++i) {
      if (L.cfg.attrs[i].id == cudaLaunchAttributeCooperative && L.cfg.attrs[i].val.cooperative)
        coop = true;
      if (L.cfg.attrs[i].id == cudaLaunchAttributeClusterDimension) {
        cluster = true;
        EXPECT(L.cfg.attrs[i].val.clusterDim.x == (unsigned)q);
        EXPECT(L.cfg.attrs[i].val.clusterDim.y == 1 && L.cfg.attrs[i].val.clusterDim.z == 1);
      }
    }
    EXPECT(cluster == (q > 1));
    EXPECT(!(cluster && coop));  // a tool may relaunch a cooperative kernel without its clusters
    // the shape asked for is accepted, and no other
    EXPECT(split_shape_ok(q, 6, 128, q, 6 * q, 128));
    for (int seen : qs)
      if (seen != q) EXPECT(!split_shape_ok(q, 6, 128, seen, 6 * q, 128));
    EXPECT(!split_shape_ok(q, 6, 128, q, 6 * q + q, 128));  // a unit past the list
    EXPECT(!split_shape_ok(q, 6, 128, q, 6 * q, 160));
  }
  EXPECT(!split_shape_ok(0, 6, 128, 0, 0, 128));
  // a phase counter before, at and past its target, also where it wraps
  for (int per : {1, 2, 16, 70, 1360, 4096})
    for (long long phase : {0LL, 1LL, 1002LL, (1LL << 31) / per, (1LL << 32) / per - 1,
                            (1LL << 32) / per, (1LL << 32) / per + 1, 2147483646LL}) {
      if (phase > 2147483646LL) continue;
      const unsigned int target = phase_target((int)phase, per);
      EXPECT(target == (unsigned int)((unsigned long long)(phase + 1) * (unsigned long long)per));
      for (int missing = 0; missing <= per; missing += per > 8 ? per / 8 : 1)
        EXPECT(count_reached(target - (unsigned int)missing, target) == (missing == 0));
      // a peer that is a phase ahead has counted some items more
      for (int more = 1; more <= per; more += per > 8 ? per / 8 : 1)
        EXPECT(count_reached(target + (unsigned int)more, target));
    }
  std::printf(fails ? "FAILED\n" : "OK\n");
  return fails != 0;
}
