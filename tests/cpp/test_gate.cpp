// Which runs that wait for their peers may be in flight together (coop_gate.h).
#include <cstdio>

#include "coop_gate.h"

using namespace mprgp;
static int fails = 0;
#define EXPECT(c)                                     \
  do {                                                \
    if (!(c)) {                                       \
      std::printf("line %d: %s\n", __LINE__, #c);     \
      ++fails;                                        \
    }                                                 \
  } while (0)

int main() {
  const int nsm = 152;
  const std::vector<GateNeed> forms = {{7, false}, {16, true}, {27, false}, {70, false},
                                       {108, true}, {140, true}, {152, false}, {1 << 16, true}};
  for (const GateNeed &need : forms) {
    EXPECT(gate_entry({}, nsm, need, 0) == 0);  // alone, whatever it takes
    for (const GateNeed &a : forms)
      for (const GateNeed &b : forms) {
        const std::vector<GateNeed> in = {a, b};
        for (int wait : {0, 1, 2, 5}) {
          const int k = gate_entry(in, nsm, need, wait);
          EXPECT(k >= -1 && k <= wait && k <= 2);
          if (wait >= 2) EXPECT(k >= 0);  // in a row there is always room
          // whatever is in flight with it leaves an SM free for every CTA still to
          // come, and half of the SMs where clusters have to be placed
          auto fits = [&](int from) {
            int sms = need.sms;
            bool clusters = need.clusters;
            for (int i = from; i < 2; ++i) {
              sms += in[i].sms;
              clusters |= in[i].clusters;
            }
            return from == 2 || sms <= (clusters ? nsm / 2 : nsm);
          };
          if (k >= 0) EXPECT(fits(k));
          if (k > 0) EXPECT(!fits(k - 1));  // and it waits for no more than that
          if (k < 0)
            for (int i = 0; i <= std::min(wait, 2); ++i) EXPECT(!fits(i));
        }
      }
  }
  // four small FP64 runs of 16 SMs are in flight together, a fifth finds no room
  std::vector<GateNeed> in;
  for (int i = 0; i < 4; ++i) {
    EXPECT(gate_entry(in, nsm, {16, true}, 0) == 0);
    in.push_back({16, true});
  }
  EXPECT(gate_entry(in, nsm, {16, true}, 0) == -1);
  EXPECT(gate_entry(in, nsm, {16, true}, 1) == 1);
  std::printf(fails ? "FAILED\n" : "OK\n");
  return fails != 0;
}
