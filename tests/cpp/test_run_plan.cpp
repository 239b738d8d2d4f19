// Which kernels of a run wait for their peers (run_plan.h), on counts alone.
#include <cstdio>
#include <initializer_list>

#include "run_plan.h"

using namespace mprgp;
static int fails = 0;
#define EXPECT(c)                                     \
  do {                                                \
    if (!(c)) {                                       \
      std::printf("line %d: %s\n", __LINE__, #c);     \
      ++fails;                                        \
    }                                                 \
  } while (0)

// A device of 152 SMs that holds one CTA of a split form an SM (clusters of q
// in GPCs of 16 and a rest), four of a small whole one.
struct Cap {
  int power(int q, int, int, int smem) const { return q > 2 ? 136 : q == 1 && smem < 100 << 10 ? 304 : 152; }
  int engine(int q, int) const { return q > 2 ? 136 : 152; }
};

static PlanSettings settings(bool alone) {
  PlanSettings s;
  s.nsm = 152;
  s.alone = alone;
  s.power_launches = 1003;
  s.power_waits = s.engine_waits = true;
  s.persistent_per_sm = 4;
  for (bool &ok : s.power_cluster_ok) ok = true;
  return s;
}
static PlanInst inst(int items, bool fp32, bool in_power = true) {
  int cls = 0;
  while ((1 << cls) < items) ++cls;
  const bool large = cls >= kClusterClasses;
  return {large, large ? -1 : cls, items, 15, fp32, in_power};
}
static bool waits(const RunPlan &R) {
  bool w = R.power_sync || R.engine_sync || R.engine_small || R.power.grid || R.engine.grid;
  for (int u : R.class_units) w |= u != 0;
  return w;
}

int main() {
  const std::vector<std::vector<PlanInst>> runs = {
      {inst(2, false)},
      {inst(7, true)},
      {inst(70, false)},
      {inst(549, true)},
      {inst(1360, true)},
      {inst(1, true), inst(3, true), inst(9, true)},
      {inst(1, false), inst(16, false)},
      {inst(900, true), inst(2, true), inst(5, true)},
      {inst(900, true), inst(2, false)},
      std::vector<PlanInst>(400, inst(5, true)),
  };
  // beside another lane's run nothing waits, the small instances' clusters neither
  for (const auto &r : runs) EXPECT(!waits(plan_run(r, settings(false), Cap())));
  // alone, each in its form
  RunPlan R = plan_run(runs[0], settings(true), Cap());
  EXPECT(R.power_sync && R.small_in_plan && R.power.q == 8 && R.power.comps == 3);
  EXPECT(R.power.grid == 16 && R.engine_small && R.engine.q == 8 && R.engine.grid == 16);
  R = plan_run(runs[1], settings(true), Cap());
  EXPECT(R.power_sync && R.power.q == 1 && R.power.grid == 7 && !R.engine_sync);
  R = plan_run(runs[2], settings(true), Cap());
  EXPECT(R.power.q == 2 && R.small_in_plan && R.engine.grid > 0 && !R.engine_small);
  R = plan_run(runs[3], settings(true), Cap());
  EXPECT(R.power.q == 0 && R.power.grid == 549 && R.engine.q == 1);
  R = plan_run(runs[4], settings(true), Cap());
  EXPECT(!R.power_sync && R.engine_sync);
  R = plan_run(runs[7], settings(true), Cap());
  EXPECT(R.power_sync && !R.small_in_plan && R.power_count.n == 1);
  EXPECT(R.class_units[1] == 2 && R.class_units[3] == 8 && R.class_n[1] == 1 && R.class_fp32[1]);
  EXPECT(R.engine_sync && R.engine_count.n == 1);
  // items past the persistent loop: the launch loop, and no waiting clusters beside
  R = plan_run({inst(1360, true), inst(2, true), inst(5, true)}, settings(true), Cap());
  EXPECT(!R.power_sync && !R.class_units[1] && !R.class_units[3] && R.engine_sync);
  // a tuning with the launch loops keeps a small FP64 instance's power method in
  // the cluster solver; past it, the waiting engine takes it as before
  PlanSettings loops = settings(true);
  loops.power_waits = false;
  EXPECT(!waits(plan_run({inst(2, false)}, loops, Cap())));
  EXPECT(!waits(plan_run({inst(2, false), inst(3, false, false)}, loops, Cap())));
  R = plan_run({inst(2, false, false)}, loops, Cap());
  EXPECT(R.engine_small && !R.power_sync);
  // compact: whole items, no clusters, and no more CTAs than items
  PlanSettings compact = settings(true);
  compact.compact = true;
  for (const auto &r : runs) {
    R = plan_run(r, compact, Cap());
    int items = 0;
    for (const PlanInst &p : r) items += p.items;
    EXPECT(R.power.q <= 1 && R.engine.q <= 1 && R.power.comps == 1 && plan_ctas(R) <= items);
    EXPECT(!R.engine_small);
  }
  R = plan_run({inst(27, false)}, compact, Cap());
  EXPECT(R.power_sync && R.power.grid == 27 && R.engine_sync && R.engine.grid == 27);
  // an error concerns the instances of the launch that reports it
  {
    const std::vector<PlanInst> r = {inst(900, true), inst(2, true), inst(5, true),
                                     inst(2, true, false)};
    R = plan_run(r, settings(true), Cap());
    EXPECT(R.power_sync && !R.small_in_plan && R.class_units[1] && R.class_units[3]);
    EXPECT(error_word(R, r[0]) == 0);
    EXPECT(error_word(R, r[1]) == 2 && error_word(R, r[2]) == 4);
    EXPECT(error_word(R, r[3]) == -1);  // past its power method: the cluster solver alone
    const std::vector<PlanInst> t = {inst(198, true), inst(2, true, false), inst(2, false, false)};
    R = plan_run(t, settings(true), Cap());
    EXPECT(R.power_sync && error_word(R, t[0]) == 0);
    EXPECT(error_word(R, t[1]) == -1 && error_word(R, t[2]) == -1);
    const std::vector<PlanInst> u = {inst(20, true), inst(3, true), inst(3, true, false)};
    R = plan_run(u, settings(true), Cap());
    EXPECT(R.small_in_plan && error_word(R, u[1]) == 0 && error_word(R, u[2]) == -1);
    const std::vector<PlanInst> w = {inst(2, false), inst(3, false, false)};
    R = plan_run(w, settings(true), Cap());
    EXPECT(R.engine_small && error_word(R, w[0]) == 0 && error_word(R, w[1]) == 0);
    R = plan_run(w, settings(false), Cap());
    EXPECT(error_word(R, w[0]) == -1 && error_word(R, w[1]) == -1);
  }
  // the waiting engine ends a large instance's launch in time, a small one's never
  EXPECT(launch_limit_ns(false, 5.0) == 100000000000LL && launch_limit_ns(false, 1e-9) == 60000000000LL);
  EXPECT(launch_limit_ns(true, 5.0) == LLONG_MAX);
  // unit counts and grids agree
  for (const auto &r : runs) {
    for (bool c : {false, true}) {
      compact.compact = c;
      R = plan_run(r, compact, Cap());
      int units = (R.power_sync ? R.power_count.units : 0) + (R.engine_sync ? R.engine_count.units : 0);
      for (int u : R.class_units) units += u;
      EXPECT(units <= plan_units_at_most(r));
    }
    R = plan_run(r, settings(true), Cap());
    if (R.power_sync && R.power.q > 0) EXPECT(R.power.grid == R.power_count.units * R.power.q);
    if (R.engine_sync && R.engine.q > 1) EXPECT(R.engine.grid == R.engine_count.units * R.engine.q);
    if (R.engine_sync) EXPECT(R.engine.grid * kEngOwn >= R.engine_count.units);
  }
  std::printf(fails ? "FAILED\n" : "OK\n");
  return fails != 0;
}
