// How one engine run is laid onto the GPU: which of its kernels wait for their
// peers, in which form, and which instances each takes.  Host arithmetic on
// counts alone, so that the CPU tests can run it; `Cap` answers how many CTAs
// of a form the device holds at once (power(q, fp32, comps, smem),
// engine(q, smem)).
#pragma once
#include <algorithm>
#include <climits>
#include <vector>

#include "engine.h"

namespace mprgp {

// One instance of a run.
struct PlanInst {
  bool large;     // on the engine (else in cluster class `cls` of the cluster solver)
  int cls;        // log2 of its cluster's size
  int items;      // of kThreads rows
  int max_len;    // blocks in a row, at most
  bool fp32;      // mixed form
  bool in_power;  // starts in a power phase
};

struct PlanSettings {
  int nsm = 0;
  // The run may hold kernels whose CTAs wait for each other: a synchronous run
  // (lane 0), and nothing of the library beside it that they must not meet.
  bool alone = false;
  bool compact = false;  // whole items only, no clusters: the fewest SMs a run can do with
  int quantum = 0, power_launches = 0, cluster_quantum = 0;
  bool power_waits = false;   // the tuning leaves the power method to the waiting forms
  bool engine_waits = false;  // ... and the other phases to the waiting engine
  bool persistent4 = false;   // the persistent power loop with up to kPowOwn items a CTA
  int persistent_per_sm = 0;  // its resident CTAs an SM
  bool power_cluster_ok[kClusterClasses] = {};  // cluster sizes its kernel can take
};

// q CTAs a unit with `comps` threads a row and smem bytes of slices each, or
// (power method, q == 0) the persistent loop; grid == 0: the form does not apply.
struct SyncPlan {
  int q = 0, comps = 1, smem = 0, grid = 0, groups = 1;
};

struct PlanCount {
  int units = 0, slots = 0, fp32 = 0, n = 0;
  void add(const PlanInst &p) {
    units += p.items;
    slots = std::max(slots, p.max_len);
    fp32 += p.fp32 ? 1 : 0;
    ++n;
  }
  bool one() const { return n > 0 && (fp32 == 0 || fp32 == n); }  // of one precision
};

struct RunPlan {
  SyncPlan power, engine;
  bool power_sync = false;    // the power method of the large instances (and, with
  bool small_in_plan = false; // small_in_plan, of the small ones) in one waiting launch
  PlanCount power_count;      // ... its instances
  int class_n[kClusterClasses] = {};      // instances whose power method runs in clusters
  int class_units[kClusterClasses] = {};  // ... their units, absent items included
  bool class_fp32[kClusterClasses] = {};
  bool engine_sync = false;   // the waiting engine, for the large instances or (engine_small)
  bool engine_small = false;  // for a run of small ones
  PlanCount engine_count;
};

template <typename Cap>
SyncPlan sync_plan(const Cap &cap, int nsm, int units, int max_slots, int fp32, bool compact) {
  SyncPlan P;
  const int slice = max_slots * kSlice * (9 * (fp32 ? 4 : 8) + 4);
  auto bytes = [&](int q) {  // a CTA's slices, in few distinct sizes
    return ((long long)slice * (kThreads / kSlice / q) + 4095) / 4096 * 4096;
  };
  auto fits = [&](int q, int comps) {
    if (bytes(q) > kSyncStageBytes || units * q > cap.power(q, fp32, comps, (int)bytes(q)))
      return false;
    P.q = q;
    P.comps = comps;
    P.smem = (int)bytes(q);
    P.grid = units * q;
    return true;
  };
  // FP64 rows by three threads, one a component, while each scheduler of an SM
  // gets one or two such warps: a row's 135 FP64 FMAs (15 blocks) take 6 us as
  // one warp's chain, a component's 45 take 2.
  // 425 vertices: 10.7 -> 7.7 us a phase, 6,720: 12.3 -> 9.3.  (Three quarters
  // of the SMs: clusters do not pack them further, and two CTAs on an SM cost
  // what the split gains: 9,464 vertices 13.2 us, 12.6 with whole rows.)
  if (!fp32 && !compact)
    for (int q = 8; q >= 4; q /= 2)
      if (4 * units * q <= 3 * nsm && fits(q, 3)) return P;
  // Else the fewest CTAs an item whose slices fit shared memory, or twice as
  // many (smaller CTAs can pack an SM better).  1,760 vertices mixed: 4.85 us
  // a phase with q = 1, 5.5 with 2, 4 or 8; 17,856 in FP64: 11.5 with q = 2,
  // 14.2 with 4, 18.3 with 8.
  int tried = 0;
  for (int q = 1; q <= (compact ? 1 : kThreads / kSlice) && tried < 2; q *= 2) {
    if (bytes(q) > kSyncStageBytes) continue;
    ++tried;
    if (fits(q, 1)) break;
  }
  return P;
}

inline SyncPlan persistent_plan(const PlanSettings &s, int units) {
  SyncPlan P;
  const int cap = s.nsm * s.persistent_per_sm;
  // Up to two items a CTA, unless the tuning asks for the persistent loop:
  // a phase takes 15.8 us against 23.2 as graph launches at 549 items, 29.9
  // against 31.1 at 833 (two a CTA), but 52.4 against 51.0 at 1,360 (three a
  // CTA, streaming from DRAM, which more CTAs hide better).
  if (cap > 0 && units <= cap * (s.persistent4 ? kPowOwn : 2)) {
    const int per = (units + cap - 1) / cap;  // equally many items a CTA
    P.grid = (units + per - 1) / per;
  }
  return P;
}

// The waiting engine's layout; grid == 0 when it does not apply.
template <typename Cap>
SyncPlan engine_plan(const Cap &cap, int nsm, int units, int max_slots, bool split, bool beside) {
  SyncPlan P;
  // FP64 items: eight or four CTAs of three threads a row, with their matrix
  // slices in shared memory, while three quarters of the SMs hold them (the
  // rule of sync_plan); else two CTAs while each has an SM of its own: an
  // item's eight row warps take 135 FP64 FMAs each, two warps a scheduler in
  // one CTA (17,856 vertices 16.6 -> 16.1 ms with two).
  if (split)
    for (int q = 8; q >= 4; q /= 2) {
      const long long bytes = (long long)max_slots * kSlice * (9 * 8 + 4) * (kThreads / kSlice / q);
      const long long smem = (bytes + 4095) / 4096 * 4096;
      if (4 * units * q > 3 * nsm || smem > kEngStageBytes || units * q > cap.engine(q, (int)smem))
        continue;
      P.q = q;
      P.smem = (int)smem;
      P.grid = q * units;
      return P;
    }
  if (split && 2 * units <= std::min(nsm, cap.engine(2, 0))) {
    P.q = 2;
    P.grid = 2 * units;
    return P;
  }
  // One CTA an SM with equally many items, in as few rounds as four groups
  // give; beside cluster solves, smaller CTAs of one group, which find room as
  // those finish (a batch of 48 takes 25.6 ms so, 28.8 with one CTA an SM).
  const int ctas = std::min(nsm, cap.engine(1, 0)) * (beside ? 4 : 1);
  const int per = ctas > 0 ? (units + ctas - 1) / ctas : kEngOwn + 1;
  if (per <= kEngOwn) {
    const int rounds = beside ? per : (per + 3) / 4;
    P.q = 1;
    P.groups = (per + rounds - 1) / rounds;
    P.grid = (units + per - 1) / per;
  }
  return P;
}

// The power method in the forms whose CTAs wait for each other (unless the
// tuning asks for the launch loops): a synchronous run's instances, small ones
// too, by the power sync loop when all their CTAs are resident at once; else
// its large ones by the persistent loop and its small ones by the same kernel
// with one cluster an instance.  Every one of them, the clusters too, only in a
// run that is alone: kernels that wait for their peers stay out of runs that
// share the SMs with a server's lanes, which keep the launch loops and the
// cluster solver.
template <typename Cap>
RunPlan plan_run(const std::vector<PlanInst> &insts, const PlanSettings &s, const Cap &cap) {
  RunPlan R;
  const int n = (int)insts.size();
  int n_large = 0, in_power = 0;  // large instances; instances in a power phase
  PlanCount all, large, cl[kClusterClasses];
  bool cl_fits[kClusterClasses] = {true, true, true, true, true};
  const bool waiting = s.alone && s.power_launches > 0 && s.power_waits;
  for (const PlanInst &p : insts) {
    n_large += p.large ? 1 : 0;
    in_power += p.in_power ? 1 : 0;
    if (!waiting || !p.in_power) continue;
    if (p.large) {
      all.add(p);
      large.add(p);
    } else if (s.cluster_quantum == 0) {
      all.add(p);
      cl[p.cls].add(p);
      cl_fits[p.cls] &= p.items <= (1 << p.cls);
    }
  }
  if (all.one()) {
    R.power = sync_plan(cap, s.nsm, all.units, all.slots, all.fp32 ? 1 : 0, s.compact);
    R.small_in_plan = R.power.grid > 0;
  }
  if (large.one() && R.power.grid == 0) R.power = persistent_plan(s, large.units);
  R.power_sync = R.power.grid > 0;
  R.power_count = R.small_in_plan ? all : large;
  for (int q = 0; q < kClusterClasses; ++q) {
    if (R.small_in_plan || !cl[q].one() || !cl_fits[q] || !s.power_cluster_ok[q]) continue;
    if (large.n > 0 && !R.power_sync) continue;  // not beside the large ones' launch loop
    R.class_n[q] = cl[q].n;
    R.class_units[q] = cl[q].n << q;
    R.class_fp32[q] = cl[q].fp32 > 0;
  }
  // The instances' other phases: the waiting engine for the large ones of a
  // synchronous run, and for small ones too when they are FP64 and few enough
  // for split units (425 vertices: a solve of 13.7 -> 9.0 ms, most of it by the
  // power loop's form).  Not when their power method has yet to run and the
  // tuning keeps it in the cluster solver.
  const bool eng_on = s.alone && s.quantum >= 0 && s.engine_waits;
  if (!eng_on) return R;
  PlanCount eng;
  for (const PlanInst &p : insts)
    if (n_large == 0 || p.large) eng.add(p);
  if (n_large == 0 && !s.compact && s.quantum == 0 && s.cluster_quantum == 0 && eng.fp32 == 0 &&
      (in_power == 0 || R.small_in_plan)) {
    R.engine = engine_plan(cap, s.nsm, eng.units, eng.slots, true, false);
    if (R.engine.q < 2) R.engine = SyncPlan();
    R.engine_small = R.engine.grid > 0;
  } else if (n_large > 0) {
    R.engine = engine_plan(cap, s.nsm, eng.units, eng.slots, eng.fp32 == 0 && !s.compact,
                           n > n_large);
  }
  R.engine_sync = R.engine.grid > 0;
  R.engine_count = eng;
  return R;
}

// CTAs that the run's waiting launches hold at once, at most (they follow each
// other; the clusters' power loops wait for nothing outside their cluster).
inline int plan_ctas(const RunPlan &R) { return std::max(R.power.grid, R.engine.grid); }

// Entries of the unit list that any plan of these instances can need: every item
// once for the power method and once for the waiting engine, or a cluster's CTAs.
inline int plan_units_at_most(const std::vector<PlanInst> &insts) {
  int n = 0;
  for (const PlanInst &p : insts) n += p.items + (p.large ? p.items : std::max(p.items, 1 << p.cls));
  return n;
}

// A run's error words: 0 for its waiting launches over the large instances (and
// whatever joins them), 1 + q for the power loops of cluster class q.  The word
// of the launch that an instance took part in, or -1: no launch that can give up
// concerns it, and its result stands whatever becomes of the others.
constexpr int kErrWords = 1 + kClusterClasses;
inline int error_word(const RunPlan &R, const PlanInst &p) {
  if (p.large || R.engine_small) return 0;
  if (!p.in_power) return -1;
  if (R.power_sync && R.small_in_plan) return 0;
  return R.class_units[p.cls] > 0 ? 1 + p.cls : -1;
}

// Bound on the time of a whole engine launch: 20 waits, a minute at least.
// Small instances have none: in the cluster solver, whose phases they take here,
// only their iterations bound them.
inline long long launch_limit_ns(bool small, double wait_s) {
  return small ? LLONG_MAX : (long long)(std::max(60.0, 20.0 * wait_s) * 1e9);
}

}  // namespace mprgp
