// Which runs of a process may hold kernels whose CTAs wait for each other.
//
// Such a kernel finishes only when all its CTAs are resident.  Two of them from
// different streams (another context's, another thread's) can each hold part of
// the SMs and wait for the rest for ever, or until their wait limit.  The gate
// of a device knows the runs in flight and lets another in while the SMs that
// all of them can need are there: at once, or behind the oldest of them on the
// device.  A kernel is counted with one SM a CTA: whatever the placement, the
// others leave an SM free for its next CTA.  A cluster takes that many free SMs
// of one GPC, so half of the SMs are the limit while a cluster form is among
// them: with the other half free, of at most ten GPCs one has seven.  A run of
// small instances that does not fit takes the cluster solver, which waits for
// nothing; a larger one whole items without clusters, behind as many of the
// others as it must.
// Solves a second of 1, 4 and 8 contexts, one launch after the other and so:
//   425 vertices, FP64      126 131 134    127 507 447
//   1,700, mixed            153 232 237    154 631 898
//   6,720, FP64             100 103 107     99 245 310
//   17,856, FP64             73  76  80     74 123 127
//   17,856, mixed           116 118 122    115 224 227
//   140,544, mixed           50  52         49  52
//
// Runs of launch loops -- a server's asynchronous lanes, and large synchronous runs
// while one of those is in flight -- and runs that wait stay apart: the former
// begin behind the latter, and while one is in flight no run waits.  (A long
// serving run with waiting kernels on the lanes once ended in a memory fault
// whose cause was not found.)  Kernels whose waits stay inside a thread-block
// cluster of their own, and ordinary ones, run beside all of them.
#pragma once
#include <algorithm>
#include <mutex>
#include <vector>

#include <cuda_runtime.h>

namespace mprgp {

struct GateNeed {  // of a run that waits
  int sms;
  bool clusters;
};
// How many of the oldest runs in flight a new one has to be behind (at most
// `wait`), or -1: it may not wait for its peers.
inline int gate_entry(const std::vector<GateNeed> &in_flight, int nsm, GateNeed need, int wait) {
  const int n = (int)in_flight.size();
  for (int k = 0; k <= std::min(wait, n); ++k) {
    int sms = need.sms;
    bool clusters = need.clusters;
    for (int i = k; i < n; ++i) {
      sms += in_flight[i].sms;
      clusters |= in_flight[i].clusters;
    }
    if (k == n || sms <= (clusters ? nsm / 2 : nsm)) return k;
  }
  return -1;
}

struct CoopGate {
  std::mutex m;
  std::vector<GateNeed> waiting;       // runs that wait, in the order of their entry,
  std::vector<cudaEvent_t> ends;       // and their ends
  int starting = 0;                // runs of launch loops being issued,
  std::vector<cudaEvent_t> loops;  // the ends of those issued by synchronous calls,
  std::vector<cudaEvent_t> lanes;  // and of lane runs not yet taken (the lanes' events)
  std::vector<cudaEvent_t> spare;

  // The rest with `m` held.
  static bool over(cudaEvent_t e) { return cudaEventQuery(e) != cudaErrorNotReady; }
  // Forgets what has ended; whether launch loops are in flight.
  bool loops_in_flight() {
    size_t w = 0;
    for (size_t i = 0; i < ends.size(); ++i) {
      if (over(ends[i])) {
        spare.push_back(ends[i]);
        continue;
      }
      waiting[w] = waiting[i];
      ends[w++] = ends[i];
    }
    waiting.resize(w);
    ends.resize(w);
    std::vector<cudaEvent_t> l;
    for (cudaEvent_t e : loops) (over(e) ? spare : l).push_back(e);
    loops.swap(l);
    bool in = starting > 0 || !loops.empty();
    for (cudaEvent_t e : lanes) in |= !over(e);
    return in;
  }
  // What comes on `stream` begins behind the oldest `count` runs that wait.
  cudaError_t behind(cudaStream_t stream, size_t count) {
    for (size_t i = 0; i < std::min(count, ends.size()); ++i) {
      const cudaError_t e = cudaStreamWaitEvent(stream, ends[i], 0);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  // An event behind what `stream` holds.
  cudaError_t end_of(cudaStream_t stream, cudaEvent_t *end) {
    cudaError_t e = cudaErrorUnknown;
    if (!spare.empty()) {
      *end = spare.back();
      spare.pop_back();
      e = cudaEventRecord(*end, stream);
    }
    if (e != cudaSuccess) {
      e = cudaEventCreateWithFlags(end, cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventRecord(*end, stream);
    }
    return e;
  }
  // What `stream` holds is a run that waits.
  cudaError_t entered(cudaStream_t stream, GateNeed need) {
    cudaEvent_t end;
    const cudaError_t e = end_of(stream, &end);
    if (e != cudaSuccess) return e;
    waiting.push_back(need);
    ends.push_back(end);
    return e;
  }
};
CoopGate &coop_gate(int device);  // capi.cu

// A run of launch loops as the gate knows it: being issued while this object
// lives, then in flight up to its end -- an event of the gate's, behind what
// `stream` holds, or a lane's own, until lane_taken.
class LoopRun {
 public:
  explicit LoopRun(CoopGate &g) : g_(g) {}
  ~LoopRun() {
    if (!on_) return;
    std::lock_guard<std::mutex> lock(g_.m);
    --g_.starting;
  }
  cudaError_t begin(cudaStream_t stream) {  // (with the gate's `m` held)
    const cudaError_t e = g_.behind(stream, g_.ends.size());
    if (e == cudaSuccess) {
      ++g_.starting;
      on_ = true;
    }
    return e;
  }
  cudaError_t issued(cudaStream_t stream) {
    if (!on_) return cudaSuccess;
    std::lock_guard<std::mutex> lock(g_.m);
    cudaEvent_t end;
    const cudaError_t e = g_.end_of(stream, &end);
    if (e != cudaSuccess) return e;
    g_.loops.push_back(end);
    --g_.starting;
    on_ = false;
    return e;
  }
  void issued_on_lane(cudaEvent_t end) {
    if (!on_) return;
    std::lock_guard<std::mutex> lock(g_.m);
    g_.lanes.push_back(end);
    --g_.starting;
    on_ = false;
  }

 private:
  CoopGate &g_;
  bool on_ = false;
};
inline void lane_taken(CoopGate &g, cudaEvent_t end) {
  std::lock_guard<std::mutex> lock(g.m);
  g.lanes.erase(std::remove(g.lanes.begin(), g.lanes.end(), end), g.lanes.end());
}

// Issues `issue()` -- a cooperative kernel of `ctas` CTAs on `stream` that has no
// other form -- behind as many runs of the current device as it must.
template <typename F>
cudaError_t gated_launch(cudaStream_t stream, int nsm, int ctas, F issue) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  CoopGate &g = coop_gate(dev);
  std::lock_guard<std::mutex> lock(g.m);
  g.loops_in_flight();
  const GateNeed need = {std::min(nsm, ctas), false};
  const int n = (int)g.waiting.size();
  e = g.behind(stream, (size_t)gate_entry(g.waiting, nsm, need, n));
  if (e == cudaSuccess) e = issue();
  if (e == cudaSuccess) e = g.entered(stream, need);
  return e;
}

}  // namespace mprgp
