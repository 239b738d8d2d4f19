// One launch at a time of the kernels whose CTAs wait for each other.
//
// A cooperative kernel finishes only when all its CTAs are resident.  Two of
// them from different streams (another context's, another thread's) can each
// hold part of the SMs and wait for the rest for ever, or until their wait
// limit.  Every such launch of the process on a device is therefore ordered, on
// the device, behind the one issued before it; the host does not wait.  Kernels
// whose waits stay inside a thread-block cluster, and ordinary ones, run beside
// them.
//
// They also stay apart from a server's asynchronous lanes, of whatever context:
// a long serving run with such kernels on the lanes once ended in a memory
// fault whose cause was not found.  A synchronous run takes other forms while a
// lane has a run in flight, and a lane's run begins behind the last of them.
#pragma once
#include <algorithm>
#include <mutex>
#include <vector>

#include <cuda_runtime.h>

namespace mprgp {

struct CoopGate {
  std::mutex m;
  cudaEvent_t last = nullptr;      // the end of the last such launch
  int starting = 0;                // lane runs being issued, of every context,
  std::vector<cudaEvent_t> lanes;  // and the ends of those issued and not yet taken

  // The rest with `m` held.
  bool lanes_idle() const {
    if (starting > 0) return false;
    for (cudaEvent_t e : lanes)
      if (cudaEventQuery(e) == cudaErrorNotReady) return false;
    return true;
  }
  cudaError_t behind_last(cudaStream_t stream) {
    return last ? cudaStreamWaitEvent(stream, last, 0) : cudaSuccess;
  }
  template <typename F>
  cudaError_t launch(cudaStream_t stream, F issue) {
    cudaError_t e = cudaSuccess;
    if (!last) e = cudaEventCreateWithFlags(&last, cudaEventDisableTiming);
    if (e == cudaSuccess) e = behind_last(stream);
    if (e == cudaSuccess) e = issue();
    if (e == cudaSuccess) e = cudaEventRecord(last, stream);
    return e;
  }
  // Counts what `stream` holds so far as such a launch.
  cudaError_t mark(cudaStream_t stream) {
    return launch(stream, [] { return cudaSuccess; });
  }
};
CoopGate &coop_gate(int device);  // capi.cu

// A lane's run as the gate knows it: being issued while this object lives, then
// in flight up to its `end` event, until lane_taken.
class LaneStart {
 public:
  LaneStart(CoopGate &g, bool on) : g_(g), on_(on) { change(1, nullptr); }
  ~LaneStart() { change(-1, nullptr); }
  void issued(cudaEvent_t end) {
    change(-1, end);
    on_ = false;
  }

 private:
  void change(int by, cudaEvent_t end) {
    if (!on_) return;
    std::lock_guard<std::mutex> lock(g_.m);
    g_.starting += by;
    if (end) g_.lanes.push_back(end);
  }
  CoopGate &g_;
  bool on_;
};
inline void lane_taken(CoopGate &g, cudaEvent_t end) {
  std::lock_guard<std::mutex> lock(g.m);
  g.lanes.erase(std::remove(g.lanes.begin(), g.lanes.end(), end), g.lanes.end());
}

// Issues `issue()` (a cooperative kernel on `stream`) behind the gate of the
// current device.
template <typename F>
cudaError_t gated_launch(cudaStream_t stream, F issue) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  CoopGate &g = coop_gate(dev);
  std::lock_guard<std::mutex> lock(g.m);
  return g.launch(stream, issue);
}

}  // namespace mprgp
