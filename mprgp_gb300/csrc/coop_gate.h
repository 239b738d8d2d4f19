// One launch at a time of the kernels whose CTAs wait for each other.
//
// A cooperative kernel finishes only when all its CTAs are resident.  Two of
// them from different streams (another context's, another thread's, a server
// lane's) can each hold part of the SMs and wait for the rest for ever, or
// until their wait limit.  Every such launch of the process on a device is
// therefore ordered, on the device, behind the one issued before it; the host
// does not wait.  Kernels whose waits stay inside a thread-block cluster, and
// ordinary ones, run beside them.
#pragma once
#include <mutex>

#include <cuda_runtime.h>

namespace mprgp {

struct CoopGate {
  std::mutex m;
  cudaEvent_t last = nullptr;  // the end of the last such launch
};
CoopGate &coop_gate(int device);  // capi.cu

// Issues `launch()` (cooperative kernels on `stream`) behind the gate of the
// current device.
template <typename F>
cudaError_t gated_launch(cudaStream_t stream, F launch) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  CoopGate &g = coop_gate(dev);
  std::lock_guard<std::mutex> lock(g.m);
  if (!g.last) e = cudaEventCreateWithFlags(&g.last, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, g.last, 0);
  if (e == cudaSuccess) e = launch();
  if (e == cudaSuccess) e = cudaEventRecord(g.last, stream);
  return e;
}

}  // namespace mprgp
