// Launch shape of the kernels whose units (an item's rows each) take q CTAs.
//
// q > 1: a cluster a unit, whose CTAs read each other's shared memory; q == 1:
// a cooperative launch.  Never both attributes: Nsight Compute relaunches a
// cooperative kernel without its cluster dimension (measured with a kernel that
// records %cluster_nctarank: 4 in the plain run, 1 under ncu, with the cluster
// attribute alone 4 in both), and a CTA that then maps a peer's shared memory
// reads an address that does not exist.  The attribute is not needed either:
// the host launches only as many clusters as the device holds at once
// (cudaOccupancyMaxActiveClusters for this very configuration) and orders such
// launches (coop_gate.h), a cluster's CTAs start together, and kernels beside
// them end by themselves.
#pragma once
#include <cstddef>

#include <cuda_runtime.h>

namespace mprgp {

struct SplitLaunch {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
};

inline void split_launch(SplitLaunch &L, int q, int grid, int block, size_t smem,
                         cudaStream_t stream) {
  L.cfg = {};
  L.cfg.gridDim = dim3((unsigned int)grid);
  L.cfg.blockDim = dim3((unsigned int)block);
  L.cfg.dynamicSmemBytes = smem;
  L.cfg.stream = stream;
  if (q > 1) {
    L.at[0].id = cudaLaunchAttributeClusterDimension;
    L.at[0].val.clusterDim.x = (unsigned int)q;
    L.at[0].val.clusterDim.y = 1;
    L.at[0].val.clusterDim.z = 1;
  } else {
    L.at[0].id = cudaLaunchAttributeCooperative;
    L.at[0].val.cooperative = 1;
  }
  L.cfg.attrs = L.at;
  L.cfg.numAttrs = 1;
}

// Whether the shape a CTA sees (`cluster` CTAs a cluster, `grid` and `block`
// from the hardware's registers) is the one its arguments were made for.  The
// same answer in every CTA of a launch, so all of them leave before the first
// access to a peer or to the unit list when it is not.
__host__ __device__ inline bool split_shape_ok(int q, int units, int rows_threads, int cluster,
                                               int grid, int block) {
  return q >= 1 && cluster == q && units >= 0 && (long long)grid == (long long)units * q &&
         block == rows_threads;
}

// Whether an instance's phase counter has reached `target`.  Both count modulo
// 2^32 -- items times phases exceeds it in a long solve -- and never differ by
// more than the items of one phase, so the sign of the difference tells.
__host__ __device__ inline bool count_reached(unsigned int count, unsigned int target) {
  return (int)(count - target) >= 0;
}
// The counter at the end of phase `phase` (0, 1, ...) when each counts `per`.
__host__ __device__ inline unsigned int phase_target(int phase, int per) {
  return ((unsigned int)phase + 1u) * (unsigned int)per;
}

}  // namespace mprgp
