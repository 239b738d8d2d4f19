// ICA (Iterative Constraint Anticipation) contact solver on the GPU: the
// reference's comparison baseline for MPRGP, src/MPRGPSolver/ICASolver.h
// (ICASolver :287-463 with ProjectedGaussSeidel :20-150), for
//   A x = r + J^T lambda,  0 <= lambda _|_ J x - p >= 0,
// A in 3x3-block rows (BSR) split as La + Da + Ua by blocks, J given as
// per-vertex planes (n, q): the row n at the vertex's columns with p = -q.
//
// Every iterate is the reference's, computed in a fixed order:
//  * c = p + J Da^-1 (LaUa x - r) and rhs = J^T lambda - Ua x + r are
//    per-vertex passes (thread per vertex);
//  * B = J Da^-1 J^T couples constraints of the same vertex only, so the
//    projected Gauss-Seidel sweep over all rows (GaussSeidel::solve :67-105)
//    is the set of per-vertex sweeps; each sweep ends in a grid reduction of
//    ||lambda - lambda_prev|| for the shared stopping test;
//  * the 3x3-block Gauss-Seidel sweep (:377-388) reads the new x of lower
//    block columns and the old x of upper ones: block rows are grouped in
//    dependency levels (a row's level is one more than the highest level of
//    its lower neighbours), each level's rows are independent and run in
//    parallel, and a grid barrier separates levels -- the same values as the
//    sequential sweep;
//  * ||A x - r - J^T lambda|| ends each iteration.
// One persistent cooperative kernel runs all iterations; grid barriers are
// bounded in time (a wait that runs out sets an error and the kernel
// returns).  Sums run in ascending column / constraint order and this file
// is compiled without fused multiply-adds (-fmad=false), so the results are
// bitwise those of the CPU restatement that performs the same operations.
#include <algorithm>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/mprgp_gpu.h"
#include "coop_gate.h"

namespace mprgp {
void set_last_error(const char *what);
int context_lanes_busy(const mprgp_context *c);
}  // namespace mprgp

namespace {

constexpr int kIcaThreads = 256;

struct IcaCtl {
  unsigned int count, gen;
  int err, pad;
};

struct IcaArgs {
  int nv, m, nlevels, max_it, gs_max_it;
  double tol, gs_tol;
  const int *row_ptr, *cols;
  const double *vals;  // 9 per block, row-major
  const double *r;
  const int *plane_ptr;
  const double *planes;  // (n, q) per constraint
  const int *order, *lvl_ptr;  // block rows by level; level starts
  double *x, *lam, *c, *rhs, *inv, *B, *part;
  IcaCtl *ctl;
  double *out;  // iterations, converged, residual, sweeps
  long long wait_ns;
};

__device__ __forceinline__ long long gtimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int atom_add_acq_rel(unsigned int *p, unsigned int v) {
  unsigned int old;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void st_release(unsigned int *p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// Grid barrier with a time bound; false when it (or another CTA's) ran out.
__device__ bool ica_barrier(IcaCtl *ctl, long long wait_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    volatile int *verr = &ctl->err;
    const unsigned int g = ld_acquire(&ctl->gen);
    const unsigned int arrived = atom_add_acq_rel(&ctl->count, 1u);
    int ok = 1;
    if (arrived == gridDim.x - 1) {
      ctl->count = 0u;
      st_release(&ctl->gen, g + 1);
    } else {
      const long long t0 = gtimer();
      while (ld_acquire(&ctl->gen) == g) {
        if (*verr) {
          ok = 0;
          break;
        }
        if (gtimer() - t0 > wait_ns) {
          atomicCAS(&ctl->err, 0, 1);
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
    }
    s_ok = ok && *verr == 0;
  }
  __syncthreads();
  return s_ok;
}

// Sum of one double per thread over the grid, the same on every CTA: block
// sums in a fixed tree, written to part[par][block], then one warp adds the
// block sums in a fixed order.  `ok` turns false if the barrier gave up.
__device__ double grid_sum(double v, double *part, int par, IcaCtl *ctl, long long wait_ns,
                           bool &ok) {
  __shared__ double sh[kIcaThreads / 32];
  __shared__ double s_tot;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kIcaThreads / 32; ++w) t += sh[w];
    part[par * gridDim.x + blockIdx.x] = t;
  }
  ok = ica_barrier(ctl, wait_ns);
  if (!ok) return 0.0;
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) t += part[par * gridDim.x + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) s_tot = t;
  }
  __syncthreads();
  return s_tot;
}

__device__ __forceinline__ void mul3(const double *M, const double *v, double *y) {
#pragma unroll
  for (int k = 0; k < 3; ++k) y[k] = (M[3 * k] * v[0] + M[3 * k + 1] * v[1]) + M[3 * k + 2] * v[2];
}

// 3x3 inverse: adjugate over the determinant expanded along row 0.
__device__ void inverse3(const double *m, double *inv) {
  const double a = m[0], b = m[1], c = m[2], d = m[3], e = m[4], f = m[5], g = m[6], h = m[7],
               i = m[8];
  const double c00 = e * i - f * h, c01 = f * g - d * i, c02 = d * h - e * g;
  const double det = (a * c00 + b * c01) + c * c02;
  const double s = 1.0 / det;
  inv[0] = c00 * s;
  inv[1] = (c * h - b * i) * s;
  inv[2] = (b * f - c * e) * s;
  inv[3] = c01 * s;
  inv[4] = (a * i - c * g) * s;
  inv[5] = (c * d - a * f) * s;
  inv[6] = c02 * s;
  inv[7] = (b * g - a * h) * s;
  inv[8] = (a * e - b * d) * s;
}

// (J^T lambda) at vertex v.
__device__ __forceinline__ void jt_lambda(const IcaArgs &a, int v, double jl[3]) {
  jl[0] = jl[1] = jl[2] = 0.0;
  for (int q = a.plane_ptr[v]; q < a.plane_ptr[v + 1]; ++q) {
    const double *pl = a.planes + 4 * (size_t)q;
    const double l = a.lam[q];
#pragma unroll
    for (int k = 0; k < 3; ++k) jl[k] = jl[k] + l * pl[k];
  }
}

// Row sums of block row v over the blocks whose column passes `take`.
template <typename Take>
__device__ __forceinline__ void row_sum(const IcaArgs &a, int v, const double *x, Take take,
                                        double acc[3]) {
  acc[0] = acc[1] = acc[2] = 0.0;
  for (int k = a.row_ptr[v]; k < a.row_ptr[v + 1]; ++k) {
    const int u = a.cols[k];
    if (!take(u)) continue;
    const double *blk = a.vals + 9 * (size_t)k;
    const double *xc = x + 3 * (size_t)u;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int b = 0; b < 3; ++b) acc[r] = acc[r] + blk[3 * r + b] * xc[b];
  }
}

__global__ void __launch_bounds__(kIcaThreads) ica_kernel(IcaArgs a) {
  __shared__ double s_blk[kIcaThreads / 32][32][12];  // per warp: 32 blocks + their x
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int gthreads = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int gwarp = gtid >> 5, gwarps = gthreads >> 5;
  // reset (:296-350): Da^-1 per block row; B = J Da^-1 J^T per vertex.
  for (int v = gtid; v < a.nv; v += gthreads) {
    double *inv = a.inv + 9 * (size_t)v;
    for (int k = a.row_ptr[v]; k < a.row_ptr[v + 1]; ++k)
      if (a.cols[k] == v) inverse3(a.vals + 9 * (size_t)k, inv);
    const int q0 = a.plane_ptr[v], nq = a.plane_ptr[v + 1] - q0;
    for (int j = 0; j < nq; ++j) {
      double t[3];
      mul3(inv, a.planes + 4 * (size_t)(q0 + j), t);
      for (int i = 0; i < nq; ++i) {
        const double *ni = a.planes + 4 * (size_t)(q0 + i);
        a.B[9 * (size_t)v + 3 * i + j] = (ni[0] * t[0] + ni[1] * t[1]) + ni[2] * t[2];
      }
    }
    for (int q = q0; q < q0 + nq; ++q) a.lam[q] = 0.0;
  }
  int par = 0, it = 0, conv = 0;
  long long sweeps = 0;
  double res = 0.0;
  bool ok = true;
  for (; it < a.max_it; ++it) {
    // c = p + J Da^-1 (LaUa x - r)                                    (:371)
    for (int v = gtid; v < a.nv; v += gthreads) {
      double u[3], w[3];
      row_sum(a, v, a.x, [v](int col) { return col != v; }, u);
#pragma unroll
      for (int k = 0; k < 3; ++k) u[k] = u[k] - a.r[3 * v + k];
      mul3(a.inv + 9 * (size_t)v, u, w);
      for (int q = a.plane_ptr[v]; q < a.plane_ptr[v + 1]; ++q) {
        const double *pl = a.planes + 4 * (size_t)q;
        a.c[q] = -pl[3] + ((pl[0] * w[0] + pl[1] * w[1]) + pl[2] * w[2]);
      }
    }
    // projected Gauss-Seidel on B, warm-started from the last lambda (:372)
    for (int s = 0; s < a.gs_max_it; ++s) {
      double ss = 0.0;
      for (int v = gtid; v < a.nv; v += gthreads) {
        const int q0 = a.plane_ptr[v], nq = a.plane_ptr[v + 1] - q0;
        const double *B = a.B + 9 * (size_t)v;
        double old[3] = {0.0, 0.0, 0.0}, l[3] = {0.0, 0.0, 0.0};
        for (int i = 0; i < nq; ++i) old[i] = a.lam[q0 + i];
        for (int i = 0; i < nq; ++i) {
          double ub = 0.0;
          for (int j = i + 1; j < nq; ++j) ub = ub + B[3 * i + j] * old[j];
          double rr = a.c[q0 + i] - ub;
          for (int j = 0; j < i; ++j) rr -= l[j] * B[3 * i + j];
          const double li = rr * (1.0 / B[3 * i + i]);
          l[i] = li > 0 ? li : 0;
        }
        for (int i = 0; i < nq; ++i) {
          a.lam[q0 + i] = l[i];
          const double d = l[i] - old[i];
          ss = ss + d * d;
        }
      }
      const double tot = grid_sum(ss, a.part, par, a.ctl, a.wait_ns, ok);
      par ^= 1;
      ++sweeps;
      if (!ok) return;
      if (sqrt(tot) <= a.gs_tol) break;
    }
    // rhs = J^T lambda - Ua x + r (old x)                              (:374)
    for (int v = gtid; v < a.nv; v += gthreads) {
      double jl[3], ua[3];
      jt_lambda(a, v, jl);
      row_sum(a, v, a.x, [v](int col) { return col > v; }, ua);
#pragma unroll
      for (int k = 0; k < 3; ++k) a.rhs[3 * v + k] = (jl[k] - ua[k]) + a.r[3 * v + k];
    }
    if (!ica_barrier(a.ctl, a.wait_ns)) return;
    // 3x3-block Gauss-Seidel sweep (:377-388), level by level, one warp per
    // block row: the lanes fetch the row's lower blocks and their x together
    // (one round of loads); lane k (k < 3) then subtracts them from scalar
    // row k in column order, and lane k forms component k of the new x.
    for (int lv = 0; lv < a.nlevels; ++lv) {
      for (int t = a.lvl_ptr[lv] + gwarp; t < a.lvl_ptr[lv + 1]; t += gwarps) {
        const int v = a.order[t];
        const int k0 = a.row_ptr[v], k1 = a.row_ptr[v + 1];
        double acc = lane < 3 ? a.rhs[3 * v + lane] : 0.0;
        for (int base = k0; base < k1; base += 32) {
          const int j = base + lane;
          const int u = j < k1 ? a.cols[j] : v;
          const bool low = u < v;
          if (low) {
            const double *blk = a.vals + 9 * (size_t)j;
            const double *xc = a.x + 3 * (size_t)u;
#pragma unroll
            for (int e = 0; e < 9; ++e) s_blk[wid][lane][e] = blk[e];
#pragma unroll
            for (int b = 0; b < 3; ++b) s_blk[wid][lane][9 + b] = xc[b];
          }
          const unsigned int lower = __ballot_sync(0xffffffffu, low);
          __syncwarp();
          if (lane < 3) {
            const int cnt = min(32, k1 - base);
            for (int q = 0; q < cnt; ++q) {
              if (!((lower >> q) & 1u)) continue;
              const double *s = s_blk[wid][q];
#pragma unroll
              for (int b = 0; b < 3; ++b) acc -= s[3 * lane + b] * s[9 + b];
            }
          }
          __syncwarp();
        }
        const double r0 = __shfl_sync(0xffffffffu, acc, 0), r1 = __shfl_sync(0xffffffffu, acc, 1),
                     r2 = __shfl_sync(0xffffffffu, acc, 2);
        if (lane < 3) {
          const double *M = a.inv + 9 * (size_t)v + 3 * lane;
          a.x[3 * (size_t)v + lane] = (M[0] * r0 + M[1] * r1) + M[2] * r2;
        }
      }
      if (!ica_barrier(a.ctl, a.wait_ns)) return;
    }
    // residual = ||A x - r - J^T lambda||                              (:390)
    double ss = 0.0;
    for (int v = gtid; v < a.nv; v += gthreads) {
      double jl[3], ax[3];
      jt_lambda(a, v, jl);
      row_sum(a, v, a.x, [](int) { return true; }, ax);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double t = (ax[k] - a.r[3 * v + k]) - jl[k];
        ss = ss + t * t;
      }
    }
    const double tot = grid_sum(ss, a.part, par, a.ctl, a.wait_ns, ok);
    par ^= 1;
    if (!ok) return;
    res = sqrt(tot);
    if (res <= a.tol) {
      conv = 1;
      break;
    }
  }
  if (gtid == 0) {
    a.out[0] = (double)it;
    a.out[1] = (double)conv;
    a.out[2] = res;
    a.out[3] = (double)sweeps;
  }
}

// ------------------------------------------------------- one cluster -----
// The same solver for bodies of up to 5,120 vertices, as one thread-block
// cluster with a copy of x in every CTA's shared memory.
//
// A small body's iteration is a chain of latencies: one grid barrier and one
// row a warp (dependent loads, then up to 47 dependent FP64 operations) for
// every dependency level, and a grid reduction for every sweep.  1,377
// vertices, 33 levels: 260 us an iteration on the grid, about 7 us a level, and
// 57 ms for the solve of 220; this form takes 85 us and 18.7 ms.  Here a level ends in a hardware cluster barrier; a lane carries one scalar
// row (ten block rows a warp), new x goes straight into every CTA's copy; and
// two halves of the warps alternate: while one half finishes level L, the
// other loads level L + 1 and takes the leading terms whose x is two levels
// old (on a grid mesh three of seven).  The residual pass forms the row sums
// that the next iteration's c and rhs need from the same products.  All sums
// run in the order of the grid form, so x, lambda and the counts are its bits
// (the residual's and the sweep test's sums differ in grouping alone).
constexpr int kCThreads = 512, kCWarps = kCThreads / 32, kCRows = 10;  // block rows a warp
constexpr int kCCtas = 16, kCLow = 8;                   // CTAs; blocks left of a diagonal
constexpr int kCOwn = kCWarps * kCRows;                 // vertices of a CTA in one round
constexpr int kCMaxRounds = 2;                          // so up to 5,120 vertices
constexpr int kCState = 18;                             // doubles a vertex: lambda, c, B, 1 / B_ii

struct IcaRow {  // a block row in level order: its blocks left of the diagonal,
  int v, k0, nlow, pre;  // and how many leading ones lie two or more levels back
};
struct IcaClusterArgs {
  IcaArgs a;
  const IcaRow *rows;
};

__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned int peer_addr(const void *p, unsigned int rank) {
  const unsigned int l = (unsigned int)__cvta_generic_to_shared(p);
  unsigned int r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(l), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_peer(unsigned int addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" : : "r"(addr), "d"(v) : "memory");
}

// Sum of one double a thread over the cluster, the same bits in every CTA.
__device__ double cluster_sum(double v, double (*red)[kCCtas * kCWarps], double *tot, int par,
                              int rank, int ncta) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane < ncta) st_peer(peer_addr(&red[par][rank * kCWarps + warp], (unsigned int)lane), v);
  cluster_barrier();
  if (warp == 0) {
    double t = 0.0;
    for (int i = lane; i < ncta * kCWarps; i += 32) t += red[par][i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) *tot = t;
  }
  __syncthreads();
  return *tot;
}

// One scalar row of the block Gauss-Seidel sweep: component `comp` of a block
// row, whose lower blocks are m[u] at the columns col[u].
struct LevelRow {
  double m[kCLow][3], acc;
  int col[kCLow], v, nlow, pre;
  __device__ __forceinline__ void load(const IcaClusterArgs &C, int t, int comp) {
    const int4 r = __ldg(reinterpret_cast<const int4 *>(C.rows) + t);
    v = r.x;
    nlow = r.z;
    pre = r.w;
    acc = C.a.rhs[3 * v + comp];
#pragma unroll
    for (int u = 0; u < kCLow; ++u) {
      if (u >= nlow) continue;
      col[u] = __ldg(C.a.cols + r.y + u);
      const double *b = C.a.vals + 9 * (size_t)(r.y + u) + 3 * comp;
      m[u][0] = __ldg(b);
      m[u][1] = __ldg(b + 1);
      m[u][2] = __ldg(b + 2);
    }
  }
  __device__ __forceinline__ void take(int from, int to, const double *x) {
#pragma unroll
    for (int u = 0; u < kCLow; ++u) {
      if (u < from || u >= to) continue;
      const double *xc = x + 3 * col[u];
      acc -= m[u][0] * xc[0];
      acc -= m[u][1] * xc[1];
      acc -= m[u][2] * xc[2];
    }
  }
};

__global__ void __launch_bounds__(kCThreads) ica_cluster_kernel(IcaClusterArgs C) {
  extern __shared__ __align__(16) double s_dyn[];
  __shared__ double s_red[2][kCCtas * kCWarps];
  __shared__ double s_tot;
  const IcaArgs &a = C.a;
  const int rank = (int)blockIdx.x, ncta = (int)gridDim.x;  // one cluster
  unsigned int csize;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
  if ((int)csize != ncta) {  // not the launch's shape: no peer to write to
    if (threadIdx.x == 0) atomicCAS(&a.ctl->err, 0, 2);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / 3, comp = lane - 3 * sub, lead = 3 * sub;  // block row of the warp
  const bool on = lane < 3 * kCRows;
  double *x = s_dyn;                    // 3 nv
  double *state = s_dyn + 3 * a.nv;     // kCState per owned vertex
  const int rounds = (a.nv + kCOwn * ncta - 1) / (kCOwn * ncta);
  auto vertex = [&](int r) { return ((r * kCWarps + warp) * ncta + rank) * kCRows + sub; };
  auto own = [&](int r) { return state + kCState * ((r * kCWarps + warp) * kCRows + sub); };
  for (int i = threadIdx.x; i < 3 * a.nv; i += kCThreads) x[i] = a.x[i];
  // reset (:296-350): Da^-1 per block row; B = J Da^-1 J^T per vertex.
  for (int r = 0; r < rounds; ++r) {
    const int v = vertex(r);
    if (!on || comp != 0 || v >= a.nv) continue;
    double *inv = a.inv + 9 * (size_t)v, *S = own(r);
    for (int k = a.row_ptr[v]; k < a.row_ptr[v + 1]; ++k)
      if (a.cols[k] == v) inverse3(a.vals + 9 * (size_t)k, inv);
    const int q0 = a.plane_ptr[v], nq = a.plane_ptr[v + 1] - q0;
    for (int j = 0; j < nq; ++j) {
      double t[3];
      mul3(inv, a.planes + 4 * (size_t)(q0 + j), t);
      for (int i = 0; i < nq; ++i) {
        const double *ni = a.planes + 4 * (size_t)(q0 + i);
        S[6 + 3 * i + j] = (ni[0] * t[0] + ni[1] * t[1]) + ni[2] * t[2];
      }
    }
    for (int j = 0; j < nq; ++j) {
      S[j] = 0.0;
      S[15 + j] = 1.0 / S[6 + 4 * j];
    }
  }
  __syncthreads();
  cluster_barrier();
  int par = 0, it = 0, conv = 0;
  long long sweeps = 0;
  double res = 0.0;
  double lu[kCMaxRounds], ua[kCMaxRounds];
  // A x, LaUa x and Ua x of the thread's scalar rows, and its share of
  // ||A x - r - J^T lambda||^2                                        (:390)
  auto pass = [&]() {
    double ss = 0.0;
#pragma unroll
    for (int r = 0; r < kCMaxRounds; ++r) {
      const int v = vertex(r);
      if (r >= rounds || !on || v >= a.nv) continue;
      double ax = 0.0, l = 0.0, u = 0.0;
      const int k1 = __ldg(a.row_ptr + v + 1);
      for (int k = __ldg(a.row_ptr + v); k < k1; ++k) {
        const int cu = __ldg(a.cols + k);
        const double *b = a.vals + 9 * (size_t)k + 3 * comp, *xc = x + 3 * cu;
        const double p0 = __ldg(b) * xc[0], p1 = __ldg(b + 1) * xc[1], p2 = __ldg(b + 2) * xc[2];
        ax = ax + p0;
        ax = ax + p1;
        ax = ax + p2;
        if (cu != v) {
          l = l + p0;
          l = l + p1;
          l = l + p2;
        }
        if (cu > v) {
          u = u + p0;
          u = u + p1;
          u = u + p2;
        }
      }
      lu[r] = l;
      ua[r] = u;
      const double *S = own(r);
      double jl = 0.0;
      const int q0 = __ldg(a.plane_ptr + v), nq = __ldg(a.plane_ptr + v + 1) - q0;
      for (int j = 0; j < nq; ++j) jl = jl + S[j] * __ldg(a.planes + 4 * (size_t)(q0 + j) + comp);
      const double t = (ax - a.r[3 * v + comp]) - jl;
      ss = ss + t * t;
    }
    return ss;
  };
  pass();
  for (; it < a.max_it; ++it) {
    // c = p + J Da^-1 (LaUa x - r)                                    (:371)
#pragma unroll
    for (int r = 0; r < kCMaxRounds; ++r) {
      if (r >= rounds) continue;
      const int v = vertex(r);
      const bool mine = on && v < a.nv;
      const double u = mine ? lu[r] - a.r[3 * v + comp] : 0.0;
      const double u0 = __shfl_sync(0xffffffffu, u, lead), u1 = __shfl_sync(0xffffffffu, u, lead + 1),
                   u2 = __shfl_sync(0xffffffffu, u, lead + 2);
      if (!mine || comp != 0) continue;
      const double uu[3] = {u0, u1, u2};
      double w[3];
      mul3(a.inv + 9 * (size_t)v, uu, w);
      const int q0 = __ldg(a.plane_ptr + v), nq = __ldg(a.plane_ptr + v + 1) - q0;
      for (int j = 0; j < nq; ++j) {
        const double *pl = a.planes + 4 * (size_t)(q0 + j);
        own(r)[3 + j] = -pl[3] + ((pl[0] * w[0] + pl[1] * w[1]) + pl[2] * w[2]);
      }
    }
    // projected Gauss-Seidel on B, warm-started from the last lambda (:372)
    for (int s = 0; s < a.gs_max_it; ++s) {
      double ss = 0.0;
      for (int r = 0; r < rounds; ++r) {
        const int v = vertex(r);
        if (!on || comp != 0 || v >= a.nv) continue;
        double *S = own(r);
        const int nq = __ldg(a.plane_ptr + v + 1) - __ldg(a.plane_ptr + v);
        double old[3] = {0.0, 0.0, 0.0}, l[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 3; ++i)
          if (i < nq) old[i] = S[i];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (i >= nq) continue;
          double ub = 0.0;
#pragma unroll
          for (int j = i + 1; j < 3; ++j)
            if (j < nq) ub = ub + S[6 + 3 * i + j] * old[j];
          double rr = S[3 + i] - ub;
#pragma unroll
          for (int j = 0; j < i; ++j) rr -= l[j] * S[6 + 3 * i + j];
          const double li = rr * S[15 + i];
          l[i] = li > 0 ? li : 0;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (i >= nq) continue;
          S[i] = l[i];
          const double d = l[i] - old[i];
          ss = ss + d * d;
        }
      }
      const double tot = cluster_sum(ss, s_red, &s_tot, par, rank, ncta);
      par ^= 1;
      ++sweeps;
      if (sqrt(tot) <= a.gs_tol) break;
    }
    __syncwarp();
    // rhs = J^T lambda - Ua x + r (old x)                              (:374)
#pragma unroll
    for (int r = 0; r < kCMaxRounds; ++r) {
      const int v = vertex(r);
      if (r >= rounds || !on || v >= a.nv) continue;
      const double *S = own(r);
      double jl = 0.0;
      const int q0 = __ldg(a.plane_ptr + v), nq = __ldg(a.plane_ptr + v + 1) - q0;
      for (int j = 0; j < nq; ++j) jl = jl + S[j] * __ldg(a.planes + 4 * (size_t)(q0 + j) + comp);
      a.rhs[3 * v + comp] = (jl - ua[r]) + a.r[3 * v + comp];
    }
    cluster_barrier();
    // 3x3-block Gauss-Seidel sweep (:377-388), level by level.
    const int half = warp & 1, hw = warp >> 1, stride = ncta * (kCWarps / 2) * kCRows;
    const int first = (hw * ncta + rank) * kCRows;  // the warp's first row of a level
    LevelRow R;
    bool have = false;  // R holds a row of the half's next level, its leading terms taken
    auto prepare_level = [&](int lv) {
      const int t = __ldg(a.lvl_ptr + lv) + first + sub;
      have = on && t < __ldg(a.lvl_ptr + lv + 1);
      if (have) {
        R.load(C, t, comp);
        R.take(0, R.pre, x);
      }
    };
    auto finish = [&](bool ok) {  // the rest of the row, then Da^-1
      if (ok) R.take(R.pre, R.nlow, x);
      const double acc = ok ? R.acc : 0.0;
      const double r0 = __shfl_sync(0xffffffffu, acc, lead), r1 = __shfl_sync(0xffffffffu, acc, lead + 1),
                   r2 = __shfl_sync(0xffffffffu, acc, lead + 2);
      if (ok) {
        const double *M = a.inv + 9 * (size_t)R.v + 3 * comp;
        const double xn = (M[0] * r0 + M[1] * r1) + M[2] * r2;
        for (int p = 0; p < ncta; ++p) st_peer(peer_addr(x + 3 * R.v + comp, (unsigned int)p), xn);
      }
    };
    if (half == 0) prepare_level(0);
    for (int lv = 0; lv < a.nlevels; ++lv) {
      if (half == (lv & 1)) {
        finish(have);
        const int end = __ldg(a.lvl_ptr + lv + 1);
        for (int t0 = __ldg(a.lvl_ptr + lv) + first + stride; t0 < end; t0 += stride) {  // a wide level
          const bool ok = on && t0 + sub < end;
          if (ok) {
            R.load(C, t0 + sub, comp);
            R.take(0, R.pre, x);
          }
          finish(ok);
        }
      } else if (lv + 1 < a.nlevels) {
        prepare_level(lv + 1);
      }
      cluster_barrier();
    }
    const double tot = cluster_sum(pass(), s_red, &s_tot, par, rank, ncta);
    par ^= 1;
    res = sqrt(tot);
    if (res <= a.tol) {
      conv = 1;
      break;
    }
  }
  for (int r = 0; r < rounds; ++r) {
    const int v = vertex(r);
    if (!on || v >= a.nv) continue;
    a.x[3 * v + comp] = x[3 * v + comp];
    if (comp != 0) continue;
    const int q0 = a.plane_ptr[v], nq = a.plane_ptr[v + 1] - q0;
    for (int j = 0; j < nq; ++j) a.lam[q0 + j] = own(r)[j];
  }
  if (rank == 0 && threadIdx.x == 0) {
    a.out[0] = (double)it;
    a.out[1] = (double)conv;
    a.out[2] = res;
    a.out[3] = (double)sweeps;
  }
  cluster_barrier();  // no CTA leaves while another may write to its x
}

// Shared memory of a CTA of the cluster form.
size_t ica_cluster_smem(int nv, int ncta) {
  const int rounds = (nv + kCOwn * ncta - 1) / (kCOwn * ncta);
  return sizeof(double) * (3 * (size_t)nv + (size_t)kCState * rounds * kCOwn);
}
cudaError_t ica_cluster_config(int ncta, size_t smem, cudaStream_t s, cudaLaunchConfig_t &cfg,
                               cudaLaunchAttribute (&at)[1]) {
  cfg = {};
  cfg.gridDim = dim3((unsigned int)ncta);
  cfg.blockDim = dim3(kCThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned int)ncta;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaFuncSetAttribute(ica_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       200 * 1024);
  if (e == cudaSuccess && ncta > 8)
    e = cudaFuncSetAttribute(ica_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

int fail(int code, const char *what) {
  mprgp::set_last_error(what);
  return code;
}

}  // namespace

extern "C" {

int mprgp_ica_solve(mprgp_context *ctx, int nv, int nnzb, const int *row_ptr, const int *cols,
                    const double *vals, const double *r, const int *plane_ptr,
                    const double *planes, double *x, double *lambda, int max_it, double tol,
                    int gs_max_it, double gs_tol, mprgp_ica_stats *stats) {
  if (!ctx || nv <= 0 || nnzb <= 0 || !row_ptr || !cols || !vals || !r || !plane_ptr || !x ||
      max_it < 0 || gs_max_it < 0 || !(tol >= 0.0) || !(gs_tol >= 0.0))
    return fail(MPRGP_INVALID, "ica_solve: arguments");
  if (mprgp::context_lanes_busy(ctx))
    return fail(MPRGP_BUSY, "ica_solve: the context has asynchronous server runs in flight");
  const int m = plane_ptr[nv];
  if (m < 0 || (m > 0 && (!planes || !lambda))) return fail(MPRGP_INVALID, "ica_solve: planes");
  if (row_ptr[0] != 0 || row_ptr[nv] != nnzb) return fail(MPRGP_INVALID, "ica_solve: row_ptr");
  // Dependency levels of the block sweep and the checks the kernel relies
  // on: a diagonal block in every row, columns in range, <= 3 planes a vertex.
  std::vector<int> level(nv, 0), cnt(1, 0);
  int nlevels = 0, max_low = 0;
  bool leading = true;  // in every row the blocks left of the diagonal come first
  for (int v = 0; v < nv; ++v) {
    if (plane_ptr[v + 1] < plane_ptr[v] || plane_ptr[v + 1] - plane_ptr[v] > 3)
      return fail(MPRGP_INVALID, "ica_solve: 0..3 planes per vertex");
    if (row_ptr[v + 1] < row_ptr[v]) return fail(MPRGP_INVALID, "ica_solve: row_ptr");
    bool diag = false;
    int lv = 0, low = 0;
    for (int k = row_ptr[v]; k < row_ptr[v + 1]; ++k) {
      const int u = cols[k];
      if (u < 0 || u >= nv) return fail(MPRGP_INVALID, "ica_solve: column out of range");
      if (u == v) diag = true;
      if (u < v) {
        lv = std::max(lv, level[u] + 1);
        leading &= k - row_ptr[v] == low;
        ++low;
      }
    }
    max_low = std::max(max_low, low);
    if (!diag) return fail(MPRGP_INVALID, "ica_solve: missing diagonal block");
    level[v] = lv;
    nlevels = std::max(nlevels, lv + 1);
  }
  std::vector<int> lvl_ptr(nlevels + 1, 0), order(nv);
  for (int v = 0; v < nv; ++v) lvl_ptr[level[v] + 1]++;
  for (int l = 0; l < nlevels; ++l) lvl_ptr[l + 1] += lvl_ptr[l];
  {
    std::vector<int> fill(lvl_ptr.begin(), lvl_ptr.end() - 1);
    for (int v = 0; v < nv; ++v) order[fill[level[v]]++] = v;
  }
  // The cluster form for small bodies (about 64 vertices a CTA, 16 CTAs at
  // most), when its row window and shared memory hold the problem and the
  // device offers the cluster.  Both sides at 1,377 vertices: 18.7 against
  // 57 ms; at 425: 13.2 against 51.
  int ncta = 1;
  while (ncta < kCCtas && 64 * ncta < nv) ncta *= 2;
  bool clustered = leading && max_low <= kCLow && nv <= kCMaxRounds * kCOwn * ncta;
  const size_t csmem = ica_cluster_smem(nv, ncta);
  cudaLaunchConfig_t ccfg;
  cudaLaunchAttribute cat[1];
  std::vector<IcaRow> rows;
  if (clustered) {
    int fits = 0;
    clustered = ica_cluster_config(ncta, csmem, (cudaStream_t)mprgp_context_stream(ctx), ccfg, cat) ==
                    cudaSuccess &&
                cudaOccupancyMaxActiveClusters(&fits, ica_cluster_kernel, &ccfg) == cudaSuccess &&
                fits >= 1;
    cudaGetLastError();
  }
  if (clustered) {
    rows.resize(nv);
    for (int t = 0; t < nv; ++t) {
      const int v = order[t], k0 = row_ptr[v];
      int low = 0, pre = 0;
      while (k0 + low < row_ptr[v + 1] && cols[k0 + low] < v) ++low;
      while (pre < low && level[cols[k0 + pre]] <= level[v] - 2) ++pre;
      rows[t] = {v, k0, low, pre};
    }
  }
  int dev = 0, nsm = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ica_kernel, kIcaThreads, 0) !=
          cudaSuccess || per_sm < 1)
    return fail(MPRGP_CUDA_ERROR, "ica_solve: occupancy");
  const int grid = std::max(1, std::min(nsm, (nv + kIcaThreads - 1) / kIcaThreads));
  cudaStream_t s = (cudaStream_t)mprgp_context_stream(ctx);
  const size_t n = 3 * (size_t)nv, mm = std::max(m, 1);
  // one device block for everything, carved in 256-byte steps
  size_t off = 0;
  auto take = [&off](size_t bytes) {
    const size_t at = off;
    off = (off + bytes + 255) & ~size_t(255);
    return at;
  };
  const size_t o_rp = take(sizeof(int) * (nv + 1)), o_cols = take(sizeof(int) * nnzb),
               o_vals = take(sizeof(double) * 9 * (size_t)nnzb), o_r = take(sizeof(double) * n),
               o_pp = take(sizeof(int) * (nv + 1)), o_pl = take(sizeof(double) * 4 * mm),
               o_ord = take(sizeof(int) * nv), o_lp = take(sizeof(int) * (nlevels + 1)),
               o_x = take(sizeof(double) * n), o_lam = take(sizeof(double) * mm),
               o_c = take(sizeof(double) * mm), o_rhs = take(sizeof(double) * n),
               o_inv = take(sizeof(double) * 9 * (size_t)nv),
               o_B = take(sizeof(double) * 9 * (size_t)nv),
               o_part = take(sizeof(double) * 2 * grid), o_ctl = take(sizeof(IcaCtl)),
               o_out = take(sizeof(double) * 4),
               o_rows = take(sizeof(IcaRow) * rows.size());
  unsigned char *d = nullptr;
  if (cudaMallocAsync((void **)&d, off, s) != cudaSuccess)
    return fail(MPRGP_OOM, "ica_solve: device memory");
  int rc = MPRGP_OK;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  double out[4] = {0, 0, 0, 0};
  float ms = 0.f;
  auto up = [&](size_t o, const void *h, size_t bytes) {
    return cudaMemcpyAsync(d + o, h, bytes, cudaMemcpyHostToDevice, s);
  };
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = up(o_rp, row_ptr, sizeof(int) * (nv + 1));
  if (e == cudaSuccess) e = up(o_cols, cols, sizeof(int) * nnzb);
  if (e == cudaSuccess) e = up(o_vals, vals, sizeof(double) * 9 * (size_t)nnzb);
  if (e == cudaSuccess) e = up(o_r, r, sizeof(double) * n);
  if (e == cudaSuccess) e = up(o_pp, plane_ptr, sizeof(int) * (nv + 1));
  if (e == cudaSuccess && m > 0) e = up(o_pl, planes, sizeof(double) * 4 * (size_t)m);
  if (e == cudaSuccess) e = up(o_ord, order.data(), sizeof(int) * nv);
  if (e == cudaSuccess) e = up(o_lp, lvl_ptr.data(), sizeof(int) * (nlevels + 1));
  if (e == cudaSuccess && clustered) e = up(o_rows, rows.data(), sizeof(IcaRow) * rows.size());
  if (e == cudaSuccess) e = up(o_x, x, sizeof(double) * n);
  if (e == cudaSuccess) e = cudaMemsetAsync(d + o_ctl, 0, sizeof(IcaCtl), s);
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  if (e == cudaSuccess) {
    IcaArgs a;
    a.nv = nv;
    a.m = m;
    a.nlevels = nlevels;
    a.max_it = max_it;
    a.gs_max_it = gs_max_it;
    a.tol = tol;
    a.gs_tol = gs_tol;
    a.row_ptr = (const int *)(d + o_rp);
    a.cols = (const int *)(d + o_cols);
    a.vals = (const double *)(d + o_vals);
    a.r = (const double *)(d + o_r);
    a.plane_ptr = (const int *)(d + o_pp);
    a.planes = (const double *)(d + o_pl);
    a.order = (const int *)(d + o_ord);
    a.lvl_ptr = (const int *)(d + o_lp);
    a.x = (double *)(d + o_x);
    a.lam = (double *)(d + o_lam);
    a.c = (double *)(d + o_c);
    a.rhs = (double *)(d + o_rhs);
    a.inv = (double *)(d + o_inv);
    a.B = (double *)(d + o_B);
    a.part = (double *)(d + o_part);
    a.ctl = (IcaCtl *)(d + o_ctl);
    a.out = (double *)(d + o_out);
    a.wait_ns = 5000000000LL;  // 5 s per barrier wait
    void *params[] = {&a};
    if (clustered) {
      e = cudaEventRecord(e0, s);
      IcaClusterArgs ca;
      ca.a = a;
      ca.rows = (const IcaRow *)(d + o_rows);
      if (e == cudaSuccess) e = cudaLaunchKernelEx(&ccfg, ica_cluster_kernel, ca);
    } else {
      e = mprgp::gated_launch(s, nsm, grid, [&] {
        const cudaError_t r = cudaEventRecord(e0, s);  // (behind the runs it waits for)
        return r != cudaSuccess ? r
                                : cudaLaunchCooperativeKernel((const void *)ica_kernel, dim3(grid),
                                                              dim3(kIcaThreads), params, 0, s);
      });
    }
    if (e == cudaSuccess) e = cudaEventRecord(e1, s);
  }
  IcaCtl ctl{};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&ctl, d + o_ctl, sizeof(IcaCtl), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, d + o_out, sizeof(out), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(x, d + o_x, sizeof(double) * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && m > 0)
    e = cudaMemcpyAsync(lambda, d + o_lam, sizeof(double) * m, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
  if (e != cudaSuccess) rc = fail(MPRGP_CUDA_ERROR, "ica_solve: CUDA call failed");
  else if (ctl.err == 2) rc = fail(MPRGP_CUDA_ERROR, "ica_solve: launched with another cluster size");
  else if (ctl.err) rc = fail(MPRGP_TIMEOUT, "ica_solve: device wait limit reached");
  cudaFreeAsync(d, s);
  cudaStreamSynchronize(s);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (rc) return rc;
  if (stats) {
    stats->iterations = (int)out[0];
    stats->converged = (int)out[1];
    stats->residual = out[2];
    stats->pgs_sweeps = (long long)out[3];
    stats->levels = nlevels;
    stats->device_ms = ms;
  }
  return out[1] != 0.0 ? MPRGP_OK : MPRGP_NOT_CONVERGED;
}

}  // extern "C"
