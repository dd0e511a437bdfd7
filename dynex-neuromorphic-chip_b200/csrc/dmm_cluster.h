// Host interface of the cluster form (dmm_cluster.cuh, cluster.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace dmm {

constexpr int kClusterSizes = 5;        // blocks per cluster: 1, 2, 4, 8, 16
constexpr int kClusterMax = 16;         // the largest (a non-portable size)
constexpr int kClusterMaxVars = 32767;  // 16-bit literals
constexpr int kClusterThreads = 1024;   // block size, at most
constexpr int kClusterThreads64 = 512;  // ... in FP64 (the sorted sums' registers)
constexpr int kClusterSmemMax = 223 * 1024;  // dynamic shared memory, at most

// Capacities of one launch (the largest of its formulas); the shared-memory layout follows.
struct ClusterCaps {
  int n;       // variables
  int tc, ts;  // clauses and literal slots of a block
  int tv, bk;  // variables and bucket entries of a block
};

// Split of a formula over R blocks: contiguous clause and variable ranges (a block's
// variables start at a multiple of 4: its dV are sent as 16-byte words).
__host__ __device__ inline int cluster_tc(int m, int R) { return (m + R - 1) / R; }
__host__ __device__ inline int cluster_tv(int n, int R) { return ((n + R - 1) / R + 3) & ~3; }

struct InstDesc;
// The kernel for a precision and clause kind, its dynamic shared memory and block size.
const void* cluster_kernel(bool fp64, bool general);
int cluster_smem(const ClusterCaps& caps, bool fp64, bool general);
int cluster_threads(const ClusterCaps& caps, bool fp64);
// Queues the largest bucket and literal-slot count of a block when each of `count` listed
// formulas is split over 1, 2, 4, 8 and 16 blocks: out[f * kClusterSizes + size].
cudaError_t cluster_need(const InstDesc* inst, const int32_t* list, int count,
                         const int32_t* vend, const int32_t* coff, int2* out, cudaStream_t s);

}  // namespace dmm
