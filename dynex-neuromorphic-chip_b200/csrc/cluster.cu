// Instantiations and launch parameters of the cluster form (dmm_cluster.cuh).
#include <algorithm>

#include "dmm_cluster.cuh"

namespace dmm {

const void* cluster_kernel(bool fp64, bool general) {
  if (fp64)
    return general ? (const void*)k_cluster<double, true> : (const void*)k_cluster<double, false>;
  return general ? (const void*)k_cluster<float, true> : (const void*)k_cluster<float, false>;
}

int cluster_smem(const ClusterCaps& caps, bool fp64, bool general) {
  return cluster_layout(caps, fp64 ? 8 : 4, general).total;
}

// A thread per clause and eight lanes per variable (FP64: one thread, or a warp), as far as
// the block goes; a step of a small block costs mostly what its warps repeat (reductions, the
// decision), so no more warps than that.
int cluster_threads(const ClusterCaps& caps, bool fp64) {
  const int per_var = !fp64 ? 8 : cluster_rank_all(caps.tv) ? 32 : 1;
  const int want = std::max(caps.tc, per_var * caps.tv);
  const int most = fp64 ? kClusterThreads64 : kClusterThreads;
  return std::min(most, std::max(fp64 ? 256 : 128, (want + 31) / 32 * 32));
}

// Largest bucket and literal-slot count of a block when each listed formula is split over
// 1, 2, 4, 8 and 16 blocks: out[f][size] = {bucket entries, slots}.  One warp per formula, one
// lane per block of each size.
static __global__ void k_cluster_need(const InstDesc* __restrict__ inst, const int32_t* __restrict__ list,
                               const int32_t* __restrict__ vend, const int32_t* __restrict__ coff,
                               int2* __restrict__ out) {
  const InstDesc I = inst[list[blockIdx.x]];
  __shared__ int mx[kClusterSizes][2];
  const int lane = threadIdx.x;
  if (lane < kClusterSizes) mx[lane][0] = mx[lane][1] = 0;
  __syncwarp();
  if (lane < 31) {
    const int q = 31 - __clz(lane + 1), R = 1 << q, b = lane + 1 - R;
    const int TV = cluster_tv(I.n, R), TC = cluster_tc(I.m, R);
    const int v0 = min(I.n, b * TV), v1 = min(I.n, v0 + TV);
    const int c0 = min(I.m, b * TC), c1 = min(I.m, c0 + TC);
    const int e0 = v0 > 0 ? vend[I.var0 + v0 - 1] : 0, e1 = v1 > 0 ? vend[I.var0 + v1 - 1] : 0;
    int ts = 3 * (c1 - c0);
    if (!I.k3)
      ts = c1 <= c0 ? 0 : (c1 < I.m ? coff[I.cls0 + c1] : I.nslots) - coff[I.cls0 + c0];
    atomicMax(&mx[q][0], e1 - e0);
    atomicMax(&mx[q][1], ts);
  }
  __syncwarp();
  if (lane < kClusterSizes)
    out[blockIdx.x * kClusterSizes + lane] = make_int2(mx[lane][0], mx[lane][1]);
}

cudaError_t cluster_need(const InstDesc* inst, const int32_t* list, int count,
                         const int32_t* vend, const int32_t* coff, int2* out, cudaStream_t s) {
  k_cluster_need<<<(unsigned)count, 32, 0, s>>>(inst, list, vend, coff, out);
  return cudaGetLastError();
}

}  // namespace dmm
