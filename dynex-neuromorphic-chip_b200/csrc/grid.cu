// Instantiations, table build and launch parameters of the resident grid form (dmm_grid.cuh).
#include <algorithm>

#include "dmm_grid.cuh"
#include "dmm_gridprep.cuh"

namespace dmm {

static_assert(sizeof(GridSync) == kGridSyncBytes, "group counters");

template <class T, bool GENERAL>
static const void* grid_kernel_t(int resident) {
  return resident == 2   ? (const void*)k_grid<T, GENERAL, 2>
         : resident == 1 ? (const void*)k_grid<T, GENERAL, 1>
                         : (const void*)k_grid<T, GENERAL, 0>;
}

const void* grid_kernel(bool fp64, bool general, int resident) {
  if (fp64) return general ? grid_kernel_t<double, true>(resident) : grid_kernel_t<double, false>(resident);
  return general ? grid_kernel_t<float, true>(resident) : grid_kernel_t<float, false>(resident);
}

GridLayout grid_shape(const GridCaps& c, bool fp64, bool general, int resident) {
  return grid_layout(c, fp64 ? 8 : 4, general, resident);
}

template <class T>
static __global__ void k_grid_unset(T* a, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    a[i] = Unset<T>::bits();
}

cudaError_t grid_unset(const GridTables& t, bool fp64, cudaStream_t s) {
  for (int q = 0; q < 2; q++) {
    void* a = q ? t.inbox : t.ux;
    const int64_t n = 2 * (q ? t.inbox_len : t.ux_len);
    const int grid = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
    if (n == 0) continue;
    if (fp64) k_grid_unset<<<grid, 256, 0, s>>>(static_cast<unsigned long long*>(a), n);
    else k_grid_unset<<<grid, 256, 0, s>>>(static_cast<unsigned int*>(a), n);
  }
  return cudaGetLastError();
}

cudaError_t grid_build(const GridGroup* groups, const int32_t* list_group, int ngroups,
                       int nlists, int max_n, int max_nct, int max_nvt, int max_rows, const int32_t* lit,
                       const int32_t* upos, const int32_t* vend, const int32_t* coff,
                       const GridTables& t, bool fp64, cudaStream_t s) {
  const int RW = std::min((max_n + 31) / 32, kXpRangeWords), kw = fp64 ? 2 : 4;
  const int smem = (max_nvt + 2 * RW) * 4;
  const void* fill = fp64 ? (const void*)k_grid_fill<true> : (const void*)k_grid_fill<false>;
  cudaError_t e = allow_smem((const void*)k_grid_count, kGridSmemMax);
  if (e == cudaSuccess) e = allow_smem(fill, kGridSmemMax);
  if (e != cudaSuccess) return e;
  if (t.pos)
    k_grid_order<<<dim3((unsigned)max_nvt, (unsigned)ngroups), kGridRowThreads, 0, s>>>(groups, vend, t);
  if (t.cord)
    k_grid_clauses<<<dim3((unsigned)max_nct, (unsigned)ngroups), kGridRowThreads, 0, s>>>(groups, coff, t);
  k_grid_count<<<nlists, kGridPrepThreads, smem, s>>>(groups, list_group, lit, coff, t, RW, kw);
  k_grid_rows<<<dim3((unsigned)max_rows, (unsigned)ngroups), kGridRowThreads, 0, s>>>(groups, t, kw);
  k_grid_scan<<<ngroups, kGridPrepThreads, 0, s>>>(groups, coff, vend, t, kw);
  if (fp64)
    k_grid_fill<true><<<nlists, kGridPrepThreads, smem, s>>>(groups, list_group, lit, upos, vend,
                                                             coff, t, RW, kw);
  else
    k_grid_fill<false><<<nlists, kGridPrepThreads, smem, s>>>(groups, list_group, lit, upos, vend,
                                                              coff, t, RW, kw);
  return cudaGetLastError();
}

void grid_functions(bool fp64, std::vector<const void*>* out) {
  for (int q = 0; q < 6; q++) out->push_back(grid_kernel(fp64, q & 1, q >> 1));
  out->push_back(fp64 ? (const void*)k_grid_unset<unsigned long long>
                      : (const void*)k_grid_unset<unsigned int>);
  out->push_back(fp64 ? (const void*)k_grid_fill<true> : (const void*)k_grid_fill<false>);
  out->insert(out->end(), {(const void*)k_grid_order, (const void*)k_grid_clauses,
                           (const void*)k_grid_count, (const void*)k_grid_rows,
                           (const void*)k_grid_scan});
}

}  // namespace dmm
