// Admission of many small formulas at once: the host lays the formulas' literals and initial
// states side by side in one page-locked block, and one launch unpacks them into the pack's
// arrays and builds every formula's occurrence lists, one block per formula.
//
// Admitting a formula by itself is about 12 launches and copies (60-110 us of host time); here
// a formula costs the host one pass over its arrays (check, copy, round) and its share of one
// copy and one launch.  The lists are the ones the per-formula build makes: ascending slots.
#pragma once

#include "dmm_kernels.cuh"
#include "dmm_xprep.cuh"

namespace dmm {

constexpr int kAdmitThreads = 1024;
constexpr int kAdmitVars = 16384;         // variables whose counters fit beside the sorters
constexpr int64_t kAdmitSlots = 1 << 18;  // larger formulas are built by the whole device

struct AdmitRec {
  InstDesc I;
  InstCtrl c;
  int64_t lit, coff, unit, x;  // byte offsets in the block (coff, unit: -1 when absent)
  int32_t idx, pad;
};

template <class T>
__global__ void __launch_bounds__(kAdmitThreads)
    k_admit(const AdmitRec* __restrict__ recs, const unsigned char* __restrict__ blob,
            InstDesc* inst, InstCtrl* ctrl, int32_t* lit_all, int32_t* vslot_all, int32_t* upos_all,
            int32_t* vend_all, int32_t* coff_all, int8_t* unit_all, T* cand, T* Xs, T* Xl,
            int32_t* active, int32_t* longv, int32_t* nlong, int32_t long_cap) {
  constexpr int NT = kAdmitThreads;
  extern __shared__ int32_t ad_smem[];
  __shared__ int wsum[32];
  __shared__ AdmitRec R;
  for (unsigned q = threadIdx.x; q < sizeof(AdmitRec) / 4; q += NT)
    reinterpret_cast<int32_t*>(&R)[q] = reinterpret_cast<const int32_t*>(recs + blockIdx.x)[q];
  __syncthreads();
  const InstDesc& I = R.I;
  const int n = I.n, m = I.m, L = I.nslots, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int32_t* const at = ad_smem;                               // [n] counts, then list cursors
  int32_t* const buf = ad_smem + ((n + 31) & ~31) + w * kSortCap;  // [kSortCap] per warp
  const int32_t* const src = reinterpret_cast<const int32_t*>(blob + R.lit);
  int32_t* const lit = lit_all + I.slot0;
  int32_t* const vslot = vslot_all + I.slot0;
  int32_t* const upos = upos_all + I.slot0;
  int32_t* const vend = vend_all + I.var0;
  for (int v = threadIdx.x; v < n; v += NT) at[v] = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < L; s += NT) {
    const int l = src[s];
    lit[s] = l;
    atomicAdd(&at[abs(l) - 1], 1);
  }
  __syncthreads();
  int carry = 0;
  for (int v0 = 0; v0 < n; v0 += NT) {
    const int v = v0 + threadIdx.x;
    const int c = v < n ? at[v] : 0;
    int tot;
    const int ex = block_exscan<NT>(c, wsum, &tot);
    if (v < n) {
      at[v] = carry + ex;
      vend[v] = carry + ex + c;
    }
    carry += tot;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < L; s += NT) vslot[atomicAdd(&at[abs(src[s]) - 1], 1)] = s;
  __syncthreads();  // at[v]: end of the list
  for (int v = w; v < n; v += NT / 32) {
    const int e0 = v > 0 ? at[v - 1] : 0, d = at[v] - e0;
    if (d <= 32) {  // rank by shuffles
      const int s = lane < d ? vslot[e0 + lane] : 0x7fffffff;
      int r = 0;
#pragma unroll
      for (int j = 0; j < 32; j++) r += __shfl_sync(0xffffffffu, s, j) < s;
      __syncwarp();
      if (lane < d) {
        vslot[e0 + r] = s;
        upos[s] = e0 + r;
      }
      continue;
    }
    if (d > kSortCap) {  // left to the host's sort; the positions follow then
      if (lane == 0) {
        const int pos = atomicAdd(nlong, 1);
        if (pos < long_cap) longv[pos] = (int32_t)I.var0 + v;
      }
      continue;
    }
    int N = 64;
    while (N < d) N <<= 1;
    for (int j = lane; j < N; j += 32) buf[j] = j < d ? vslot[e0 + j] : 0x7fffffff;
    __syncwarp();
    for (int k = 2; k <= N; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int e = lane; e < N; e += 32) {
          const int p = e ^ j;
          if (p > e) {
            const bool up = (e & k) == 0;
            const int32_t x = buf[e], y = buf[p];
            if (up ? (y < x) : (x < y)) {
              buf[e] = y;
              buf[p] = x;
            }
          }
        }
        __syncwarp();
      }
    for (int j = lane; j < d; j += 32) {
      vslot[e0 + j] = buf[j];
      upos[buf[j]] = e0 + j;
    }
    __syncwarp();
  }
  const T* const x = reinterpret_cast<const T*>(blob + R.x);
  for (int v = threadIdx.x; v < n; v += NT) cand[I.var0 + v] = x[v];
  for (int c = threadIdx.x; c < m; c += NT) {
    Xs[I.cls0 + c] = x[n + c];
    Xl[I.cls0 + c] = x[n + m + c];
  }
  for (int v = threadIdx.x; v < n; v += NT)
    unit_all[I.var0 + v] = R.unit >= 0 ? reinterpret_cast<const int8_t*>(blob + R.unit)[v] : 0;
  if (R.coff >= 0)
    for (int c = threadIdx.x; c < m; c += NT)
      coff_all[I.cls0 + c] = reinterpret_cast<const int32_t*>(blob + R.coff)[c];
  if (threadIdx.x == 0) {
    inst[R.idx] = I;
    ctrl[R.idx] = R.c;
    if (blockIdx.x == 0) atomicAdd(active, (int)gridDim.x);
  }
}

// Reported assignments (signs of the current V) of `count` formulas: out[off[k] ..], formula k by
// the blocks (k, y): one block each is enough for the small formulas of a large batch, but a large
// one among them would be a chain of loads in one block.
template <class T>
__global__ void k_signs_all(const InstDesc* __restrict__ inst, const InstCtrl* __restrict__ ctrl,
                            const int32_t* __restrict__ idx, const int64_t* __restrict__ off,
                            const T* __restrict__ cand, int64_t var_cap, int8_t* __restrict__ out) {
  const int i = idx[blockIdx.x];
  const T* v = cand + (int64_t)(ctrl[i].set * kTrials + ctrl[i].kcur) * var_cap + inst[i].var0;
  int8_t* o = out + off[blockIdx.x];
  const int n = inst[i].n;
  for (int k = blockIdx.y * blockDim.x + threadIdx.x; k < n; k += gridDim.y * blockDim.x)
    o[k] = v[k] > T(0) ? 1 : -1;
}

}  // namespace dmm
