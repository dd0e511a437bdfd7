// Device construction of the resident grid form's tables (dmm_grid.cuh), all groups at once.
//
//   k_grid_count  (one block per block of the grid) rank of every slot within its chunk
//                 (clause tile t, variable tile v), chunk sizes, staging offsets; the block's
//                 number of distinct variables and how many lie below each block's variables.
//   k_grid_scan   (one block per group) offsets over tiles and blocks, the limits.
//   k_grid_fill   (one block per block of the grid) variable lists, local literals, staging
//                 places and destinations, bucket places in variable-major order, send lists.
//
// Slot order inside a chunk is arbitrary: both sides use the same rank, and a variable's
// contributions are summed in CSR order through their bucket places.
#pragma once

#include "dmm_grid.h"
#include "dmm_step.cuh"
#include "dmm_xprep.cuh"

namespace dmm {

constexpr int kGridPrepThreads = 1024;

// First slot of clause c (c may be m) of a group's formula.
__device__ __forceinline__ int grid_slot(const GridGroup& g, const int32_t* coff, int c) {
  return g.k3 ? 3 * c : c < g.m ? coff[g.cls0 + c] : g.L;
}

__global__ void __launch_bounds__(kGridPrepThreads)
    k_grid_count(const GridGroup* __restrict__ groups, const int32_t* __restrict__ blk_group,
                 const int32_t* __restrict__ lit_all, const int32_t* __restrict__ coff, GridTables t,
                 int RW, int kw) {
  constexpr int NT = kGridPrepThreads;
  extern __shared__ __align__(16) int gp_smem[];
  __shared__ int wsum[32];
  const GridGroup g = groups[blk_group[blockIdx.x]];
  const int b = blockIdx.x - g.blk0, nvt = g.nvt;
  const int32_t* lit = lit_all + g.slot0;
  int* c_s = gp_smem;
  unsigned* bits = reinterpret_cast<unsigned*>(gp_smem + nvt);
  int* wpre = gp_smem + nvt + RW;
  for (int i = 0; i < g.kc; i++) {
    const int ct = b * g.kc + i;
    const int s_lo = grid_slot(g, coff, min(g.m, ct * g.TC)),
              s_hi = grid_slot(g, coff, min(g.m, (ct + 1) * g.TC));
    for (int v = threadIdx.x; v < nvt; v += NT) c_s[v] = 0;
    __syncthreads();
    for (int s = s_lo + threadIdx.x; s < s_hi; s += NT)
      t.spos[g.o_slot + s] = (uint16_t)atomicAdd(&c_s[(abs(__ldg(lit + s)) - 1) / g.TV], 1);
    __syncthreads();
    int at = 0;
    for (int v0 = 0; v0 < nvt; v0 += NT) {
      const int v = v0 + threadIdx.x;
      const int c = v < nvt ? c_s[v] : 0, p = (c + kw - 1) / kw * kw;
      int tot;
      const int ex = block_exscan<NT>(p, wsum, &tot);
      if (v < nvt) {
        t.cnt[g.o_pair + (int64_t)ct * nvt + v] = c;
        t.sb[g.o_pair + (int64_t)ct * nvt + v] = at + ex;
      }
      at += tot;
    }
    if (threadIdx.x == 0) t.st[g.o_ct + ct] = at;
  }
  // distinct variables, and those below each block's first variable
  const int s_lo = grid_slot(g, coff, min(g.m, b * g.kc * g.TC)),
            s_hi = grid_slot(g, coff, min(g.m, (b + 1) * g.kc * g.TC));
  const int TVb = g.TV * g.kv;
  int32_t* dlo = t.dlo + g.o_bb + (int64_t)b * (g.B + 1);
  int before = 0;
  for (int r0 = 0; r0 < g.n; r0 += 32 * RW) {
    const int nr = xp_bitmap<NT>(lit, s_lo, s_hi, bits, wpre, r0, RW, wsum);
    for (int c = threadIdx.x; c < g.B; c += NT) {
      const int64_t x = (int64_t)c * TVb - r0;
      if (x >= 0 && x < 32 * RW)
        dlo[c] = before + wpre[x >> 5] + __popc(bits[x >> 5] & ((1u << (x & 31)) - 1u));
    }
    before += nr;
    __syncthreads();
  }
  for (int c = threadIdx.x; c <= g.B; c += NT)
    if (c == g.B || (int64_t)c * TVb >= ((int64_t)(g.n + 32 * RW - 1) / (32 * RW)) * 32 * RW)
      dlo[c] = before;
  if (threadIdx.x == 0) t.dcnt[g.o_blk + b] = before;
}

__global__ void __launch_bounds__(kGridPrepThreads)
    k_grid_scan(const GridGroup* __restrict__ groups, const int32_t* __restrict__ coff,
                const int32_t* __restrict__ vend, GridTables t, int kw) {
  constexpr int NT = kGridPrepThreads;
  __shared__ int s_bad, s_max[8], s_tot[1024];
  const GridGroup g = groups[blockIdx.x];
  const int nct = g.nct, nvt = g.nvt, B = g.B;
  if (threadIdx.x < 8) s_max[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0;
    for (int b = 0; b < B; b++) {
      const int d = t.dcnt[g.o_blk + b];
      t.dinfo[g.o_blk + b] = make_int2(at, d);
      at += (d + 3) & ~3;
      s_max[1] = max(s_max[1], (d + 3) & ~3);
    }
    if (s_max[1] > kGridMaxDistinct) atomicExch(&s_bad, 1);
  } else if (threadIdx.x == 32) {
    int at = 0, mx = 0;
    for (int c = 0; c < nct; c++) {
      const int st = t.st[g.o_ct + c];
      t.woff[g.o_ct + c] = at;
      at += st / kw;
      mx = max(mx, st);
    }
    t.woff[g.o_ct + nct] = at;
    s_max[2] = mx;
    if (mx > 65535) atomicExch(&s_bad, 2);
  }
  // chunk offsets inside each bucket: one thread per variable tile; send lists: one per block
  for (int v = threadIdx.x; v < nvt; v += NT) {
    int at = 0;
    for (int c = 0; c < nct; c++) {
      t.bt[g.o_pair + (int64_t)v * nct + c] = at;
      at += (t.cnt[g.o_pair + (int64_t)c * nvt + v] + kw - 1) / kw * kw;
    }
    s_tot[v] = at;
    atomicMax(&s_max[3], at);
    if (at + kw > 65535) atomicExch(&s_bad, 3);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0;
    for (int v = 0; v < nvt; v++) {
      t.boff[g.o_vt + v] = at;
      at += s_tot[v];
    }
    t.boff[g.o_vt + nvt] = at;
  }
  __syncthreads();
  for (int b = threadIdx.x; b < B; b += NT) {
    int at = 0;
    for (int c = 0; c < B; c++) {
      const int32_t* dlo = t.dlo + g.o_bb + (int64_t)c * (B + 1);
      t.pinfo[g.o_bb + (int64_t)b * (B + 1) + c] = make_int2(at, t.dinfo[g.o_blk + c].x + dlo[b]);
      at += dlo[b + 1] - dlo[b];
    }
    t.pinfo[g.o_bb + (int64_t)b * (B + 1) + B] = make_int2(at, 0);
    s_tot[b] = at;
    atomicMax(&s_max[4], at);
    const int TVb = g.TV * g.kv, v0 = min(g.n, b * TVb), v1 = min(g.n, v0 + TVb);
    atomicMax(&s_max[7], (v1 > 0 ? vend[g.var0 + v1 - 1] : 0) - (v0 > 0 ? vend[g.var0 + v0 - 1] : 0));
    const int TCb = g.TC * g.kc;
    atomicMax(&s_max[5], grid_slot(g, coff, min(g.m, (b + 1) * TCb)) -
                             grid_slot(g, coff, min(g.m, b * TCb)));
    atomicMax(&s_max[6], t.woff[g.o_ct + (b + 1) * g.kc] - t.woff[g.o_ct + b * g.kc]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // the send lists of all blocks, one after another
    int base = 0;
    for (int b = 0; b < B; b++) {
      t.st[g.o_ct + b] = base;  // (the staging sizes are no longer needed)
      base += s_tot[b];
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < B * (B + 1); q += NT)
    t.pinfo[g.o_bb + q].x += t.st[g.o_ct + q / (B + 1)];
  if (threadIdx.x < 8) t.out[kGridOut * blockIdx.x + threadIdx.x] = threadIdx.x == 0 ? s_bad : s_max[threadIdx.x];
}

// ROW64: rows as the FP64 sums read them (32 variables side by side), else as the FP32 sums do.
template <bool ROW64>
__global__ void __launch_bounds__(kGridPrepThreads)
    k_grid_fill(const GridGroup* __restrict__ groups, const int32_t* __restrict__ blk_group,
                const int32_t* __restrict__ lit_all, const int32_t* __restrict__ upos_all,
                const int32_t* __restrict__ vend_all, const int32_t* __restrict__ coff, GridTables t,
                int RW, int kw) {
  constexpr int NT = kGridPrepThreads;
  extern __shared__ __align__(16) int gp_smem[];
  __shared__ int wsum[32];
  const int gi = blk_group[blockIdx.x];
  const GridGroup g = groups[gi];
  if (t.out[kGridOut * gi] != 0) return;  // a limit failed: the tables are not used
  const int b = blockIdx.x - g.blk0, nvt = g.nvt, nct = g.nct;
  const int32_t* lit = lit_all + g.slot0;
  const int32_t* upos = upos_all + g.slot0;
  const int32_t* vend = vend_all + g.var0;
  int* s_sb = gp_smem;  // [nvt] staging offset, then the bucket offset of this tile's chunk
  unsigned* bits = reinterpret_cast<unsigned*>(gp_smem + nvt);
  int* wpre = gp_smem + nvt + RW;
  for (int i = 0; i < g.kc; i++) {
    const int ct = b * g.kc + i;
    const int s_lo = grid_slot(g, coff, min(g.m, ct * g.TC)),
              s_hi = grid_slot(g, coff, min(g.m, (ct + 1) * g.TC));
    __syncthreads();
    for (int v = threadIdx.x; v < nvt; v += NT) s_sb[v] = t.sb[g.o_pair + (int64_t)ct * nvt + v];
    __syncthreads();
    for (int s = s_lo + threadIdx.x; s < s_hi; s += NT) {
      const int v = abs(__ldg(lit + s)) - 1, vt = v / g.TV;
      const int r = t.spos[g.o_slot + s];
      t.spos[g.o_slot + s] = (uint16_t)(s_sb[vt] + r);
      // place in the bucket (its first word is the padding entry of the rows)
      const uint16_t at = (uint16_t)(kw + t.bt[g.o_pair + (int64_t)vt * nct + ct] + r);
      const int p = __ldg(upos + s), j = p - (v > 0 ? __ldg(vend + v - 1) : 0);
      t.idx[g.o_slot + p] = at;
      const int vi = v - vt * g.TV;
      uint16_t* row = t.rows + g.o_row + (int64_t)vt * g.TVr * 32;
      if (j < 32)
        row[ROW64 ? ((vi >> 5) * 128 + (j >> 3) * 32 + (vi & 31)) * 8 + (j & 7)
                  : 32 * vi + 8 * (j & 3) + (j >> 2)] = at;
    }
    // destinations of the staging area's words
    const int w0 = t.woff[g.o_ct + ct];
    for (int v = threadIdx.x >> 5; v < nvt; v += NT / 32) {
      const int nw = (t.cnt[g.o_pair + (int64_t)ct * nvt + v] + kw - 1) / kw;
      const int d0 = (t.boff[g.o_vt + v] + t.bt[g.o_pair + (int64_t)v * nct + ct]) / kw;
      for (int q = threadIdx.x & 31; q < nw; q += 32)
        t.wdst[g.o_word + w0 + s_sb[v] / kw + q] = (uint32_t)(d0 + q);
    }
  }
  __syncthreads();
  // the block's variable list (ascending), local literals and entries of the send lists,
  // range by range
  const int s_lo = grid_slot(g, coff, min(g.m, b * g.kc * g.TC)),
            s_hi = grid_slot(g, coff, min(g.m, (b + 1) * g.kc * g.TC));
  const int TVb = g.TV * g.kv, d0 = t.dinfo[g.o_blk + b].x;
  const int32_t* dlo = t.dlo + g.o_bb + (int64_t)b * (g.B + 1);
  int before = 0;
  for (int r0 = 0; r0 < g.n; r0 += 32 * RW) {
    const int nr = xp_bitmap<NT>(lit, s_lo, s_hi, bits, wpre, r0, RW, wsum);
    for (int w = threadIdx.x; w < RW; w += NT) {
      unsigned x = bits[w];
      int k = before + wpre[w];
      while (x) {
        const int v = r0 + 32 * w + __ffs(x) - 1;
        x &= x - 1;
        t.dlist[g.o_list + d0 + k] = v;
        const int c = v / TVb;  // the block that owns v sends its dV here
        t.sends[g.o_push + t.pinfo[g.o_bb + (int64_t)c * (g.B + 1) + b].x + k - dlo[c]] =
            (uint32_t)(v - c * TVb) | ((uint32_t)b << 16);
        k++;
      }
    }
    for (int s = s_lo + threadIdx.x; s < s_hi; s += NT) {
      const int l = __ldg(lit + s);
      const int v = abs(l) - 1 - r0;
      if (v < 0 || v >= 32 * RW) continue;
      const int loc = before + wpre[v >> 5] + __popc(bits[v >> 5] & ((1u << (v & 31)) - 1u));
      t.llit[g.o_slot + s] = (int16_t)(l > 0 ? loc + 1 : -(loc + 1));
    }
    before += nr;
    __syncthreads();  // the next range rebuilds bits / wpre
  }
}

}  // namespace dmm
