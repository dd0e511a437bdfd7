// Device construction of the resident grid form's tables (dmm_grid.cuh), all groups at once.
//
//   k_grid_count  (one block per variable list, i.e. per block of the grid form or clause tile
//                 of the streaming form) rank of every slot within its chunk (clause tile t,
//                 variable tile v), chunk sizes, staging offsets; the list's number of distinct
//                 variables and how many lie below each block's variables.
//   k_grid_rows   (one block per variable tile and per sending block) offsets of the chunks
//                 inside a bucket and inside a send list.
//   k_grid_scan   (one block per group) offsets over tiles, lists and blocks, the limits.
//   k_grid_fill   (as k_grid_count) variable lists, local literals, staging places and
//                 destinations, bucket places in variable-major order, send lists.
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

// Exclusive prefix sums over i < count by the block: put(i, sum of get(0..i-1)); returns the
// total.
template <int NT, class Get, class Put>
__device__ int block_prefix(int count, int* wsum, Get get, Put put) {
  int at = 0;
  for (int i0 = 0; i0 < count; i0 += NT) {
    const int i = i0 + threadIdx.x;
    const int v = i < count ? get(i) : 0;
    int tot;
    const int ex = block_exscan<NT>(v, wsum, &tot);
    if (i < count) put(i, at + ex);
    at += tot;
  }
  return at;
}

__global__ void __launch_bounds__(kGridPrepThreads)
    k_grid_count(const GridGroup* __restrict__ groups, const int32_t* __restrict__ list_group,
                 const int32_t* __restrict__ lit_all, const int32_t* __restrict__ coff, GridTables t,
                 int RW, int kw) {
  constexpr int NT = kGridPrepThreads;
  extern __shared__ __align__(16) int gp_smem[];
  __shared__ int wsum[32];
  const GridGroup g = groups[list_group[blockIdx.x]];
  const int b = blockIdx.x - g.list0, nvt = g.nvt;
  const int32_t* lit = lit_all + g.slot0;
  int* c_s = gp_smem;
  unsigned* bits = reinterpret_cast<unsigned*>(gp_smem + nvt);
  int* wpre = gp_smem + nvt + RW;
  for (int i = 0; i < g.lt; i++) {
    const int ct = b * g.lt + i;
    const int s_lo = grid_slot(g, coff, min(g.m, ct * g.TC)),
              s_hi = grid_slot(g, coff, min(g.m, (ct + 1) * g.TC));
    __syncthreads();
    for (int v = threadIdx.x; v < nvt; v += NT) c_s[v] = 0;
    __syncthreads();
    for (int s = s_lo + threadIdx.x; s < s_hi; s += NT)
      t.spos[g.o_slot + s] = (uint16_t)atomicAdd(&c_s[(abs(__ldg(lit + s)) - 1) / g.TV], 1);
    __syncthreads();
    int at = 0;
    for (int v0 = 0; v0 < nvt; v0 += NT) {
      const int v = v0 + threadIdx.x;
      const int c = v < nvt ? c_s[v] : 0, p = (c + g.pad - 1) / g.pad * g.pad;
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
  const int s_lo = grid_slot(g, coff, min(g.m, b * g.lt * g.TC)),
            s_hi = grid_slot(g, coff, min(g.m, (b + 1) * g.lt * g.TC));
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
  __syncthreads();
  // places: each owning block's variables padded to whole words
  int32_t* dlp = t.dlp + g.o_bb + (int64_t)b * (g.B + 1);
  const int padded = block_prefix<NT>(
      g.B, wsum, [&](int c) { return (dlo[c + 1] - dlo[c] + kw - 1) / kw * kw; },
      [&](int c, int at) { dlp[c] = at; });
  if (threadIdx.x == 0) {
    dlp[g.B] = padded;
    t.dcnt[g.o_blk + b] = padded;
  }
}

constexpr int kGridRowThreads = 256;

// Places of every variable tile's variables by falling list length (a counting sort over
// lengths up to 255; longer ones first, in any order among equals: sums do not depend on it).
__global__ void __launch_bounds__(kGridRowThreads)
    k_grid_order(const GridGroup* __restrict__ groups, const int32_t* __restrict__ vend_all,
                 GridTables t) {
  __shared__ int bin[256], wsum[32];
  const GridGroup& g = groups[blockIdx.y];
  const int vt = blockIdx.x;
  if (vt >= g.nvt) return;
  const int v0 = min(g.n, vt * g.TV), v1 = min(g.n, v0 + g.TV);
  const int32_t* vend = vend_all + g.var0;
  auto key = [&](int v) { return 255 - min(255, vend[v] - (v > 0 ? vend[v - 1] : 0)); };
  bin[threadIdx.x] = 0;
  __syncthreads();
  for (int v = v0 + threadIdx.x; v < v1; v += kGridRowThreads) atomicAdd(&bin[key(v)], 1);
  __syncthreads();
  int tot;
  const int ex = block_exscan<kGridRowThreads>(bin[threadIdx.x], wsum, &tot);
  bin[threadIdx.x] = ex;
  __syncthreads();
  for (int v = v0 + threadIdx.x; v < v1; v += kGridRowThreads) {
    const int p = atomicAdd(&bin[key(v)], 1);
    t.pos[g.o_var + v] = (uint16_t)p;
    t.perm[g.o_var + v0 + p] = (uint16_t)(v - v0);
  }
}

// Places of every clause tile's clauses by falling length, in their own order among equals (so
// that neighbours stay close): counts per thread's range and length, one scan over them.
__global__ void __launch_bounds__(kGridRowThreads)
    k_grid_clauses(const GridGroup* __restrict__ groups, const int32_t* __restrict__ coff,
                   GridTables t) {
  constexpr int K = 16;  // lengths 0 .. 14, and longer ones
  __shared__ int at[K * kGridRowThreads], wsum[32];
  const GridGroup& g = groups[blockIdx.y];
  const int ct = blockIdx.x, tid = threadIdx.x;
  if (ct >= g.nct) return;
  const int c0 = min(g.m, ct * g.TC), n = min(g.m, c0 + g.TC) - c0;
  const int per = (n + kGridRowThreads - 1) / kGridRowThreads;
  const int i0 = min(n, tid * per), i1 = min(n, i0 + per);
  auto key = [&](int i) {
    return K - 1 - min(K - 1, grid_slot(g, coff, c0 + i + 1) - grid_slot(g, coff, c0 + i));
  };
  for (int k = 0; k < K; k++) at[k * kGridRowThreads + tid] = 0;
  for (int i = i0; i < i1; i++) at[key(i) * kGridRowThreads + tid]++;
  __syncthreads();
  int own = 0, tot;
  for (int k = 0; k < K; k++) own += at[tid * K + k];
  int sum = block_exscan<kGridRowThreads>(own, wsum, &tot);
  for (int k = 0; k < K; k++) {
    const int v = at[tid * K + k];
    at[tid * K + k] = sum;
    sum += v;
  }
  __syncthreads();
  for (int i = i0; i < i1; i++)
    t.cord[g.o_cls + c0 + at[key(i) * kGridRowThreads + tid]++] = (uint16_t)i;
}

__global__ void __launch_bounds__(kGridRowThreads)
    k_grid_rows(const GridGroup* __restrict__ groups, GridTables t, int kw) {
  __shared__ int wsum[32];
  const GridGroup& g = groups[blockIdx.y];
  const int nct = g.nct, nvt = g.nvt, r = blockIdx.x;
  if (r < nvt) {
    const int tot = block_prefix<kGridRowThreads>(
        nct, wsum,
        [&](int c) { return (t.cnt[g.o_pair + (int64_t)c * nvt + r] + g.pad - 1) / g.pad * g.pad; },
        [&](int c, int at) { t.bt[g.o_pair + (int64_t)r * nct + c] = at; });
    if (threadIdx.x == 0) t.btot[g.o_vt + r] = tot;
  } else if (r < nvt + g.B) {
    const int b = r - nvt;
    const int tot = block_prefix<kGridRowThreads>(
        g.NL, wsum,
        [&](int l) {
          const int32_t* dlp = t.dlp + g.o_bb + (int64_t)l * (g.B + 1) + b;
          return (dlp[1] - dlp[0]) / kw;
        },
        [&](int l, int at) { t.poff[g.o_bb + (int64_t)l * (g.B + 1) + b] = at; });
    if (threadIdx.x == 0) t.ptot[g.o_blk + b] = tot;
  }
}

__global__ void __launch_bounds__(kGridPrepThreads)
    k_grid_scan(const GridGroup* __restrict__ groups, const int32_t* __restrict__ coff,
                const int32_t* __restrict__ vend, GridTables t, int kw) {
  constexpr int NT = kGridPrepThreads;
  __shared__ int wsum[32], s_bad, s_max[8];
  const GridGroup g = groups[blockIdx.x];
  const int nct = g.nct, nvt = g.nvt, B = g.B, NL = g.NL;
  if (threadIdx.x < 8) s_max[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  block_prefix<NT>(
      NL, wsum, [&](int l) { return (t.dcnt[g.o_blk + l] + 3) & ~3; },
      [&](int l, int at) {
        const int d = t.dcnt[g.o_blk + l];
        t.dinfo[g.o_blk + l] = make_int2(at, d);
        atomicMax(&s_max[1], (d + 3) & ~3);
      });
  const int words = block_prefix<NT>(
      nct, wsum, [&](int c) { return t.st[g.o_ct + c] / kw; },
      [&](int c, int at) {
        t.woff[g.o_ct + c] = at;
        atomicMax(&s_max[2], t.st[g.o_ct + c]);
      });
  const int uxn = block_prefix<NT>(
      nvt, wsum, [&](int v) { return t.btot[g.o_vt + v]; },
      [&](int v, int at) {
        t.boff[g.o_vt + v] = at;
        atomicMax(&s_max[3], t.btot[g.o_vt + v]);
      });
  if (threadIdx.x == 0) {
    t.woff[g.o_ct + nct] = words;
    t.boff[g.o_vt + nvt] = uxn;
    if (s_max[1] > kGridMaxDistinct) s_bad = 1;
    else if (s_max[2] > 65535) s_bad = 2;
    else if (s_max[3] + kw > 65535) s_bad = 3;
  }
  // send words of all blocks, one block after another
  block_prefix<NT>(
      B, wsum, [&](int b) { return t.ptot[g.o_blk + b]; },
      [&](int b, int at) { t.sinfo[g.o_blk + b] = make_int2(at, t.ptot[g.o_blk + b]); });
  __syncthreads();
  for (int b = threadIdx.x; b < B; b += NT) {
    atomicMax(&s_max[4], t.ptot[g.o_blk + b]);
    const int TVb = g.TV * g.kv, v0 = min(g.n, b * TVb), v1 = min(g.n, v0 + TVb);
    atomicMax(&s_max[7], (v1 > 0 ? vend[g.var0 + v1 - 1] : 0) - (v0 > 0 ? vend[g.var0 + v0 - 1] : 0));
    const int TCb = g.TC * g.kc;
    atomicMax(&s_max[5], grid_slot(g, coff, min(g.m, (b + 1) * TCb)) -
                             grid_slot(g, coff, min(g.m, b * TCb)));
    atomicMax(&s_max[6], t.woff[g.o_ct + (b + 1) * g.kc] - t.woff[g.o_ct + b * g.kc]);
  }
  __syncthreads();
  if (threadIdx.x < 8) t.out[kGridOut * blockIdx.x + threadIdx.x] = threadIdx.x == 0 ? s_bad : s_max[threadIdx.x];
}

// ROW64: rows as the FP64 sums read them (32 variables side by side), else as the FP32 sums do.
template <bool ROW64>
__global__ void __launch_bounds__(kGridPrepThreads)
    k_grid_fill(const GridGroup* __restrict__ groups, const int32_t* __restrict__ list_group,
                const int32_t* __restrict__ lit_all, const int32_t* __restrict__ upos_all,
                const int32_t* __restrict__ vend_all, const int32_t* __restrict__ coff, GridTables t,
                int RW, int kw) {
  constexpr int NT = kGridPrepThreads;
  extern __shared__ __align__(16) int gp_smem[];
  __shared__ int wsum[32];
  const int gi = list_group[blockIdx.x];
  const GridGroup g = groups[gi];
  if (t.out[kGridOut * gi] != 0) return;  // a limit failed: the tables are not used
  const int b = blockIdx.x - g.list0, nvt = g.nvt, nct = g.nct;
  const int32_t* lit = lit_all + g.slot0;
  const int32_t* upos = upos_all + g.slot0;
  const int32_t* vend = vend_all + g.var0;
  int* s_sb = gp_smem;  // [nvt] staging offset, then the bucket offset of this tile's chunk
  unsigned* bits = reinterpret_cast<unsigned*>(gp_smem + nvt);
  int* wpre = gp_smem + nvt + RW;
  for (int i = 0; i < g.lt; i++) {
    const int ct = b * g.lt + i;
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
      const int vi = t.pos ? t.pos[g.o_var + v] : v - vt * g.TV;
      uint16_t* row = t.rows + g.o_row + (int64_t)vt * g.TVr * 32;
      if (j < 32)
        row[ROW64 ? ((vi >> 5) * 128 + (j >> 3) * 32 + (vi & 31)) * 8 + (j & 7)
                  : 32 * vi + 8 * (j & 3) + (j >> 2)] = at;
    }
    // destinations of the staging area's words
    const int w0 = t.woff[g.o_ct + ct];
    for (int v = threadIdx.x >> 5; v < nvt; v += NT / 32) {
      const int nw = (t.cnt[g.o_pair + (int64_t)ct * nvt + v] + g.pad - 1) / g.pad * g.pad / kw;
      const int d0 = (t.boff[g.o_vt + v] + t.bt[g.o_pair + (int64_t)v * nct + ct]) / kw;
      for (int q = threadIdx.x & 31; q < nw; q += 32)
        t.wdst[g.o_word + w0 + s_sb[v] / kw + q] = (uint32_t)(d0 + q);
    }
  }
  __syncthreads();
  // the block's variable list (ascending), local literals and entries of the send lists,
  // range by range
  const int s_lo = grid_slot(g, coff, min(g.m, b * g.lt * g.TC)),
            s_hi = grid_slot(g, coff, min(g.m, (b + 1) * g.lt * g.TC));
  const int TVb = g.TV * g.kv, d0 = t.dinfo[g.o_blk + b].x;
  const int32_t* dlo = t.dlo + g.o_bb + (int64_t)b * (g.B + 1);
  const int32_t* dlp = t.dlp + g.o_bb + (int64_t)b * (g.B + 1);
  const int32_t* poff = t.poff + g.o_bb + (int64_t)b * (g.B + 1);
  // the words of the owning blocks' chunks
  for (int c = threadIdx.x >> 5; c < g.B; c += NT / 32) {
    const int nw = (dlp[c + 1] - dlp[c]) / kw;
    const int64_t w0 = g.o_push + t.sinfo[g.o_blk + c].x + poff[c];
    for (int q = threadIdx.x & 31; q < nw; q += 32)
      t.sdst[w0 + q] = (uint32_t)((d0 + dlp[c]) / kw + q);
    if ((threadIdx.x & 31) == 0)
      for (int k = dlp[c] + dlo[c + 1] - dlo[c]; k < dlp[c + 1]; k++) {  // padding
        t.dlist[g.o_list + d0 + k] = -1;
        t.ids[w0 * kw + k - dlp[c]] = 0;
      }
  }
  int before = 0;
  for (int r0 = 0; r0 < g.n; r0 += 32 * RW) {
    const int nr = xp_bitmap<NT>(lit, s_lo, s_hi, bits, wpre, r0, RW, wsum);
    for (int w = threadIdx.x; w < RW; w += NT) {
      unsigned x = bits[w];
      int k = before + wpre[w];
      while (x) {
        const int v = r0 + 32 * w + __ffs(x) - 1;
        x &= x - 1;
        const int c = v / TVb, at = dlp[c] + k - dlo[c];  // the block that owns v sends it here
        t.dlist[g.o_list + d0 + at] = v;
        t.ids[(g.o_push + t.sinfo[g.o_blk + c].x + poff[c]) * kw + at - dlp[c]] =
            (uint16_t)(t.pos ? v / g.TV * g.TV - c * TVb + t.pos[g.o_var + v] : v - c * TVb);
        k++;
      }
    }
    for (int s = s_lo + threadIdx.x; s < s_hi; s += NT) {
      const int l = __ldg(lit + s);
      const int v = abs(l) - 1 - r0;
      if (v < 0 || v >= 32 * RW) continue;
      const int k = before + wpre[v >> 5] + __popc(bits[v >> 5] & ((1u << (v & 31)) - 1u));
      const int c = (abs(l) - 1) / TVb, loc = dlp[c] + k - dlo[c];
      t.llit[g.o_slot + s] = (int16_t)(l > 0 ? loc + 1 : -(loc + 1));
    }
    before += nr;
    __syncthreads();  // the next range rebuilds bits / wpre
  }
}

}  // namespace dmm
