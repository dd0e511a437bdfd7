// Cluster form of the integration step: one small formula per thread-block cluster, many
// steps per launch, everything the steps read or write held in the cluster's shared memory.
//
// A small formula's step is bound by latency: on the grid-wide forms it is two grid barriers
// through L2 (1.6-2 us each) and a chain of dependent L2 reads, with a few hundred cycles of
// arithmetic between them.  Here the R blocks of a cluster (1 to 16) split the clauses and the
// variables evenly and exchange through distributed shared memory:
//
//   A  every block holds all n voltages; it evaluates its clauses from shared memory and puts
//      each contribution into a staging area grouped by the block that owns the variable;
//      the area's 16-byte words go to those blocks' buckets; cluster barrier;
//   B  the block sums its variables' contributions in the canonical order (through a table
//      of their bucket places), finds its largest trial index, and sends its dV, trial index
//      and clause counts to every block; cluster barrier;
//   F  every block takes the step decision and applies V <- clamp(V + h dV) to its own copy
//      of the voltages (the accepted candidate, same arithmetic).
//
// Measured (r = 8, 16 blocks, microseconds per step in 256-step launches, against the grid-wide
// forms at 148 blocks): FP32 n = 200 2.8 / 7.1, 1,000 3.8 / 7.2, 2,000 5.0 / 7.4, 4,000 7.3 / 7.7;
// FP64 n = 200 4.2 / 14.4, 1,000 6.3 / 14.8, 2,000 10.1 / 15.4, 3,000 11.6 / 16.0.  What is
// left is latency: about 0.7 us for each of the two exchanges, the rest the dependent chains
// of shared-memory loads and arithmetic of the phases.
//
// Storing each contribution straight to its place in the owner's bucket instead of staging
// it costs about 1.9 cycles per 4-byte remote store and block (measured, 16 blocks), four
// times the staged 16-byte words.
//
// The clause memories, literals and tables stay in shared memory for the launch (the tables
// are made in its prologue); global memory is read when a launch starts and written when it
// ends.  The energy of the last right-hand side is summed from the kept C_m at the end.
//
// The arithmetic is the other forms' (same clause, canonical-sum and candidate code), so the
// states are identical to theirs; an FP64 energy, here the exact sum rounded once, differs from the
// tile forms' plain sums in its last bits.
#pragma once

#include "dmm_cluster.h"
#include "dmm_step.cuh"

namespace dmm {

struct ClusterLayout {
  int v, dv, stage, bk, xs, xl, cp, wdst, vend, off, idx, row, rank, spos, lit, unit, total;
};

// FP64: lists of up to kRankMax entries that a whole warp sums by ranking them, and the warps
// that do so (with 16 bytes of shared memory per entry each).  With few variables per block
// every list goes that way, else the ones past one thread's network.
constexpr int kRankMax = 64;
__host__ __device__ inline bool cluster_rank_all(int tv) { return tv <= 16; }
__host__ __device__ inline int cluster_rank_warps(int tv) {
  return cluster_rank_all(tv) ? kClusterThreads64 / 32 : 4;
}

// Chunks (one per pair of blocks) are padded to whole 16-byte words.
__host__ __device__ inline int cluster_pad(int tsize) { return (16 / tsize - 1) * kClusterMax; }

__host__ __device__ inline ClusterLayout cluster_layout(const ClusterCaps& c, int tsize,
                                                        bool general) {
  ClusterLayout L;
  int o = 0;
  auto take = [&](int bytes) {
    const int at = o;
    o += (bytes + 15) & ~15;
    return at;
  };
  const int pad = cluster_pad(tsize);
  L.v = take(tsize * c.n);
  L.dv = take(tsize * (c.n + 4));
  L.stage = take(tsize * (c.ts + pad + 1));  // one more entry: the padding of the rows
  L.bk = take(tsize * (c.bk + pad + 1));
  L.xs = take(tsize * c.tc);
  L.xl = take(tsize * c.tc);
  L.cp = take(tsize * c.tc);
  L.wdst = take(4 * ((c.ts + pad) * tsize / 16 + 1));
  L.vend = take(4 * (c.tv + 1));
  L.off = take(general ? 4 * (c.tc + 1) : 0);
  L.idx = take(2 * c.bk);
  L.row = take(64 * ((c.tv + 31) & ~31));
  L.rank = take(tsize == 8 ? 16 * kRankMax * cluster_rank_warps(c.tv) : 0);
  L.spos = take(2 * c.ts);
  L.lit = take(2 * c.ts);
  L.unit = take(general ? c.n : 0);
  L.total = o;
  return L;
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Address in the cluster's shared memory of this block's shared address `a` in block `rank`.
__device__ __forceinline__ unsigned cluster_map(unsigned a, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_i(unsigned a, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_h(unsigned a, unsigned short v) {
  asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(a), "h"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster2(unsigned a, int x, int y) {
  asm volatile("st.shared::cluster.v2.s32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void st_cluster4(unsigned a, int x, int y, int z, int w) {
  asm volatile("st.shared::cluster.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y),
               "r"(z), "r"(w)
               : "memory");
}
// Barrier over the cluster with release / acquire of shared memory; a lone block needs only
// its own barrier.  The hardware barrier ends once every thread of the cluster has arrived;
// every thread runs the same number of steps (all take the same decisions).
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync(unsigned R) {
  if (R == 1) {
    __syncthreads();
  } else {
    cluster_arrive();
    cluster_wait();
  }
}

// General clause (k literals) without a per-thread array: the first pass finds the two
// smallest a_j, the second forms the contributions from recomputed a_j.  The same values as
// clause_general.  lit(j): literal; val(l): its voltage; pos(j): place of the contribution;
// put(p, u): contribution.
// Four literals at a time, loaded together: a literal on its own is a chain of two shared-memory
// loads and the arithmetic, twice, and a warp waits for its longest clause.  Step at 6.6 clauses
// of 1 to 8 literals per variable, one at a time / four, us: n = 1,000 FP64 7.6 / 7.2; n = 30,000
// FP32 14.6 / 13.6, FP64 20.8 / 20.4.
template <class T, class Lit, class Val, class Pos, class Put>
__device__ __forceinline__ T clause_any(int k, Lit lit, Val val, T Xs, T Xl,
                                        const ClauseConsts<T>& kc, Pos pos, Put put,
                                        bool& strict_sat) {
  const T one = T(1), half = T(0.5), zero = T(0);
  strict_sat = false;
  if (k == 0) return mul(T(2147483647.0), half);
  if (k == 1) {
    const int l = lit(0);
    const T v = val(l);
    strict_sat = (v > zero && l > 0) || (v < zero && l < 0);
    put(pos(0), zero);
    return zero;
  }
  T mn = T(2147483647.0), mn2 = T(2147483647.0);
  int arg = -1;
  for (int j0 = 0; j0 < k; j0 += 4) {
    int l[4];
    T v[4];
#pragma unroll
    for (int r = 0; r < 4; r++) l[r] = lit(min(j0 + r, k - 1));
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] = val(l[r]);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const bool neg = l[r] < 0, in = j0 + r < k;
      strict_sat |= neg ? v[r] < zero : v[r] > zero;  // past the end: the last literal again
      const T a = sub(one, neg_if(clampv(v[r], -one, one), neg));
      const bool lt = in && a < mn, lt2 = in && a < mn2;
      mn2 = lt ? mn : lt2 ? a : mn2;
      mn = lt ? a : mn;
      arg = lt ? j0 + r : arg;
    }
  }
  const T C = mul(mn, half);
  const T xs = clampv(Xs, zero, one), xl = clampv(Xl, one, kc.xlmax);
  const T xlxs = mul(xl, xs);
  const T rfac = mul(add(one, mul(kc.zeta, xl)), sub(one, xs));
  for (int j0 = 0; j0 < k; j0 += 4) {
    int l[4], p[4];
    T v[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int j = min(j0 + r, k - 1);
      l[r] = lit(j);
      p[r] = pos(j);
    }
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] = val(l[r]);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const bool neg = l[r] < 0;
      const T q = neg ? -one : one;
      const T c = clampv(v[r], -one, one);
      const T a = sub(one, neg_if(c, neg));
      const T others = (j0 + r == arg) ? mn2 : mn;
      const T g = mul(mul(q, others), half);
      const T rr = (C == mul(a, half)) ? mul(sub(q, c), half) : zero;
      if (j0 + r < k) put(p[r], add(mul(xlxs, g), mul(rfac, rr)));
    }
  }
  return C;
}

// Largest / sum over a warp by the integer reduction unit.
__device__ __forceinline__ int redux_max(int v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ int redux_add(int v) { return __reduce_add_sync(0xffffffffu, v); }

// tree_sum (G = 8) of a variable's contributions u[.] through tables in shared memory: the
// first 32 places come from its row (lane l's entries l, l + 8, l + 16, l + 24 as one 8-byte
// word; places past the list lead to a zero, which changes no partial sum), the rest from
// the list idx[0..d).
__device__ __forceinline__ float row_sum(const float* u, const uint2* row, const uint16_t* idx,
                                         int d, int lane) {
  const uint2 q = row[lane];
  float p[4];
  p[0] = add(0.f, u[q.x & 0xffffu]);
  p[1] = add(0.f, u[q.x >> 16]);
  p[2] = add(0.f, u[q.y & 0xffffu]);
  p[3] = add(0.f, u[q.y >> 16]);
  for (int base = 32; base < d; base += 32) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int j = base + lane + 8 * i;
      if (j < d) p[i] = add(p[i], u[idx[j]]);
    }
  }
  float r = add(add(p[0], p[2]), add(p[1], p[3]));
#pragma unroll
  for (int off = 4; off >= 1; off >>= 1) r = add(r, __shfl_xor_sync(0xffffffffu, r, off));
  return r;
}

// Left-to-right sum of the d <= 32 smallest contributions of one thread's row (32 places, eight per
// 16-byte word, words of neighbouring rows side by side; places past the list lead to +inf) after
// sorting them.  One network also for shorter lists: a block runs the code once or twice per step,
// so that warps in two or three networks' straight-line code fetch it instead of sharing it (FP64
// step at n = 1,000: 5.94 us with networks of 16, 24 and 32 chosen by the warp's longest list, 5.81
// with one; n = 10,000: 10.7 and 10.4).
__device__ __forceinline__ double row_net_sum(const double* u, const uint4* row, int d) {
  constexpr int N = 32;
  double a[N];
#pragma unroll
  for (int c = 0; c < N / 8; c++) {
    const uint4 q = row[32 * c];
    a[8 * c + 0] = u[q.x & 0xffffu];
    a[8 * c + 1] = u[q.x >> 16];
    a[8 * c + 2] = u[q.y & 0xffffu];
    a[8 * c + 3] = u[q.y >> 16];
    a[8 * c + 4] = u[q.z & 0xffffu];
    a[8 * c + 5] = u[q.z >> 16];
    a[8 * c + 6] = u[q.w & 0xffffu];
    a[8 * c + 7] = u[q.w >> 16];
  }
  sort_net<N>(a);
  double acc = 0.0;
#pragma unroll
  for (int r = 0; r < N; r++) {
    const double s = __dadd_rn(acc, a[r]);
    acc = r < d ? s : acc;
  }
  return acc;
}

// Left-to-right sum of the sorted u[idx[0..d)], d <= kRankMax, by one warp: each lane counts
// the entries before its own (by value, then place), the values go to their ranks in shared
// memory (buf: 2 kRankMax doubles) and every lane adds them in order.  A few hundred cycles
// where a 64-entry network over the lanes with its shuffled sum takes some 3,000.
template <bool GLOBAL = false>  // where the list is
__device__ __forceinline__ double rank_sum(const double* u, const uint16_t* idx, int d,
                                           double* buf, int lane) {
  const double pinf = inf_val<double>();
  const double x0 = lane < d ? u[list_at<GLOBAL>(idx, lane)] : pinf;
  const double x1 = lane + 32 < d ? u[list_at<GLOBAL>(idx, lane + 32)] : pinf;
  buf[lane] = x0;
  buf[lane + 32] = x1;
  __syncwarp();
  int r0 = 0, r1 = 0;
#pragma unroll 8
  for (int j = 0; j < d; j++) {
    const double y = buf[j];
    r0 += (y < x0) | ((y == x0) & (j < lane));
    r1 += (y < x1) | ((y == x1) & (j < lane + 32));
  }
  double* out = buf + kRankMax;
  if (lane < d) out[r0] = x0;
  if (lane + 32 < d) out[r1] = x1;
  // NaN has no rank: the sum is NaN wherever one takes part
  const bool nan = __any_sync(0xffffffffu, x0 != x0 || x1 != x1);
  __syncwarp();
  double acc = 0.0;
#pragma unroll 8
  for (int j = 0; j < d; j++) acc = __dadd_rn(acc, out[j]);
  __syncwarp();
  return nan ? __longlong_as_double(0x7ff8000000000000ll) : acc;
}

// A sum with its rounding errors carried along (Knuth's two-sum): the energies of the forms that split
// a formula over blocks come out as the exact sum of the C_m rounded once, whatever the split.  As
// plain sums they were up to one unit in the last place off, in one formula's case or another's
// depending on the split; the sums run once per launch.
struct Sum2 {
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double x) {
    const double t = __dadd_rn(s, x), b = __dsub_rn(t, s);
    c = __dadd_rn(c, __dadd_rn(__dsub_rn(s, __dsub_rn(t, b)), __dsub_rn(x, b)));
    s = t;
  }
  __device__ __forceinline__ void add(const Sum2& o) {
    add(o.s);
    c = __dadd_rn(c, o.c);
  }
  __device__ __forceinline__ double value() const { return __dadd_rn(s, c); }
};
// The lanes' sum, in every lane.
__device__ __forceinline__ Sum2 warp_sum2(Sum2 a) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    Sum2 o;
    o.s = __shfl_xor_sync(0xffffffffu, a.s, off);
    o.c = __shfl_xor_sync(0xffffffffu, a.c, off);
    a.add(o);
  }
  return a;
}

struct ClusterShared {
  InstDesc I;
  InstCtrl S;
  int4 x[kClusterMax];      // from every block: unsatisfied, strict failures, trial index
  double e[kClusterMax][2];  // energy partials (block 0, at the end of the launch)
  int base[kClusterMax + 1];  // CSR position where each block's variables start
  int nout[kClusterMax];      // contributions this block sends to each block
  int nin[kClusterMax];       // ... and receives from each
  int rin[kClusterMax];       // where this block's chunk starts in each block's bucket
  int soff[kClusterMax + 1];  // where each block's chunk starts in the staging area
  double red[32][2];
  int cnt[3][32];
  int nlong;
  int32_t longq[kLongQueue];
};

template <class T, bool GENERAL>
__global__ void __launch_bounds__(sizeof(T) == 8 ? kClusterThreads64 : kClusterThreads, 1)
    k_cluster(PackView<T> P, const int32_t* __restrict__ order, int nsteps, ClusterCaps caps) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  __shared__ __align__(16) ClusterShared sc;
  const ClusterLayout LY = cluster_layout(caps, sizeof(T), GENERAL);
  {
    unsigned have;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(have));
    if ((unsigned)LY.total > have) return;  // (the host sizes the launch by the same layout)
  }
  const unsigned R = cluster_size(), rank = cluster_rank();
  T* const sV = reinterpret_cast<T*>(cl_smem + LY.v);
  T* const sdV = reinterpret_cast<T*>(cl_smem + LY.dv);
  T* const stage = reinterpret_cast<T*>(cl_smem + LY.stage);
  // a lone block's staging area is its bucket
  T* const bk = R == 1 ? stage : reinterpret_cast<T*>(cl_smem + LY.bk);
  T* const xs_s = reinterpret_cast<T*>(cl_smem + LY.xs);
  T* const xl_s = reinterpret_cast<T*>(cl_smem + LY.xl);
  T* const cp_s = reinterpret_cast<T*>(cl_smem + LY.cp);
  unsigned* const wdst = reinterpret_cast<unsigned*>(cl_smem + LY.wdst);
  int* const vend_s = reinterpret_cast<int*>(cl_smem + LY.vend);
  int* const off_s = reinterpret_cast<int*>(cl_smem + LY.off);
  uint16_t* const idx_s = reinterpret_cast<uint16_t*>(cl_smem + LY.idx);
  uint16_t* const row_s = reinterpret_cast<uint16_t*>(cl_smem + LY.row);
  double* const rank_s = reinterpret_cast<double*>(cl_smem + LY.rank);
  uint16_t* const spos = reinterpret_cast<uint16_t*>(cl_smem + LY.spos);
  int16_t* const lit_s = reinterpret_cast<int16_t*>(cl_smem + LY.lit);
  int8_t* const unit_s = reinterpret_cast<int8_t*>(cl_smem + LY.unit);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, NT = blockDim.x, W = NT >> 5;
  constexpr int kWord = 16 / (int)sizeof(T);  // values per 16-byte word

  // ---- launch prologue: description, control state, this block's share of the formula
  if (tid == 0) {
    const int ii = order[blockIdx.x / R];
    sc.I = P.inst[ii];
    sc.S = P.ctrl[ii];
    sc.S.pad0 = ii;
  }
  __syncthreads();
  if (sc.S.done != 0) return;  // cluster-uniform, before any exchange
  const InstDesc& I = sc.I;
  const int n = I.n, m = I.m;
  const int TC = cluster_tc(m, R), TV = cluster_tv(n, R);
  const int c0 = min(m, (int)rank * TC), tc = min(m, c0 + TC) - c0;
  const int v0 = min(n, (int)rank * TV), nv = min(n, v0 + TV) - v0;
  const int32_t* const vend = P.vend + I.var0;
  const int32_t* const coff = P.coff + I.cls0;
  const int s0 = GENERAL ? (tc > 0 ? coff[c0] : 0) : 3 * c0;
  const int ns = tc <= 0 ? 0
                 : GENERAL ? (c0 + tc < m ? coff[c0 + tc] : I.nslots) - s0
                           : 3 * tc;
  if (tid <= (int)R) {
    const int v = min(n, tid * TV);
    sc.base[tid] = v > 0 ? vend[v - 1] : 0;
  }
  {
    const T* cur = P.cand + (int64_t)(sc.S.set * kTrials + sc.S.kcur) * P.var_cap + I.var0;
    for (int v = tid; v < n; v += NT) sV[v] = cur[v];
    // (a formula of 3-literal clauses has no unit clauses)
    const int8_t* unit = P.unit + I.var0;
    if (GENERAL)
      for (int v = tid; v < n; v += NT) unit_s[v] = unit[v];
  }
  for (int c = tid; c < tc; c += NT) {
    xs_s[c] = P.Xs[I.cls0 + c0 + c];
    xl_s[c] = P.Xl[I.cls0 + c0 + c];
    cp_s[c] = P.Cp[I.cls0 + c0 + c];
  }
  if constexpr (GENERAL) {
    for (int c = tid; c < tc; c += NT) off_s[c] = coff[c0 + c] - s0;
    if (tid == 0) off_s[tc] = ns;
  }
  if (tid < kClusterMax) sc.nout[tid] = 0;
  if (tid == 0) sc.nlong = 0;
  __syncthreads();
  const int b0 = sc.base[rank];
  for (int i = tid; i <= nv; i += NT) vend_s[i] = (v0 + i > 0 ? vend[v0 + i - 1] : 0) - b0;
  // chunk sizes, exchanged so that every block can place the chunks it receives one after
  // another in its bucket and tell the senders where theirs starts
  const int32_t* const lit = P.lit + I.slot0 + s0;
  for (int s = tid; s < ns; s += NT) {
    const int l = lit[s];
    lit_s[s] = (int16_t)l;
    const int r = (abs(l) - 1) / TV;
    spos[s] = (uint16_t)atomicAdd(&sc.nout[r], 1);
  }
  cluster_sync(R);  // (every block runs; its shared memory may be written)
  auto pad_word = [](int k) { return (k + kWord - 1) / kWord * kWord; };
  if (tid < (int)R)
    st_cluster_i(cluster_map((unsigned)__cvta_generic_to_shared(&sc.nin[rank]), tid), sc.nout[tid]);
  if (tid == 0) {
    int at = 0;
    for (unsigned r = 0; r < R; r++) {
      sc.soff[r] = at;
      at += pad_word(sc.nout[r]);
    }
    sc.soff[R] = at;
  }
  cluster_sync(R);
  if (tid < (int)R) {
    int at = 0;
    for (int r = 0; r < tid; r++) at += pad_word(sc.nin[r]);
    st_cluster_i(cluster_map((unsigned)__cvta_generic_to_shared(&sc.rin[rank]), tid), at);
  }
  cluster_sync(R);
  const int nword = R == 1 ? 0 : sc.soff[R] / kWord;
  {
    const int32_t* upos = P.upos + I.slot0 + s0;
    const unsigned ia = (unsigned)__cvta_generic_to_shared(idx_s);
    for (int s = tid; s < ns; s += NT) {
      const int r = (abs((int)lit_s[s]) - 1) / TV, k = spos[s];
      spos[s] = (uint16_t)(sc.soff[r] + k);
      st_cluster_h(cluster_map(ia + 2u * (unsigned)(upos[s] - sc.base[r]), r),
                   (unsigned short)(sc.rin[r] + k));
    }
    const unsigned bka = (unsigned)__cvta_generic_to_shared(bk);
    for (int q = tid; q < nword; q += NT) {
      int r = 0;
      while (sc.soff[r + 1] <= q * kWord) r++;
      wdst[q] = cluster_map(bka + (unsigned)sizeof(T) * (unsigned)(sc.rin[r] + q * kWord - sc.soff[r]), r);
    }
  }
  const T* const acm = I.has_alpha_cm ? P.alpha_cm + I.cls0 + c0 : nullptr;
  const int ndw = (nv + kWord - 1) / kWord;  // 16-byte words of the block's dV
  const unsigned dva = (unsigned)__cvta_generic_to_shared(sdV);
  const unsigned xa = (unsigned)__cvta_generic_to_shared(&sc.x[0]);
  ClauseConsts<T> kc = make_consts<T>(I, sc.S.h_state);
  bool pending = sc.S.pending != 0;
  int step = sc.S.step, set = sc.S.set, kcur = sc.S.kcur, best_loc = sc.S.best_loc, done = 0;
  int loc = 0, vfail = 0;
  double t = sc.S.t, best_t = sc.S.best_t, solved_t = 0.0, hs = sc.S.h_state;
  const int max_steps = I.max_steps;
  cluster_sync(R);  // the lists are complete
  {
    // rows of the first 32 places of each of the block's variables; the place past the
    // bucket holds the value that padding leads to
    const int pad = R == 1 ? caps.ts + cluster_pad(sizeof(T)) : caps.bk + cluster_pad(sizeof(T));
    if (tid == 0) bk[pad] = sizeof(T) == 4 ? T(0) : inf_val<T>();
    // FP64: the variables that whole warps sum
    if (sizeof(T) == 8)
      for (int i = tid; i < nv; i += NT)
        if (cluster_rank_all(caps.tv) || vend_s[i + 1] - vend_s[i] > 32) {
          const int q = atomicAdd(&sc.nlong, 1);
          if (q < kLongQueue) sc.longq[q] = i;
        }
    const int rows = (nv + 31) & ~31;
    for (int q = tid; q < 32 * rows; q += NT) {
      const int i = q >> 5, j = q & 31;
      int at = pad;
      if (i < nv && vend_s[i] + j < vend_s[i + 1]) at = idx_s[vend_s[i] + j];
      if (sizeof(T) == 4) row_s[32 * i + 4 * (j & 7) + (j >> 3)] = (uint16_t)at;
      else row_s[((i >> 5) * 128 + (j >> 3) * 32 + (i & 31)) * 8 + (j & 7)] = (uint16_t)at;
    }
  }
  __syncthreads();

  for (int s = 0; s < nsteps; s++) {
    // ---- A: clauses
    int unsat = 0, vf = 0;
    for (int c = tid; c < tc; c += NT) {
      T xs = xs_s[c], xl = xl_s[c];
      const T al = acm ? acm[c] : kc.alpha;
      if (pending) {
        advance_memory(xs, xl, cp_s[c], al, kc);
        xs_s[c] = xs;
        xl_s[c] = xl;
      }
      bool ss;
      T C;
      if constexpr (!GENERAL) {
        const int l0 = lit_s[3 * c], l1 = lit_s[3 * c + 1], l2 = lit_s[3 * c + 2];
        const int d0 = spos[3 * c], d1 = spos[3 * c + 1], d2 = spos[3 * c + 2];
        T u0, u1, u2;
        C = clause3(l0, l1, l2, sV[abs(l0) - 1], sV[abs(l1) - 1], sV[abs(l2) - 1], xs, xl, kc,
                    u0, u1, u2, ss);
        stage[d0] = u0;
        stage[d1] = u1;
        stage[d2] = u2;
      } else {
        const int o = off_s[c];
        C = clause_any<T>(
            off_s[c + 1] - o, [&](int j) { return (int)lit_s[o + j]; },
            [&](int l) { return sV[abs(l) - 1]; }, xs, xl, kc,
            [&](int j) { return (int)spos[o + j]; }, [&](int p, T u) { stage[p] = u; }, ss);
      }
      cp_s[c] = C;
      unsat += !(C < T(0.5));
      vf += !ss;
    }
    if (R > 1) {
      __syncthreads();
      const int4* src = reinterpret_cast<const int4*>(stage);
      for (int q = tid; q < nword; q += NT) {
        const int4 v = src[q];
        st_cluster4(wdst[q], v.x, v.y, v.z, v.w);
      }
    }
    if (R > 1) cluster_arrive();
    unsat = redux_add(unsat);  // while the other blocks arrive
    vf = redux_add(vf);
    if (lane == 0) {
      sc.cnt[0][w] = unsat;
      sc.cnt[1][w] = vf;
    }
    if (R > 1) cluster_wait();
    else __syncthreads();

    // ---- B: variables
    int kmax = 0;
    if constexpr (sizeof(T) == 4) {
      constexpr int G = 8;
      const int VPP = NT / G;
      const int grp = tid / G, gl = tid % G;
      for (int vb = 0; vb < nv; vb += VPP) {
        const int i = vb + grp;
        const bool valid = i < nv;
        int a0 = 0, a1 = 0;
        if (valid) {
          a0 = vend_s[i];
          a1 = vend_s[i + 1];
        }
        const T dv = row_sum(reinterpret_cast<const float*>(bk), reinterpret_cast<const uint2*>(row_s) + 8 * min(i, nv - 1),
                             idx_s + a0, a1 - a0, gl);
        bool acc_k = false;
        if (valid) {
          if (gl == 0) sdV[v0 + i] = dv;
          if (gl < kTrials) {  // lane k forms candidate k
            const T V = sV[v0 + i];
            const int8_t un = GENERAL ? unit_s[v0 + i] : 0;
            const T h = gl == 0 ? T(0.125) : gl == 1 ? T(0.0625) : gl == 2 ? T(0.03125)
                                                                           : T(0.015625);
            T c = add(V, mul(h, dv));
            if (un != 0) c = T(un);
            c = clampv(c, T(-1), T(1));
            acc_k = !(fabs((double)c - (double)V) >= 1.0);
          }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, acc_k);
        const unsigned gb = (bal >> (lane & ~(G - 1))) & ((1u << kTrials) - 1u);
        if (valid) kmax = max(kmax, gb ? __ffs(gb) - 1 : kTrials);
      }
    } else {
      // FP64 reference sums: one thread per variable (lists of up to 32); longer lists are queued
      // and summed by whole warps
      const double* ud = reinterpret_cast<const double*>(bk);
      auto finish = [&](int i, T dv) {
        const T V = sV[v0 + i];
        const int8_t un = GENERAL ? unit_s[v0 + i] : 0;
        int kv = kTrials;
#pragma unroll
        for (int k = kTrials - 1; k >= 0; k--) {
          const T h = T(0.125 / (double)(1 << k));
          T c = add(V, mul(h, dv));
          if (un != 0) c = T(un);
          c = clampv(c, T(-1), T(1));
          if (!(fabs((double)c - (double)V) >= 1.0)) kv = k;
        }
        kmax = max(kmax, kv);
        sdV[v0 + i] = dv;
      };
      const bool rank_all = cluster_rank_all(caps.tv);
      const int RW = min(W, cluster_rank_warps(caps.tv)), nq = min(sc.nlong, kLongQueue);
      auto warp_sum = [&](int i) {
        const int e0 = vend_s[i], d = vend_s[i + 1] - e0;
        const double dv =
            d <= kRankMax ? rank_sum(ud, idx_s + e0, d, rank_s + 2 * kRankMax * (W - 1 - w), lane)
                          : sorted_sum<false, uint16_t, false>(ud, idx_s + e0, d, lane);
        if (lane == 0) finish(i, T(dv));
      };
      // the last warps take the lists that whole warps sum, the first ones start with the rest
      if (W - 1 - w < RW)
        for (int q = W - 1 - w; q < nq; q += RW) warp_sum(sc.longq[q]);
      for (int vb = rank_all ? nv : 32 * w; vb < nv; vb += NT) {
        const int i = vb + lane;
        const int d = i < nv ? vend_s[i + 1] - vend_s[i] : 0;
        const bool small = i < nv && d <= 32;
        const int ds = small ? d : 0;
        const uint4* row = reinterpret_cast<const uint4*>(row_s) + 4 * vb + lane;
        const double dv = row_net_sum(ud, row, ds);
        if (small) finish(i, T(dv));
      }
      // lists past the queue's end
      if (W - 1 - w < RW && sc.nlong > kLongQueue)
        for (int i = W - 1 - w; i < nv; i += RW) {
          if (vend_s[i + 1] - vend_s[i] <= 32) continue;
          bool queued = false;
          for (int q = lane; q < nq; q += 32) queued |= sc.longq[q] == i;
          if (!__any_sync(0xffffffffu, queued)) warp_sum(i);
        }
    }
    kmax = redux_max(kmax);
    if (lane == 0) sc.cnt[2][w] = kmax;
    __syncthreads();
    for (int q = tid; q < ndw * (int)(R - 1); q += NT) {  // the block's dV to the others
      const int o = q / ndw, r = o < (int)rank ? o : o + 1, at = v0 / kWord + q - o * ndw;
      const int4 v = reinterpret_cast<const int4*>(sdV)[at];
      st_cluster4(cluster_map(dva + 16u * (unsigned)at, r), v.x, v.y, v.z, v.w);
    }
    if (w == W - 1) {  // the block's trial index to every block
      const int k = redux_max(lane < W ? sc.cnt[2][lane] : 0);
      if (lane < (int)R) st_cluster_i(cluster_map(xa + 16 * rank + 8, lane), k);
    } else if (w == W - 2) {  // ... and its clause counts
      const int lu = redux_add(lane < W ? sc.cnt[0][lane] : 0);
      const int lf = redux_add(lane < W ? sc.cnt[1][lane] : 0);
      if (lane < (int)R) st_cluster2(cluster_map(xa + 16 * rank, lane), lu, lf);
    }
    cluster_sync(R);

    // ---- F: decision (every warp) and the accepted candidate
    int4 x = make_int4(0, 0, 0, 0);
    if (lane < (int)R) x = sc.x[lane];
    kmax = redux_max(x.z);
    loc = redux_add(x.x);
    vfail = redux_add(x.y);
    const int kacc = kmax < kTrials - 1 ? kmax : kTrials - 1;
    hs = kacc == 0 ? 0.125 : kacc == 1 ? 0.0625 : kacc == 2 ? 0.03125 : 0.015625;
    if (loc < best_loc) {
      best_loc = loc;
      best_t = t;
    }
    if (loc == 0 && vfail == 0) {
      done = 1;
      solved_t = t;
    } else if (max_steps > 0 && step + 1 >= max_steps) {
      done = 2;
    }
    if (done == 1) {  // V(step) of this block's variables, for the solution report
      T* sol = P.cand + (int64_t)(set * kTrials + kcur) * P.var_cap + I.var0;
      for (int i = tid; i < nv; i += NT) sol[v0 + i] = sV[v0 + i];
      __syncthreads();
    }
    t = __dadd_rn(t, kmax < kTrials ? hs : 0.0078125);
    step += 1;
    const T h = T(hs);
    for (int v = tid; v < n; v += NT) {
      T c = add(sV[v], mul(h, sdV[v]));
      const int8_t un = GENERAL ? unit_s[v] : 0;
      if (un != 0) c = T(un);
      sV[v] = clampv(c, T(-1), T(1));
    }
    if (done == 1) {
      sc.S.solved_step = step - 1;  // same value from every thread
      sc.S.sol_set = set;
      sc.S.sol_k = kcur;
    }
    set ^= 1;
    kcur = kacc;
    kc.h = h;
    pending = true;
    __syncthreads();
    if (done) break;  // cluster-uniform
  }

  // ---- end of the launch: state, energy of the last right-hand side, control record
  {
    T* cur = P.cand + (int64_t)(set * kTrials + kcur) * P.var_cap + I.var0;
    for (int i = tid; i < nv; i += NT) cur[v0 + i] = sV[v0 + i];
  }
  Sum2 e;
  for (int c = tid; c < tc; c += NT) {
    P.Xs[I.cls0 + c0 + c] = xs_s[c];
    P.Xl[I.cls0 + c0 + c] = xl_s[c];
    const T C = cp_s[c];
    P.Cp[I.cls0 + c0 + c] = C;
    e.add((double)C);
  }
  e = warp_sum2(e);
  if (lane == 0) {
    sc.red[w][0] = e.s;
    sc.red[w][1] = e.c;
  }
  __syncthreads();
  if (w == 0) {
    Sum2 p;
    if (lane < W) {
      p.s = sc.red[lane][0];
      p.c = sc.red[lane][1];
    }
    e = warp_sum2(p);
  }
  if (tid == 0) {
    const unsigned at = cluster_map((unsigned)__cvta_generic_to_shared(&sc.e[0][0]) + 16 * rank, 0);
    st_cluster(at, e.s);
    st_cluster(at + 8, e.c);
  }
  cluster_sync(R);
  if (rank == 0 && tid == 0) {
    Sum2 total;
    for (unsigned r = 0; r < R; r++) {
      Sum2 p;
      p.s = sc.e[r][0];
      p.c = sc.e[r][1];
      total.add(p);
    }
    const double es = total.value();
    InstCtrl* S = P.ctrl + sc.S.pad0;
    S->step = step;
    S->set = set;
    S->kcur = kcur;
    S->pending = pending ? 1 : 0;
    S->best_loc = best_loc;
    S->best_t = best_t;
    S->loc = loc;
    S->vfail = vfail;
    S->t = t;
    S->h_state = hs;
    S->energy = es;
    if (done == 1) {
      S->solved_step = sc.S.solved_step;
      S->solved_t = solved_t;
      S->sol_set = sc.S.sol_set;
      S->sol_k = sc.S.sol_k;
    }
    if (done) {
      S->done = done;
      atomicSub(P.active, 1);
      const int pos = atomicAdd(P.ring_tail, 1);
      P.ring[pos % P.ring_cap] = sc.S.pad0;
    }
    __threadfence();
  }
}

}  // namespace dmm
