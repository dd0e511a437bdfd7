// Resident grid form of the integration step: one cooperative launch runs many steps of one or
// several formulas, each on its own group of blocks (one block per SM), with the voltages a
// block's clauses read kept in its shared memory from step to step.
//
// Per step a block
//   A  evaluates its clauses tile by tile through 16-bit block-local literals, each
//      contribution going to a staging area grouped by destination variable tile, whose
//      16-byte words it then stores to those tiles' buckets in global memory (L2);
//   B  loads the buckets of its variable tiles into shared memory (each is contiguous), sums
//      every variable's contributions in the canonical order through a table of bucket
//      places, and sends dV to the inboxes of the blocks whose clauses contain the variable
//      (contiguous chunks on both sides);
//   F  once every block has reported its largest trial index, takes the step's decision and
//      applies V <- clamp(V + h dV) to its copy of the voltages, dV coming from its inbox in
//      list order.
//
// Sending dV, which is known before the step's decision, instead of gathering the accepted
// candidate after it takes the scattered 4-byte reads of all voltages and the four candidates
// out of the step; the places table takes out the shared-memory scatter of the bucket.
//
// No grid barriers: a bucket or inbox entry is its own flag.  Unset entries hold a signalling
// NaN, which no arithmetic operation returns; the reader polls the words it needs until every
// entry is set and sets them back to unset at once.  A barrier would add, to the one trip of
// the data through L2, a wait for the acknowledgement of all stores, the arrival's trip and
// the polls' (1.7 us in all, twice per step).  Buckets and inboxes exist twice, for steps of
// even and odd number.  A writer of step s + 2 cannot overtake the reader that unsets the same
// entry in step s: it has seen the decision of step s + 1, to which the reader's block reported
// after a fence that follows the unsetting.  The decision itself is one word of byte-wide
// counters (blocks reported, blocks with trial index >= 1 .. 4, blocks with unsatisfied
// clauses), so it needs no second read.  Every poll is bounded.
//
// RES 1: the tables of the variable phase live in shared memory for the launch; RES 2: so do
// the clause memories and all other tables (formulas up to about 40,000 variables in FP32).
//
// FP64: the variables of a tile are kept by falling list length, the order being made with the
// tables.  The lists that whole warps sum come first and need no queue, and a warp of the others
// holds lists of like length; every per-variable array of the block is in that order, the
// global ones are not.  Step with variables in their own order / by length, us: n = 5,000 8.9 /
// 8.4, 10,000 10.8 / 10.2, 30,000 16.1 / 15.6, 50,000 23.0 / 21.8.  FP32 sums take four lanes a list and gain nothing.
// Splitting the network over two or four lanes was slower (n = 10,000 10.6 and 11.5): the
// exchanges across lanes cost more than the shorter code saves.
//
// Clauses of other lengths than three: a block goes through a tile's clauses by falling length
// (a table, with equal ones in their own order), so that a warp's clauses take alike many
// iterations, and the clauses of three literals among them take the unrolled path.  The clause
// phase is bound by instructions there: at 6.6 clauses of 1 to 8 literals per variable, in their
// own order / by length, us: n = 30,000 FP32 13.6 / 11.7, FP64 20.4 / 17.0 (of which the clause
// phase 8.8 / 5.4); n = 10,000 FP32 8.0 / 7.6, FP64 11.8 / 11.2; n = 60,000, where the clause
// memories are read from L2 in that order, FP32 25.9 / 22.1, FP64 38.4 / 38.3.
//
// Every clause value and per-variable sum is computed from the same operands in the same order
// as in the other forms: the states are identical.
#pragma once

#include "dmm_cluster.cuh"
#include "dmm_grid.h"
#include "dmm_xpose.cuh"

namespace dmm {

inline GridLayout grid_layout(const GridCaps& c, int tsize, bool general,
                                                  int resident) {
  GridLayout L;
  int o = 0;
  auto take = [&](int bytes) {
    const int at = o;
    o += (bytes + 15) & ~15;
    return at;
  };
  L.sv = take(tsize * c.dl);
  // staging area (A) / bucket behind one padding word (B)
  L.raw = take((tsize * c.st > 16 + tsize * c.bk ? tsize * c.st : 16 + tsize * c.bk));
  L.cur = take(tsize * c.tv);
  L.dv = take(tsize * c.tv);
  L.vend = take(8 * c.tv);
  L.unit = take(general ? c.tv : 0);
  L.rank = take(tsize == 8 ? 16 * kRankMax * (kGridThreads64 / 32) : 0);
  L.xs = L.xl = L.cp = L.lit = L.spos = L.off = L.ord = L.wdst = L.row = L.csr = L.snd = 0;
  if (resident >= 1) {
    L.row = take(2 * c.row);
    L.csr = take(2 * c.csr);
  }
  if (resident >= 2) {
    L.xs = take(tsize * c.tc);
    L.xl = take(tsize * c.tc);
    L.cp = take(tsize * c.tc);
    L.lit = take(2 * c.ts);
    L.spos = take(2 * c.ts);
    L.off = take(general ? 4 * (c.tc + 1) : 0);
    L.ord = take(general ? 2 * c.tc : 0);
    L.wdst = take(4 * c.wd);
    L.snd = take((4 + 2 * (16 / tsize)) * c.snd);
  }
  L.total = o;
  return L;
}

// Counters of a group (zero before a launch; the last block of the group to leave zeroes
// them).  The decision words and counts of a step are in slot step mod 4 of the launch: slot
// s + 2 is zeroed in step s, when every block has taken the decision of step s - 2.
struct GridStepSlot {
  unsigned long long word;  // bytes: blocks reported; with trial index >= 1, 2, 3, 4; with
                            // unsatisfied clauses
  int loc, vfail;           // unsatisfied clauses, strict-sign failures
};
struct alignas(128) GridSync {
  GridStepSlot slot[4];
  unsigned int exits;
  int best_loc, loc, vfail;  // of block 0, for the control record
  double best_t;
  int pad[26];
};

// The value of an exchange entry that is not set: a signalling NaN.
template <class B>
struct Unset;
template <>
struct Unset<unsigned int> {
  __host__ __device__ static unsigned int bits() { return 0x7fa0dbadu; }
};
template <>
struct Unset<unsigned long long> {
  __host__ __device__ static unsigned long long bits() { return 0x7ff4dbad7fa0dbadull; }
};

// Exchange accesses (ordered among themselves as volatile; each entry is its own flag, so they
// need no order against other memory and the loads around them may be batched).  The memory
// model treats a vector access as one access per element, so the elements are whole entries:
// with 4-byte elements the two halves of an FP64 entry could be seen one without the other.
template <class T>
__device__ __forceinline__ int4 ld_word(const int4* p) {
  int4 v;
  if constexpr (sizeof(T) == 4) {
    asm volatile("ld.relaxed.gpu.global.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
  } else {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p));
    v = make_int4((int)a, (int)(a >> 32), (int)b, (int)(b >> 32));
  }
  return v;
}
// The entries of an FP64 word.
__host__ __device__ __forceinline__ unsigned long long entry64(int lo, int hi) {
  return (unsigned int)lo | (unsigned long long)(unsigned int)hi << 32;
}
template <class T>
__device__ __forceinline__ void st_word(int4* p, int4 v) {
  if constexpr (sizeof(T) == 4)
    asm volatile("st.relaxed.gpu.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x),
                 "r"(v.y), "r"(v.z), "r"(v.w));
  else
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(entry64(v.x, v.y)),
                 "l"(entry64(v.z, v.w)));
}
// Whether all entries of a word are set.
template <class T>
__device__ __forceinline__ bool word_set(const int4& v) {
  if constexpr (sizeof(T) == 4) {
    const int u = (int)Unset<unsigned int>::bits();
    return v.x != u && v.y != u && v.z != u && v.w != u;
  } else {
    const unsigned long long u = Unset<unsigned long long>::bits();
    return entry64(v.x, v.y) != u && entry64(v.z, v.w) != u;
  }
}
template <class T>
__device__ __forceinline__ int4 unset_word() {
  if constexpr (sizeof(T) == 4) {
    const int u = (int)Unset<unsigned int>::bits();
    return make_int4(u, u, u, u);
  } else {
    const int lo = (int)(unsigned int)Unset<unsigned long long>::bits();
    const int hi = (int)(Unset<unsigned long long>::bits() >> 32);
    return make_int4(lo, hi, lo, hi);
  }
}

constexpr int kGridPollLimit = 1 << 21;  // polls of an exchange word (about a second)

// Takes up to N words of p[q0 + r step], r < N (those below n): polls all of them together until
// their entries are set, then unsets them.  Clears ok when the limit runs out (and does not
// poll on once it is clear).
template <class T, int N>
__device__ __forceinline__ void take_words(int4* p, int q0, int step, int n, int4 (&v)[N], bool& ok) {
  int it = ok ? 0 : kGridPollLimit;
  for (;;) {
    bool set = true;
#pragma unroll
    for (int r = 0; r < N; r++)
      if (q0 + r * step < n) v[r] = ld_word<T>(p + q0 + r * step);
#pragma unroll
    for (int r = 0; r < N; r++)
      if (q0 + r * step < n) set = set && word_set<T>(v[r]);
    if (set) break;
    if (++it >= kGridPollLimit) {
      ok = false;
      break;
    }
  }
#pragma unroll
  for (int r = 0; r < N; r++)
    if (q0 + r * step < n) st_word<T>(p + q0 + r * step, unset_word<T>());
}

// A block's copy of the control state of its formula.
struct GridCtrl {
  int done, step, set, kcur, pending, best_loc, sol_k, loc, vfail;
  double h, t, t_rhs, best_t, solved_t;
};

// Block-uniform pointers and counts, kept in shared memory to spare registers (clause c of the
// block, slot s from the block's first slot, ...).
template <class T>
struct GridPtrs {
  T *ux, *inbox, *Xs, *Xl, *Cp, *cand;
  const T* acm;
  const int32_t *woff, *boff, *coff;
  const int16_t* llit;
  const uint16_t *spos, *rows, *idx, *ord;
  const uint16_t* ids;
  const uint32_t *wdst, *sdst;
  int in_place, dcnt, nsend;
};

// tree_sum (G = 4) of a variable's contributions u[.]: the first 32 places come from its row
// (lane l's entries l, l + 4, ... as one 16-byte word; padding leads to u[0] = 0, which
// changes no partial sum), the rest from the list idx[0..d).
template <bool GLOBAL>
__device__ __forceinline__ float row_sum4(const float* u, uint4 q, const uint16_t* idx, int d,
                                          int lane) {
  float p[8];
  p[0] = add(0.f, u[q.x & 0xffffu]);
  p[1] = add(0.f, u[q.x >> 16]);
  p[2] = add(0.f, u[q.y & 0xffffu]);
  p[3] = add(0.f, u[q.y >> 16]);
  p[4] = add(0.f, u[q.z & 0xffffu]);
  p[5] = add(0.f, u[q.z >> 16]);
  p[6] = add(0.f, u[q.w & 0xffffu]);
  p[7] = add(0.f, u[q.w >> 16]);
  for (int base = 32; base < d; base += 32) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int j = base + lane + 4 * i;
      if (j < d) p[i] = add(p[i], u[list_at<GLOBAL>(idx, j)]);
    }
  }
  float r = add(add(add(p[0], p[4]), add(p[2], p[6])), add(add(p[1], p[5]), add(p[3], p[7])));
#pragma unroll
  for (int off = 2; off >= 1; off >>= 1) r = add(r, __shfl_xor_sync(0xffffffffu, r, off));
  return r;
}

template <class T, bool GENERAL, int RES>
__global__ void __launch_bounds__(sizeof(T) == 8 ? kGridThreads64 : kGridThreads, 1)
    k_grid(PackView<T> P, GridTables tb, const GridGroup* __restrict__ groups,
           const int32_t* __restrict__ blk_group, GridLayout LY, int nsteps, GridSync* sync_all,
           double2* __restrict__ epart, int* err) {
  constexpr int NT = sizeof(T) == 8 ? kGridThreads64 : kGridThreads;
  constexpr int W = NT / 32;
  constexpr int kw = 16 / (int)sizeof(T);  // values per 16-byte word
  extern __shared__ __align__(16) unsigned char gr_smem[];
  __shared__ InstDesc I;
  __shared__ GridGroup g;
  __shared__ GridCtrl lc;
  __shared__ GridPtrs<T> sp;
  __shared__ ClauseConsts<T> s_kc;
  __shared__ int cnt[3][W];
  __shared__ double red[W][2];
  __shared__ int s_ok, s_last, s_unsat, s_next;
  __shared__ int s_nq[kGridMaxTiles];  // lists of each variable tile that whole warps sum
  {
    unsigned have;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(have));
    if ((unsigned)LY.total > have) return;  // (the host sizes the launch by the same layout)
  }
  T* const sV = reinterpret_cast<T*>(gr_smem + LY.sv);
  T* const stage = reinterpret_cast<T*>(gr_smem + LY.raw);
  T* const raw = stage;
  T* const s_cur = reinterpret_cast<T*>(gr_smem + LY.cur);
  T* const s_dv = reinterpret_cast<T*>(gr_smem + LY.dv);
  int2* const s_list = reinterpret_cast<int2*>(gr_smem + LY.vend);  // start and length of each list
  int8_t* const s_unit = reinterpret_cast<int8_t*>(gr_smem + LY.unit);
  double* const s_rank = reinterpret_cast<double*>(gr_smem + LY.rank);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

  trace_launch(P, 0);
  // ---- launch prologue
  if (tid == 0) {
    g = groups[blk_group[blockIdx.x]];
    I = P.inst[g.inst];
    const volatile InstCtrl* S = P.ctrl + g.inst;
    lc.done = S->done;
    // a wait of the launch before gave up (the host has not seen it yet): the exchanges hold
    // entries of the abandoned step, so none is taken
    if (*reinterpret_cast<volatile int*>(err) != 0) lc.done = -1;
    lc.step = S->step;
    lc.set = S->set;
    lc.kcur = S->kcur;
    lc.pending = S->pending;
    lc.best_loc = S->best_loc;
    lc.h = S->h_state;
    lc.t = S->t;
    lc.best_t = S->best_t;
    s_kc = make_consts<T>(I, lc.h);
  }
  __syncthreads();
  const int b = blockIdx.x - g.blk0, B = g.B;
  GridSync* const gs = sync_all + blk_group[blockIdx.x];
  const int m = I.m;
  const int TCb = g.TC * g.kc, TVb = g.TV * g.kv;
  const int c0 = min(m, b * TCb), c1 = min(m, c0 + TCb);
  const int v0 = min(I.n, b * TVb), nv = min(I.n, v0 + TVb) - v0;
  const int s0 = grid_slot(g, P.coff, c0);
  const int32_t* const vend = P.vend + I.var0;
  const int vend0 = v0 > 0 ? vend[v0 - 1] : 0;
  if (tid == 0) {
    const int2 di = tb.dinfo[g.o_blk + b];
    const int2 si = tb.sinfo[g.o_blk + b];
    const int32_t* const woff = tb.woff + g.o_ct + b * g.kc;
    sp.ux = static_cast<T*>(tb.ux) + g.o_ux;
    sp.inbox = static_cast<T*>(tb.inbox) + g.o_list;
    sp.in_place = di.x;
    sp.dcnt = di.y;
    sp.nsend = si.y;
    sp.woff = woff;
    sp.boff = tb.boff + g.o_vt + b * g.kv;
    sp.llit = tb.llit + g.o_slot + s0;
    sp.spos = tb.spos + g.o_slot + s0;
    sp.wdst = tb.wdst + g.o_word + woff[0];
    sp.rows = tb.rows + g.o_row + (int64_t)b * g.kv * g.TVr * 32;
    sp.sdst = tb.sdst + g.o_push + si.x;
    sp.ids = tb.ids + (g.o_push + si.x) * kw;
    sp.idx = tb.idx + g.o_slot + vend0;  // from the block's first CSR entry
    sp.Xs = P.Xs + I.cls0 + c0;
    sp.Xl = P.Xl + I.cls0 + c0;
    sp.Cp = P.Cp + I.cls0 + c0;
    sp.acm = I.has_alpha_cm ? P.alpha_cm + I.cls0 + c0 : nullptr;
    sp.coff = P.coff + I.cls0 + c0;
    sp.ord = tb.cord + g.o_cls + c0;
    sp.cand = P.cand + I.var0 + v0;
  }
  __syncthreads();
  int32_t* const off_s = reinterpret_cast<int32_t*>(gr_smem + LY.off);
  // variable (from the block's first) at place i of the block: FP64 tiles keep their variables
  // by falling list length, so that a warp's lists have similar lengths
  auto var_at = [&](int i) {
    if constexpr (sizeof(T) == 4) {
      return i;
    } else {
      const int t0 = i / g.TV * g.TV;
      return t0 + (int)tb.perm[g.o_var + v0 + i];
    }
  };
  if (lc.done == 0) {
    const T* V0 = P.cand + (int64_t)(lc.set * kTrials + lc.kcur) * P.var_cap + I.var0;
    const int32_t* dl = tb.dlist + g.o_list + sp.in_place;
    const int dcnt = sp.dcnt;
    for (int k = tid; k < dcnt; k += NT) sV[k] = dl[k] >= 0 ? V0[dl[k]] : T(0);
    for (int i = tid; i < nv; i += NT) {
      const int v = v0 + var_at(i);
      s_cur[i] = V0[v];
      const int e0 = v > 0 ? vend[v - 1] : 0;
      s_list[i] = make_int2(e0 - vend0, vend[v] - e0);
      if (GENERAL) s_unit[i] = P.unit[I.var0 + v];
    }
    // no entry of the areas may look unset (the padding of chunks is sent too)
    for (int q = tid; q < (LY.cur - LY.raw) / 16; q += NT)
      reinterpret_cast<int4*>(gr_smem + LY.raw)[q] = make_int4(0, 0, 0, 0);
    if constexpr (sizeof(T) == 8) {
      // how many of a tile's first lists whole warps sum: the ones past one thread's network
      for (int j = tid; j < kGridMaxTiles; j += NT) s_nq[j] = 0;
      __syncthreads();
      for (int i = tid; i < nv; i += NT) {
        const int j = i / g.TV;
        const bool last = i + 1 == nv || (i + 1) % g.TV == 0;
        if (s_list[i].y > 32 && (last || s_list[i + 1].y <= 32)) s_nq[j] = i + 1 - j * g.TV;
      }
    }
    if constexpr (RES >= 1) {
      auto bring = [&](int at, const auto* src, int count) {
        using E = typename std::remove_cv<typename std::remove_reference<decltype(*src)>::type>::type;
        E* d = reinterpret_cast<E*>(gr_smem + at);
        for (int i = tid; i < count; i += NT) d[i] = src[i];
      };
      bring(LY.row, sp.rows, g.kv * g.TVr * 32);
      bring(LY.csr, sp.idx, nv > 0 ? vend[v0 + nv - 1] - vend0 : 0);
      if constexpr (RES == 2) {
        const int ns = grid_slot(g, P.coff, c1) - s0;
        bring(LY.xs, sp.Xs, c1 - c0);
        bring(LY.xl, sp.Xl, c1 - c0);
        bring(LY.cp, sp.Cp, c1 - c0);
        bring(LY.lit, sp.llit, ns);
        bring(LY.spos, sp.spos, ns);
        bring(LY.wdst, sp.wdst, sp.woff[g.kc] - sp.woff[0]);
        bring(LY.snd, sp.sdst, sp.nsend);
        bring(LY.snd + 4 * sp.nsend, sp.ids, kw * sp.nsend);
        if (GENERAL) {
          for (int c = tid; c <= c1 - c0; c += NT) off_s[c] = grid_slot(g, P.coff, c0 + c) - s0;
          bring(LY.ord, sp.ord, c1 - c0);
        }
      }
    }
  }
  __syncthreads();

  int steps_run = 0, best_loc = lc.best_loc, loc = 0, vfail = 0;  // (counts: block 0's last warp)
  double best_t = lc.best_t;
  bool gave_up = false;
  for (int s = 0; s < nsteps; s++) {
    if (lc.done != 0) break;  // group-uniform: every block applies the same decisions
    trace_stamp(P, s, 0);
    GridStepSlot* const slot = &gs->slot[s & 3];
    const int set = lc.set, kcur = lc.kcur;
    const bool pending = lc.pending != 0;
    const ClauseConsts<T>& kc = s_kc;
    if (P.trace) {
      trace_stamp(P, s, 1);
      trace_stamp(P, s, 2);
    }

    // ---- A: the block's clause tiles
    const int16_t* const llit = RES == 2 ? reinterpret_cast<const int16_t*>(gr_smem + LY.lit) : sp.llit;
    const uint16_t* const spos = RES == 2 ? reinterpret_cast<const uint16_t*>(gr_smem + LY.spos) : sp.spos;
    T* const Xs = RES == 2 ? reinterpret_cast<T*>(gr_smem + LY.xs) : sp.Xs;
    T* const Xl = RES == 2 ? reinterpret_cast<T*>(gr_smem + LY.xl) : sp.Xl;
    T* const Cp = RES == 2 ? reinterpret_cast<T*>(gr_smem + LY.cp) : sp.Cp;
    const T* const acm = sp.acm;
    int unsat = 0, vf = 0;
    auto one = [&](int l0, int l1, int l2, int p0, int p1, int p2, T& xs, T& xl, T cp, T al) -> T {
      if (pending) advance_memory(xs, xl, cp, al, kc);
      bool ss;
      T u0, u1, u2;
      const T C = clause3(l0, l1, l2, sV[abs(l0) - 1], sV[abs(l1) - 1], sV[abs(l2) - 1], xs, xl,
                          kc, u0, u1, u2, ss);
      stage[p0] = u0;
      stage[p1] = u1;
      stage[p2] = u2;
      unsat += !(C < T(0.5));
      vf += !ss;
      return C;
    };
    for (int i = 0; i < g.kc; i++) {
      const int t0 = min(c1 - c0, i * g.TC), t1 = min(c1 - c0, t0 + g.TC);
      if constexpr (GENERAL) {
        // longest clauses first
        const uint16_t* const ord =
            RES == 2 ? reinterpret_cast<const uint16_t*>(gr_smem + LY.ord) : sp.ord;
        for (int q = t0 + tid; q < t1; q += NT) {
          const int c = t0 + ord[q];
          int o, o1;
          if constexpr (RES == 2) {
            o = off_s[c];
            o1 = off_s[c + 1];
          } else {
            o = g.k3 ? 3 * c : __ldg(sp.coff + c) - s0;
            o1 = g.k3 ? 3 * c + 3 : c0 + c + 1 < m ? __ldg(sp.coff + c + 1) - s0 : g.L - s0;
          }
          T xs = Xs[c], xl = Xl[c], C;
          const T al = acm ? acm[c] : kc.alpha;
          if (pending) advance_memory(xs, xl, Cp[c], al, kc);
          bool ss, three = o1 - o == 3;
          int l0 = 0, l1 = 0, l2 = 0;
          T V0 = T(0), V1 = T(0), V2 = T(0);
          if (three) {
            l0 = llit[o];
            l1 = llit[o + 1];
            l2 = llit[o + 2];
            V0 = sV[abs(l0) - 1];
            V1 = sV[abs(l1) - 1];
            V2 = sV[abs(l2) - 1];
            // a NaN is passed over by the general clause's minimum, not by clause3's
            const T t = add(add(V0, V1), V2);
            three = t == t;
          }
          if (three) {
            T u0, u1, u2;
            C = clause3(l0, l1, l2, V0, V1, V2, xs, xl, kc, u0, u1, u2, ss);
            stage[spos[o]] = u0;
            stage[spos[o + 1]] = u1;
            stage[spos[o + 2]] = u2;
          } else {
            C = clause_any<T>(
                o1 - o, [&](int j) { return (int)llit[o + j]; },
                [&](int l) { return sV[abs(l) - 1]; }, xs, xl, kc,
                [&](int j) { return (int)spos[o + j]; }, [&](int p, T u) { stage[p] = u; }, ss);
          }
          unsat += !(C < T(0.5));
          vf += !ss;
          Xs[c] = xs;
          Xl[c] = xl;
          Cp[c] = C;
        }
      } else if constexpr (RES == 2) {
        for (int c = t0 + tid; c < t1; c += NT) {
          T xs = Xs[c], xl = Xl[c];
          const T al = acm ? acm[c] : kc.alpha;
          Cp[c] = one(llit[3 * c], llit[3 * c + 1], llit[3 * c + 2], spos[3 * c], spos[3 * c + 1],
                        spos[3 * c + 2], xs, xl, Cp[c], al);
          Xs[c] = xs;
          Xl[c] = xl;
        }
      } else {
        // pairs of clauses: 4-byte words of literals and places, 2-wide loads of the memories
        // (the tile starts at a multiple of 4 clauses of a 32-aligned range)
        using T2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
        struct Pair {
          int lw[3];
          unsigned qw[3];
          T2 xs, xl, cp;
        };
        auto load_pair = [&](Pair& p, int c) {
          const int* L3 = reinterpret_cast<const int*>(llit + 3 * c);
          const unsigned* Q3 = reinterpret_cast<const unsigned*>(spos + 3 * c);
#pragma unroll
          for (int r = 0; r < 3; r++) {
            p.lw[r] = __ldg(L3 + r);
            p.qw[r] = __ldg(Q3 + r);
          }
          p.xs = *reinterpret_cast<const T2*>(Xs + c);
          p.xl = *reinterpret_cast<const T2*>(Xl + c);
          p.cp.x = p.cp.y = T(0);
          if (pending) p.cp = *reinterpret_cast<const T2*>(Cp + c);
        };
        auto do_pair = [&](const Pair& p, int c) {
          auto lit = [&](int k) {
            return (k & 1) ? (p.lw[k >> 1] >> 16) : (int)(short)(p.lw[k >> 1] & 0xffff);
          };
          auto pos = [&](int k) {
            return (int)((k & 1) ? (p.qw[k >> 1] >> 16) : (p.qw[k >> 1] & 0xffffu));
          };
          T2 al2;
          al2.x = al2.y = kc.alpha;
          if (acm) al2 = *reinterpret_cast<const T2*>(acm + c);
          T xs[2] = {p.xs.x, p.xs.y}, xl[2] = {p.xl.x, p.xl.y}, cc[2];
          cc[0] = one(lit(0), lit(1), lit(2), pos(0), pos(1), pos(2), xs[0], xl[0], p.cp.x, al2.x);
          cc[1] = one(lit(3), lit(4), lit(5), pos(3), pos(4), pos(5), xs[1], xl[1], p.cp.y, al2.y);
          T2 o;
          o.x = xs[0];
          o.y = xs[1];
          *reinterpret_cast<T2*>(Xs + c) = o;
          o.x = xl[0];
          o.y = xl[1];
          *reinterpret_cast<T2*>(Xl + c) = o;
          o.x = cc[0];
          o.y = cc[1];
          *reinterpret_cast<T2*>(Cp + c) = o;
        };
        auto single = [&](int c) {
          T xs = Xs[c], xl = Xl[c];
          const T cp = pending ? Cp[c] : T(0);
          const T al = acm ? acm[c] : kc.alpha;
          Cp[c] = one(llit[3 * c], llit[3 * c + 1], llit[3 * c + 2], spos[3 * c], spos[3 * c + 1],
                      spos[3 * c + 2], xs, xl, cp, al);
          Xs[c] = xs;
          Xl[c] = xl;
        };
        if constexpr (sizeof(T) == 4) {
          // rounds of 4 clauses per thread; a remainder of at most 2 NT clauses goes out as
          // pairs over twice as many threads
          const int count = t1 - t0, full_end = t0 + count / (4 * NT) * (4 * NT);
          const bool pairs = t1 - full_end <= 2 * NT;
          const int g_end = pairs ? full_end : full_end + ((t1 - full_end) & ~3);
          for (int c = t0 + 4 * tid; c < g_end; c += 4 * NT) {
            Group4 q;
            load_words4(q, llit, spos, c);
            load_state4(q, Xs, Xl, Cp, acm, kc.alpha, pending, c);
            T xs[4] = {q.xs.x, q.xs.y, q.xs.z, q.xs.w};
            T xl[4] = {q.xl.x, q.xl.y, q.xl.z, q.xl.w};
            T cc[4];
#pragma unroll
            for (int r = 0; r < 4; r++)
              cc[r] = one(i16_at(q.lw, 3 * r), i16_at(q.lw, 3 * r + 1), i16_at(q.lw, 3 * r + 2),
                          u16_at(q.qw, 3 * r), u16_at(q.qw, 3 * r + 1), u16_at(q.qw, 3 * r + 2),
                          xs[r], xl[r], f4_at(q.cp, r), f4_at(q.al, r));
            *reinterpret_cast<float4*>(Xs + c) = make_float4(xs[0], xs[1], xs[2], xs[3]);
            *reinterpret_cast<float4*>(Xl + c) = make_float4(xl[0], xl[1], xl[2], xl[3]);
            *reinterpret_cast<float4*>(Cp + c) = make_float4(cc[0], cc[1], cc[2], cc[3]);
          }
          if (pairs) {
            const int c = full_end + 2 * tid;
            if (c + 2 <= t1) {
              Pair p;
              load_pair(p, c);
              do_pair(p, c);
            } else if (c < t1) {
              single(c);
            }
          } else if (g_end + tid < t1) {
            single(g_end + tid);  // fewer than 4 clauses
          }
        } else {
          for (int c = t0 + 2 * tid; c < t1; c += 2 * NT) {
            if (c + 2 <= t1) {
              Pair p;
              load_pair(p, c);
              do_pair(p, c);
            } else {
              single(c);
            }
          }
        }
      }
      __syncthreads();  // the staging area is complete
      {
        const uint32_t* const wdst =
            RES == 2 ? reinterpret_cast<const uint32_t*>(gr_smem + LY.wdst) : sp.wdst;
        const int32_t* const woff = sp.woff;
        const int w0 = woff[i] - woff[0], nw = woff[i + 1] - woff[i];
        const int4* src = reinterpret_cast<const int4*>(stage);
        int4* dst = reinterpret_cast<int4*>(sp.ux + (s & 1) * tb.ux_len);
        for (int q0 = tid; q0 < nw; q0 += 4 * NT) {
          uint32_t at[4];
#pragma unroll
          for (int r = 0; r < 4; r++)
            if (q0 + r * NT < nw) at[r] = wdst[w0 + q0 + r * NT];
#pragma unroll
          for (int r = 0; r < 4; r++)
            if (q0 + r * NT < nw) st_word<T>(dst + at[r], src[q0 + r * NT]);
        }
      }
      if (i + 1 < g.kc) __syncthreads();  // before the next tile reuses the area
    }
    unsat = redux_add(unsat);
    vf = redux_add(vf);
    if (lane == 0) {
      cnt[0][w] = unsat;
      cnt[1][w] = vf;
    }
    if (tid == 0) s_ok = 1;
    trace_stamp(P, s, 3);
    __syncthreads();
    // the block's counts and, in block 0, the slot of step s + 2; then a fence, so that the
    // report of phase F carries them and the unsetting of the previous step's entries
    if (w == W - 1) {
      const int tu = redux_add(lane < W ? cnt[0][lane] : 0);
      const int tv = redux_add(lane < W ? cnt[1][lane] : 0);
      if (lane == 0) {
        if (b == 0) {
          GridStepSlot* z = &gs->slot[(s + 2) & 3];
          *reinterpret_cast<volatile unsigned long long*>(&z->word) = 0ull;
          *reinterpret_cast<volatile int*>(&z->loc) = 0;
          *reinterpret_cast<volatile int*>(&z->vfail) = 0;
        }
        if (tu) atomicAdd(&slot->loc, tu);
        if (tv) atomicAdd(&slot->vfail, tv);
        s_unsat = tu != 0 || tv != 0;
        __threadfence();
      }
    }
    if (P.trace) {
      trace_stamp(P, s, 4);
      trace_stamp(P, s, 5);
    }

    // ---- B: the block's variable tiles
    const uint16_t* const idx = RES >= 1 ? reinterpret_cast<const uint16_t*>(gr_smem + LY.csr) : sp.idx;
    int kmax = 0;
    for (int j = 0; j < g.kv; j++) {
      const int i0 = min(nv, j * g.TV), i1 = min(nv, i0 + g.TV);
      const int bb = sp.boff[j], be = sp.boff[j + 1];
      if (j > 0) __syncthreads();  // the previous bucket is no longer read
      {
        // the bucket's words, four polls in flight per thread
        int4* const src = reinterpret_cast<int4*>(sp.ux + (s & 1) * tb.ux_len + bb);
        int4* const dst = reinterpret_cast<int4*>(raw) + 1;
        const int nw = (be - bb) / kw;
        bool ok = true;
        for (int q0 = tid; q0 < nw; q0 += 4 * NT) {
          int4 v[4];
          take_words<T>(src, q0, NT, nw, v, ok);
#pragma unroll
          for (int r = 0; r < 4; r++)
            if (q0 + r * NT < nw) dst[q0 + r * NT] = v[r];
        }
        if (!ok) s_ok = 0;
      }
      if (tid == 0) {
        raw[0] = sizeof(T) == 4 ? T(0) : inf_val<T>();
        s_next = 0;
      }
      const uint16_t* const rt =
          (RES >= 1 ? reinterpret_cast<const uint16_t*>(gr_smem + LY.row) : sp.rows) + j * g.TVr * 32;
      if constexpr (sizeof(T) == 4) {
        constexpr int VPP = NT / 4;
        const int gl = tid & 3;
        uint4 q = make_uint4(0, 0, 0, 0);
        if (i0 + tid / 4 < i1) q = reinterpret_cast<const uint4*>(rt)[tid];
        __syncthreads();
        if (j == 0) trace_stamp(P, s, 6);
        for (int vb = i0; vb < i1; vb += VPP) {
          const int i = vb + tid / 4;
          const bool valid = i < i1;
          const uint4 qc = q;
          if (vb + VPP < i1 && i + VPP < i1)
            q = reinterpret_cast<const uint4*>(rt)[4 * (i + VPP - i0) + gl];
          int d = 0, e0 = 0;
          if (valid) {
            const int2 list = s_list[i];
            e0 = list.x;
            d = list.y;
          }
          const T dv = row_sum4<RES == 0>(reinterpret_cast<const float*>(raw), qc, idx + e0, d, gl);
          bool acc_k = false;
          if (valid) {  // lane k forms candidate k
            const T V = s_cur[i];
            const int8_t un = GENERAL ? s_unit[i] : 0;
            if (gl == 0) s_dv[i] = un != 0 ? T(un) * inf_val<T>() : dv;
            const T h = gl == 0 ? T(0.125) : gl == 1 ? T(0.0625) : gl == 2 ? T(0.03125)
                                                                           : T(0.015625);
            T c = add(V, mul(h, dv));
            if (un != 0) c = T(un);
            c = clampv(c, T(-1), T(1));
            acc_k = !(fabs((double)c - (double)V) >= 1.0);
          }
          const unsigned bal = __ballot_sync(0xffffffffu, acc_k);
          const unsigned gb = (bal >> (lane & ~3)) & 15u;
          if (valid) kmax = max(kmax, gb ? __ffs(gb) - 1 : kTrials);
        }
      } else {
        __syncthreads();
        if (j == 0) trace_stamp(P, s, 6);
        const double* ud = reinterpret_cast<const double*>(raw);
        auto finish = [&](int i, T dv) {
          const T V = s_cur[i];
          const int8_t un = GENERAL ? s_unit[i] : 0;
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
          s_dv[i] = un != 0 ? T(un) * inf_val<T>() : dv;
        };
        // the last four warps start with the lists that whole warps sum, the others with the
        // rest, and all of them end with what is left of the former
        const int q1 = s_nq[j];
        auto queue = [&]() {
          for (;;) {
            int q = 0;
            if (lane == 0) q = atomicAdd(&s_next, 1);
            q = __shfl_sync(0xffffffffu, q, 0);
            if (q >= q1) break;
            const int2 list = s_list[i0 + q];
            const double dv =
                list.y <= kRankMax
                    ? rank_sum<RES == 0>(ud, idx + list.x, list.y, s_rank + 2 * kRankMax * w, lane)
                    : sorted_sum<false, uint16_t, RES == 0>(ud, idx + list.x, list.y, lane);
            if (lane == 0) finish(i0 + q, T(dv));
          }
        };
        if (w >= W - 4) queue();
        for (int vb = i0 + q1 + 32 * w; vb < i1; vb += NT) {
          const int i = min(vb + lane, i1 - 1), r = i - i0;
          const int2 list = s_list[i];
          const uint4* row = reinterpret_cast<const uint4*>(rt) + (r >> 5) * 128 + (r & 31);
          const double dv = row_net_sum(ud, row, list.y);
          if (vb + lane < i1) finish(i, T(dv));
        }
        queue();
      }
    }
    kmax = redux_max(kmax);
    if (lane == 0) cnt[2][w] = kmax;
    __syncthreads();
    // the block's report: its trial index and whether it has unsatisfied clauses, from the
    // thread whose fence in phase A orders the block's counts and unset entries before it
    if (w == W - 1) {
      const int km = redux_max(lane < W ? cnt[2][lane] : 0);
      if (lane == 0) {
        unsigned long long add_w = 1ull;
#pragma unroll
        for (int k = 1; k <= kTrials; k++) add_w += (unsigned long long)(km >= k) << (8 * k);
        add_w += (unsigned long long)s_unsat << 40;
        atomicAdd(&slot->word, add_w);
      }
    }
    // dV to the inboxes of the blocks that read it
    {
      const int nsend = sp.nsend;
      const uint32_t* const sdst =
          RES == 2 ? reinterpret_cast<const uint32_t*>(gr_smem + LY.snd) : sp.sdst;
      const uint16_t* const ids =
          RES == 2 ? reinterpret_cast<const uint16_t*>(gr_smem + LY.snd + 4 * nsend) : sp.ids;
      int4* const in = reinterpret_cast<int4*>(sp.inbox + (s & 1) * tb.inbox_len);
      for (int q0 = tid; q0 < nsend; q0 += 4 * NT) {
        uint32_t at[4], e[4][kw / 2];  // two 16-bit variables per word
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const int q = q0 + r * NT;
          if (q < nsend) {
            at[r] = sdst[q];
            // (4-byte loads: with RES the lists start at any multiple of 4 bytes)
#pragma unroll
            for (int k = 0; k < kw / 2; k++)
              e[r][k] = reinterpret_cast<const uint32_t*>(ids)[q * (kw / 2) + k];
          }
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
          if (q0 + r * NT < nsend) {
            union {
              T v[kw];
              int4 q;
            } u;
#pragma unroll
            for (int k = 0; k < kw; k++)
              u.v[k] = s_dv[(e[r][k >> 1] >> (16 * (k & 1))) & 0xffffu];
            st_word<T>(in + at[r], u.q);
          }
      }
    }
    trace_stamp(P, s, 7);

    // ---- F: the last warp waits for the reports of all blocks, the others take the words of
    // the inbox meanwhile
    constexpr int kHeld = 4, NI = NT - 32;
    const int nin = sp.dcnt / kw;  // whole words
    int4 held[kHeld];
    int4* const in_w = reinterpret_cast<int4*>(sp.inbox + (s & 1) * tb.inbox_len + sp.in_place);
    bool in_ok = true;
    if (w != W - 1) {
      if (tid < nin) take_words<T>(in_w, tid, NI, nin, held, in_ok);
    } else if (lane == 0) {
      unsigned long long a;
      int ok = 1;
      long long it = 0;
      const unsigned want = (unsigned)B + (s == 0 ? P.barrier_extra : 0);
      while (((a = ld_acquire64(&slot->word)) & 0xffu) < want) {
        if (++it > kBarrierSpinLimit) {
          ok = 0;
          atomicExch(err, 1);
          break;
        }
      }
      if (!ok) s_ok = 0;
      const int kx = (a >> 32) & 0xff ? 4 : (a >> 24) & 0xff ? 3 : (a >> 16) & 0xff ? 2
                                                             : (a >> 8) & 0xff ? 1 : 0;
      const int unsat_any = (int)((a >> 40) & 0xff);
      const StepDecision d = decide(unsat_any, 0, kx, lc.step, I.max_steps);
      if (d.status == 1) {
        lc.solved_t = lc.t;
        lc.sol_k = kcur;
      }
      lc.done = d.status;
      lc.t_rhs = lc.t;
      lc.t = __dadd_rn(lc.t, d.ht);
      lc.step += 1;
      lc.set = set ^ 1;
      lc.kcur = d.kacc;
      lc.h = d.hs;
      s_kc.h = T(d.hs);
      lc.pending = 1;
    }
    __syncthreads();
    trace_stamp(P, s, 8);
    const T h = s_kc.h;
    auto apply = [&](int q, const int4& v) {
      const T* dv = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int r = 0; r < kw; r++) {
        const int k = kw * q + r;
        T c = add(sV[k], mul(h, dv[r]));
        // a pinned variable's owner sends its sign as an infinity
        if (GENERAL && fabs(dv[r]) == inf_val<T>()) c = dv[r];
        sV[k] = clampv(c, T(-1), T(1));
      }
    };
    if (w != W - 1) {
#pragma unroll
      for (int r = 0; r < kHeld; r++)
        if (tid + r * NI < nin) apply(tid + r * NI, held[r]);
      for (int q0 = tid + kHeld * NI; q0 < nin; q0 += kHeld * NI) {
        take_words<T>(in_w, q0, NI, nin, held, in_ok);
#pragma unroll
        for (int r = 0; r < kHeld; r++)
          if (q0 + r * NI < nin) apply(q0 + r * NI, held[r]);
      }
    }
    if (!in_ok) s_ok = 0;
    if (lc.done == 1) {  // V(step) for the solution report
      T* sol = sp.cand + (int64_t)(set * kTrials + kcur) * P.var_cap;
      for (int i = tid; i < nv; i += NT) sol[var_at(i)] = s_cur[i];
    }
    for (int i = tid; i < nv; i += NT) {
      T c = add(s_cur[i], mul(h, s_dv[i]));
      const int8_t un = GENERAL ? s_unit[i] : 0;
      if (un != 0) c = T(un);
      s_cur[i] = clampv(c, T(-1), T(1));
    }
    if (b == 0 && w == W - 1 && lane == 0) {  // the step's counts, complete with its reports
      loc = *reinterpret_cast<volatile int*>(&slot->loc);
      vfail = *reinterpret_cast<volatile int*>(&slot->vfail);
      if (loc < best_loc) {
        best_loc = loc;
        best_t = lc.t_rhs;
      }
    }
    steps_run++;
    __syncthreads();
    if (!s_ok) {
      if (tid == 0) atomicExch(err, 1);
      gave_up = true;
      break;  // every block gives up in turn
    }
    trace_stamp(P, s, 9);
  }

  // ---- end of the launch: state, energy of the last right-hand side, control record
  if (!gave_up && steps_run > 0) {
    T* cur = sp.cand + (int64_t)(lc.set * kTrials + lc.kcur) * P.var_cap;
    for (int i = tid; i < nv; i += NT) cur[var_at(i)] = s_cur[i];
    Sum2 e;
    for (int c = tid; c < c1 - c0; c += NT) {
      T C;
      if constexpr (RES == 2) {
        C = reinterpret_cast<T*>(gr_smem + LY.cp)[c];
        sp.Cp[c] = C;
        sp.Xs[c] = reinterpret_cast<T*>(gr_smem + LY.xs)[c];
        sp.Xl[c] = reinterpret_cast<T*>(gr_smem + LY.xl)[c];
      } else {
        C = sp.Cp[c];
      }
      e.add((double)C);
    }
    e = warp_sum2(e);
    if (lane == 0) {
      red[w][0] = e.s;
      red[w][1] = e.c;
    }
    __syncthreads();
    if (w == 0) {
      Sum2 p;
      if (lane < W) {
        p.s = red[lane][0];
        p.c = red[lane][1];
      }
      e = warp_sum2(p);
      if (lane == 0) epart[blockIdx.x] = make_double2(e.s, e.c);
    }
  }
  if (b == 0 && w == W - 1 && lane == 0) {
    gs->best_loc = best_loc;
    gs->best_t = best_t;
    gs->loc = loc;
    gs->vfail = vfail;
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(&gs->exits, 1u) == (unsigned)B - 1;
  }
  __syncthreads();
  Sum2 energy;
  if (s_last && w == 0) {  // the last block of the group to leave
    __threadfence();
    for (int q = lane; q < B; q += 32) {
      const double2 v = __ldcg(epart + g.blk0 + q);
      Sum2 p;
      p.s = v.x;
      p.c = v.y;
      energy.add(p);
    }
    energy = warp_sum2(energy);
  }
  if (s_last && tid == 0) {
    if (!gave_up && steps_run > 0) {
      InstCtrl* S = P.ctrl + g.inst;
      S->step = lc.step;
      S->set = lc.set;
      S->kcur = lc.kcur;
      S->pending = 1;
      S->best_loc = *reinterpret_cast<volatile int*>(&gs->best_loc);
      S->best_t = *reinterpret_cast<volatile double*>(&gs->best_t);
      S->loc = *reinterpret_cast<volatile int*>(&gs->loc);
      S->vfail = *reinterpret_cast<volatile int*>(&gs->vfail);
      S->t = lc.t;
      S->h_state = lc.h;
      S->energy = energy.value();
      if (lc.done == 1) {
        S->solved_step = lc.step - 1;
        S->solved_t = lc.solved_t;
        S->sol_set = lc.set ^ 1;
        S->sol_k = lc.sol_k;
      }
      if (lc.done) {
        S->done = lc.done;
        atomicSub(P.active, 1);
        const int pos = atomicAdd(P.ring_tail, 1);
        P.ring[pos % P.ring_cap] = g.inst;
      }
    }
    volatile unsigned int* z = reinterpret_cast<volatile unsigned int*>(gs);
    for (unsigned i = 0; i < sizeof(GridSync) / 4; i++) z[i] = 0u;
    __threadfence();
  }
  trace_launch(P, 1);
}

}  // namespace dmm
