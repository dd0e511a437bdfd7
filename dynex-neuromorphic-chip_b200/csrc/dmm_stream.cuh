// Streaming form of the FP32 integration step for one large formula, whose blocks cannot keep the
// voltages of all their clauses: clause tiles and variable tiles pass through shared memory one
// after another, many steps per cooperative launch, three grid barriers per step.
//
//   A  per clause tile: its voltage list (contiguous in the tile's inbox, arriving by asynchronous
//      copies while the previous tile is evaluated), clauses through 16-bit list-local literals,
//      contributions into a staging area grouped by variable tile, whose 16-byte words go to
//      those tiles' buckets;                                            grid barrier
//   B  per variable tile: its bucket (contiguous, arriving while the previous tile is summed),
//      canonical sums through a table of bucket places, dV to global memory;
//                                                      grid barrier, step decision
//   C  the accepted voltages of the block's variables, and from them every inbox entry they
//      belong to (16-byte words, contiguous per list and block);        grid barrier
//
// Gathering a tile's voltages from the voltage array instead reads one 32-byte sector per
// 4-byte entry once a formula is much larger than a tile (n = 10^6: 757 MB of sectors and a 94 MB
// index list per step); written by their owners they are 94 MB in and 94 MB out, at the price
// of the third barrier (about 3 us).
//
// Measured (FP32, 8 clauses per variable, us per step against the staged form's several tiles per
// block): n = 4 10^5 89 / 96, 6 10^5 138 / 146, 10^6 235 / 267, 1.5 10^6 398 / 416; clauses of
// 1 to 8 literals, n = 4 10^5 156 / 189 (tile form).  Bound by memory traffic: about 900 MB per step
// at n = 10^6 (clause memories 192, literal and place words 96, buckets and lists in and out
// 430, row tables 64, send words 72, destinations 30).  Tried: L2 evict-last for the
// exchanged words with evict-first tables (247), clause groups of 4 loaded ahead (285: spills),
// chunks padded to 16 bytes instead of whole sectors (240; smaller tiles 260-330).
//
// Values and sums are computed from the same operands in the same order as in the other forms.
#pragma once

#include "dmm_cluster.cuh"
#include "dmm_grid.cuh"

namespace dmm {

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits for all but the newest `N` groups of this thread's copies.
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Steps of the launch: counters in the launch area of the pack (StepAcc slots alternate by step,
// as in k_staged).
template <bool GENERAL>
__global__ void __launch_bounds__(kStreamThreads, 1)
    k_stream(PackView<float> P, GridTables tb, const GridGroup* __restrict__ groups,
             StreamLayout LY, float* __restrict__ dv_all, int nsteps, unsigned int* bar,
             double* __restrict__ epart, int* err) {
  using T = float;
  constexpr int NT = kStreamThreads;
  constexpr int W = NT / 32;
  constexpr int kw = 4;  // values per 16-byte word
  extern __shared__ __align__(16) unsigned char st_smem[];
  __shared__ InstDesc I;
  __shared__ GridGroup g;
  __shared__ GridCtrl lc;
  __shared__ ClauseConsts<T> s_kc;
  __shared__ int cnt[3][W];
  __shared__ double red[W];
  __shared__ int s_ok, s_last;
  {
    unsigned have;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(have));
    if ((unsigned)LY.total > have) return;  // (the host sizes the launch by the same layout)
  }
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, b = blockIdx.x;
  trace_launch(P, 0);
  if (tid == 0) {
    g = groups[0];
    I = P.inst[g.inst];
    const volatile InstCtrl* S = P.ctrl + g.inst;
    lc.done = S->done;
    // a wait of the launch before gave up (the host has not seen it yet): the lists and
    // buckets are those of the abandoned step, so none is taken
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
    s_ok = 1;
  }
  __syncthreads();
  const int TVb = g.TV * g.kv;
  const int v0 = min(I.n, b * TVb), nv = min(I.n, v0 + TVb) - v0;
  T* const ux = static_cast<T*>(tb.ux) + g.o_ux;
  T* const inbox = static_cast<T*>(tb.inbox) + g.o_list;
  T* const dv_g = dv_all + I.var0;
  const int32_t* const vend = P.vend + I.var0;
  unsigned int target = 0;
  bool ok = true;

  // C: voltages of the block's variables at `cur` (their new value when h is given) to the
  // inboxes (unless no step of this launch will read them)
  auto send = [&](const T* cur, T* nxt, bool step_h, T h, bool lists) {
    T* const sv = reinterpret_cast<T*>(st_smem);
    for (int i = tid; i < nv; i += NT) {
      T c = cur[v0 + i];
      if (step_h) {
        c = add(c, mul(h, dv_g[v0 + i]));
        if (GENERAL) {
          const int8_t un = P.unit[I.var0 + v0 + i];
          if (un != 0) c = T(un);
        }
        c = clampv(c, T(-1), T(1));
        nxt[v0 + i] = c;
      }
      sv[i] = c;
    }
    __syncthreads();
    int2 si = tb.sinfo[g.o_blk + b];
    if (!lists) si.y = 0;
    const uint32_t* const sdst = tb.sdst + g.o_push + si.x;
    const uint2* const ids = reinterpret_cast<const uint2*>(tb.ids + (g.o_push + si.x) * kw);
    int4* const in = reinterpret_cast<int4*>(inbox);
    for (int q0 = tid; q0 < si.y; q0 += 4 * NT) {
      uint32_t at[4];
      uint2 e[4];
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (q0 + r * NT < si.y) {
          at[r] = __ldcs(sdst + q0 + r * NT);
          e[r] = __ldcs(ids + q0 + r * NT);
        }
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (q0 + r * NT < si.y) {
          const unsigned int* k = reinterpret_cast<const unsigned int*>(&e[r]);
          union {
            T v[kw];
            int4 q;
          } u;
#pragma unroll
          for (int j = 0; j < kw; j++) u.v[j] = sv[(k[j >> 1] >> (16 * (j & 1))) & 0xffffu];
          in[at[r]] = u.q;
        }
    }
  };

  // the voltages of the first step
  if (lc.done == 0) {
    send(P.cand + (int64_t)(lc.set * kTrials + lc.kcur) * P.var_cap + I.var0, nullptr, false, T(0), true);
    target += P.barrier_extra;
    ok = grid_barrier<NT>(bar, target, err, &s_ok);
  }
  int steps_run = 0;
  for (int s = 0; s < nsteps && ok; s++) {
    if (lc.done != 0) break;  // grid-uniform: every block applies the same decisions
    trace_stamp(P, s, 0);
    StepAcc* acc = P.acc2 + (s & 1);
    const int set = lc.set, kcur = lc.kcur;
    const bool pending = lc.pending != 0;
    const ClauseConsts<T>& kc = s_kc;
    int unsat = 0, vf = 0;

    // ---- A: the block's clause tiles
    auto bring_list = [&](int i) {
      const int2 di = tb.dinfo[g.o_blk + b * g.kc + i];
      T* const dst = reinterpret_cast<T*>(st_smem + ((i & 1) ? LY.v1 : LY.v0));
      for (int q = kw * tid; q < di.y; q += kw * NT) cp_async16(dst + q, inbox + di.x + q);
      cp_async_commit();
    };
    bring_list(0);
    for (int i = 0; i < g.kc; i++) {
      const int ct = b * g.kc + i;
      if (i + 1 < g.kc) {
        bring_list(i + 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (i == 0) trace_stamp(P, s, 1);
      const T* const sV = reinterpret_cast<const T*>(st_smem + ((i & 1) ? LY.v1 : LY.v0));
      T* const stage = reinterpret_cast<T*>(st_smem + LY.stage);
      const int t0 = min(I.m, ct * g.TC), t1 = min(I.m, t0 + g.TC);
      T* const Xs = P.Xs + I.cls0;
      T* const Xl = P.Xl + I.cls0;
      T* const Cp = P.Cp + I.cls0;
      const T* const acm = I.has_alpha_cm ? P.alpha_cm + I.cls0 : nullptr;
      const int16_t* const llit = tb.llit + g.o_slot;
      const uint16_t* const spos = tb.spos + g.o_slot;
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
      auto single = [&](int c) {
        T xs = Xs[c], xl = Xl[c];
        const T cp = pending ? Cp[c] : T(0);
        const T al = acm ? acm[c] : kc.alpha;
        const int64_t q = 3 * (int64_t)c;
        Cp[c] = one(llit[q], llit[q + 1], llit[q + 2], spos[q], spos[q + 1], spos[q + 2], xs, xl, cp,
                    al);
        Xs[c] = xs;
        Xl[c] = xl;
      };
      if constexpr (GENERAL) {
        const int32_t* const coff = P.coff + I.cls0;
        for (int c = t0 + tid; c < t1; c += NT) {
          const int o = g.k3 ? 3 * c : __ldg(coff + c);
          const int o1 = g.k3 ? 3 * c + 3 : c + 1 < I.m ? __ldg(coff + c + 1) : g.L;
          T xs = Xs[c], xl = Xl[c];
          const T al = acm ? acm[c] : kc.alpha;
          if (pending) advance_memory(xs, xl, Cp[c], al, kc);
          bool ss;
          const T C = clause_any<T>(
              o1 - o, [&](int j) { return (int)__ldg(llit + o + j); },
              [&](int l) { return sV[abs(l) - 1]; }, xs, xl, kc,
              [&](int j) { return (int)__ldg(spos + o + j); }, [&](int p, T u) { stage[p] = u; },
              ss);
          Xs[c] = xs;
          Xl[c] = xl;
          Cp[c] = C;
          unsat += !(C < T(0.5));
          vf += !ss;
        }
      } else {
        auto pair = [&](int c) {
          const int* L3 = reinterpret_cast<const int*>(llit + 3 * (int64_t)c);
          const unsigned* Q3 = reinterpret_cast<const unsigned*>(spos + 3 * (int64_t)c);
          int lw[3];
          unsigned qw[3];
#pragma unroll
          for (int r = 0; r < 3; r++) {
            lw[r] = __ldg(L3 + r);
            qw[r] = __ldg(Q3 + r);
          }
          auto lit = [&](int k) {
            return (k & 1) ? (lw[k >> 1] >> 16) : (int)(short)(lw[k >> 1] & 0xffff);
          };
          auto pos = [&](int k) {
            return (int)((k & 1) ? (qw[k >> 1] >> 16) : (qw[k >> 1] & 0xffffu));
          };
          using T2 = float2;
          const T2 xs2 = __ldcs(reinterpret_cast<const T2*>(Xs + c));
          const T2 xl2 = __ldcs(reinterpret_cast<const T2*>(Xl + c));
          T2 cp2, al2;
          cp2.x = cp2.y = T(0);
          al2.x = al2.y = kc.alpha;
          if (pending) cp2 = __ldcs(reinterpret_cast<const T2*>(Cp + c));
          if (acm) al2 = *reinterpret_cast<const T2*>(acm + c);
          T xs[2] = {xs2.x, xs2.y}, xl[2] = {xl2.x, xl2.y}, cc[2];
          cc[0] = one(lit(0), lit(1), lit(2), pos(0), pos(1), pos(2), xs[0], xl[0], cp2.x, al2.x);
          cc[1] = one(lit(3), lit(4), lit(5), pos(3), pos(4), pos(5), xs[1], xl[1], cp2.y, al2.y);
          T2 o;
          o.x = xs[0];
          o.y = xs[1];
          __stcs(reinterpret_cast<T2*>(Xs + c), o);
          o.x = xl[0];
          o.y = xl[1];
          __stcs(reinterpret_cast<T2*>(Xl + c), o);
          o.x = cc[0];
          o.y = cc[1];
          __stcs(reinterpret_cast<T2*>(Cp + c), o);
        };
        for (int c = t0 + 2 * tid; c < t1; c += 2 * NT) {
          if (c + 2 <= t1) pair(c);
          else single(c);
        }
      }
      __syncthreads();  // the staging area is complete
      {
        const int w0 = tb.woff[g.o_ct + ct], nw = tb.woff[g.o_ct + ct + 1] - w0;
        const uint32_t* const wdst = tb.wdst + g.o_word + w0;
        const int4* src = reinterpret_cast<const int4*>(stage);
        int4* dst = reinterpret_cast<int4*>(ux);
#pragma unroll 4
        for (int q = tid; q < nw; q += NT) dst[__ldg(wdst + q)] = src[q];
      }
      __syncthreads();  // before the next tile reuses the area and the list after it arrives
    }
    unsat = redux_add(unsat);
    vf = redux_add(vf);
    if (lane == 0) {
      cnt[0][w] = unsat;
      cnt[1][w] = vf;
    }
    __syncthreads();
    if (w == 0) {
      const int tu = redux_add(lane < W ? cnt[0][lane] : 0);
      const int tv = redux_add(lane < W ? cnt[1][lane] : 0);
      if (lane == 0 && tu) atomicAdd(&acc->loc, tu);
      if (lane == 0 && tv) atomicAdd(&acc->vfail, tv);
    }
    trace_stamp(P, s, 3);
    ok = grid_barrier<NT>(bar, target, err, &s_ok);
    if (!ok) break;
    trace_stamp(P, s, 4);
    // every block has finished step s-1, whose decision read the other slot last
    if (tid == 0 && b == 0) {
      StepAcc* z = P.acc2 + ((s + 1) & 1);
      z->loc = 0;
      z->vfail = 0;
      z->kmax = 0;
    }

    // ---- B: the block's variable tiles
    const T* const cur = P.cand + (int64_t)(set * kTrials + kcur) * P.var_cap + I.var0;
    auto bring_bucket = [&](int j) {
      const int vt = b * g.kv + j;
      const int bb = tb.boff[g.o_vt + vt], be = tb.boff[g.o_vt + vt + 1];
      T* const dst = reinterpret_cast<T*>(st_smem + ((j & 1) ? LY.b1 : LY.b0));
      for (int q = tid; q < (be - bb) / kw; q += NT) cp_async16(dst + kw * (q + 1), ux + bb + kw * q);
      if (tid == 0) dst[0] = T(0);
      cp_async_commit();
    };
    int kmax = 0;
    bring_bucket(0);
    for (int j = 0; j < g.kv; j++) {
      const int vt = b * g.kv + j;
      const int i0 = min(I.n, vt * g.TV), i1 = min(I.n, i0 + g.TV);
      if (j + 1 < g.kv) {
        bring_bucket(j + 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (j == 0) trace_stamp(P, s, 5);
      const T* const raw = reinterpret_cast<const T*>(st_smem + ((j & 1) ? LY.b1 : LY.b0));
      const uint16_t* const rt = tb.rows + g.o_row + (int64_t)vt * g.TVr * 32;
      const uint16_t* const idx = tb.idx + g.o_slot;
      constexpr int VPP = NT / 4;
      const int gl = tid & 3;
      uint4 q = make_uint4(0, 0, 0, 0);
      if (i0 + tid / 4 < i1) q = __ldg(reinterpret_cast<const uint4*>(rt) + tid);
      for (int vb = i0; vb < i1; vb += VPP) {
        const int v = vb + tid / 4;
        const bool valid = v < i1;
        const uint4 qc = q;
        if (v + VPP < i1) q = __ldg(reinterpret_cast<const uint4*>(rt) + 4 * (v + VPP - i0) + gl);
        int d = 0, e0 = 0;
        T V = T(0);
        if (valid) {
          const int e1 = __ldg(vend + v);
          e0 = v > 0 ? __ldg(vend + v - 1) : 0;
          d = e1 - e0;
          V = cur[v];
        }
        const T dv = row_sum4<true>(raw, qc, idx + e0, d, gl);
        bool acc_k = false;
        if (valid) {  // lane k forms candidate k
          if (gl == 0) dv_g[v] = dv;
          const int8_t un = GENERAL ? P.unit[I.var0 + v] : 0;
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
      __syncthreads();  // before the next bucket but one arrives in this place
    }
    kmax = redux_max(kmax);
    if (lane == 0) cnt[2][w] = kmax;
    __syncthreads();
    if (w == 0) {
      const int km = redux_max(lane < W ? cnt[2][lane] : 0);
      if (lane == 0 && km) atomicMax(&acc->kmax, km);
    }
    trace_stamp(P, s, 6);
    ok = grid_barrier<NT>(bar, target, err, &s_ok);
    if (!ok) break;
    trace_stamp(P, s, 7);

    // ---- the step decision
    if (tid == 0) {
      const volatile StepAcc* A = acc;
      const int loc = A->loc, vfail = A->vfail, kx = A->kmax;
      const StepDecision d = decide(loc, vfail, kx, lc.step, I.max_steps);
      if (loc < lc.best_loc) {
        lc.best_loc = loc;
        lc.best_t = lc.t;
      }
      if (d.status == 1) {
        lc.solved_t = lc.t;
        lc.sol_k = kcur;
      }
      lc.done = d.status;
      lc.t = __dadd_rn(lc.t, d.ht);
      lc.step += 1;
      lc.set = set ^ 1;
      lc.kcur = d.kacc;
      lc.h = d.hs;
      s_kc.h = T(d.hs);
      lc.pending = 1;
      lc.loc = loc;
      lc.vfail = vfail;
    }
    __syncthreads();
    steps_run++;

    // ---- C: the accepted voltages, and the inboxes.  The launch's last step has no reader for
    // the latter (us per step at n = 10^6 with and without them there: launches of one step
    // 299 / 256, of 32 steps 236.7 / 235.4; leaving early instead of a loop bound of zero, and
    // skipping the barrier too, made the step's code slower: 261 / 242)
    send(cur, P.cand + (int64_t)(lc.set * kTrials + lc.kcur) * P.var_cap + I.var0, true, s_kc.h,
         s + 1 < nsteps && lc.done == 0);
    trace_stamp(P, s, 8);
    ok = grid_barrier<NT>(bar, target, err, &s_ok);
    trace_stamp(P, s, 9);
  }

  // ---- end of the launch: energy of the last right-hand side, control record
  cp_async_wait_all();
  if (ok && steps_run > 0) {
    double e = 0.0;
    const int c0 = min(I.m, b * g.TC * g.kc), c1 = min(I.m, c0 + g.TC * g.kc);
    for (int c = c0 + tid; c < c1; c += NT) e = __dadd_rn(e, (double)P.Cp[I.cls0 + c]);
    e = warp_sum_d(e);
    if (lane == 0) red[w] = e;
    __syncthreads();
    if (w == 0) {
      e = warp_sum_d(lane < W ? red[lane] : 0.0);
      if (lane == 0) epart[b] = e;
    }
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(bar + 1, 1u) == gridDim.x - 1;
    if (s_last) {  // the last block to leave
      __threadfence();
      if (ok && steps_run > 0) {
        double e = 0.0;
        for (unsigned q = 0; q < gridDim.x; q++) e = __dadd_rn(e, __ldcg(epart + q));
        InstCtrl* S = P.ctrl + g.inst;
        S->step = lc.step;
        S->set = lc.set;
        S->kcur = lc.kcur;
        S->pending = 1;
        S->best_loc = lc.best_loc;
        S->best_t = lc.best_t;
        S->loc = lc.loc;
        S->vfail = lc.vfail;
        S->t = lc.t;
        S->h_state = lc.h;
        S->energy = e;
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
      volatile unsigned int* z = bar;
      for (int q = 0; q < kLaunchAreaInts; q++) z[q] = 0u;
      __threadfence();
    }
  }
  trace_launch(P, 1);
}

}  // namespace dmm
