// Right-hand side of a 3-SAT formula for callers that cannot allocate device memory.
//
// Some callers run where cudaMalloc is not available to them: inside a host framework
// whose caching allocator owns all device memory (a second allocator would fragment it or
// fail), or in a plug-in that may only touch the buffers it is handed.
// dmm_rhs3_f32_noalloc serves them: the caller passes device inputs and outputs, and the
// intermediate data (per-literal contributions, clause values, the variable->slot CSR and
// counters) lives in one file-scope __device__ array of fixed size, so the call performs
// no device allocation of its own.
//
// The array, g_na_scratch, is about 2.1 MB on every GPU that loads the
// library, for the life of the process.  It bounds the formula: at most NA_MAX_VARS
// variables and NA_MAX_CLAUSES clauses of exactly three literals, each variable in at
// most NA_MAX_OCC literal slots.  The clause memory rate is the scalar alpha of the
// parameters (no per-clause alpha).
//
// Four launches: one checks the literals and counts occurrences, one lays out the variables' slot
// lists, one evaluates the clauses and fills the lists, one sums them; a failed check keeps the
// last two from writing dxdt or loc.  The last block of the last launch writes the counters
// (literals out of range, over-long variable lists) to page-locked host memory and the call waits
// for the caller's stream once to read them, so it blocks the calling thread until the work
// queued before it and its own finish.
//
// The launches are ordinary ones: a block runs wherever an SM has room.  One cooperative launch
// with three grid barriers needs room for all its blocks at once, so it would wait for every SM
// that a kernel on another of the caller's streams holds, and could not run at all beside one that
// waits for this call's result.  As programmatic dependents (na_wait) they cost no more than the
// one launch did; what is left is launch and host latency, the atomics that count and place the
// slots, and the chain of dependent loads of a list.  us per call at (n, m) = (1,000, 8,000) /
// (8,009, 64,007) / (32,000, 65,536): nine launches with two host waits 67 / 98 / 155; one
// cooperative launch 30.6 / 43.9 / 44.3; four launches one after another 36.1 / 50.1 / 46.0; as
// dependents 30.9 / 43.1 / 40.2.
//
// Every call uses the same array and leaves its contents behind, but for the parts that must
// start at zero: it zeroes them at its end and checks them at its start (counts left by calls
// that raced are cleared and the launches repeated).  Calls whose work overlaps on the GPU
// (different streams, or different host threads on one device) race on the array and must be
// serialized by the caller.
//
// Host code cannot use g_na_scratch's name as a device address.  On its first call on a
// device, the entry point looks the address up with cudaGetSymbolAddress while that
// device is current and keeps it for later calls on that device.
//
// The arithmetic is the production FP32 path's (the same clause and canonical-sum device
// functions), so the output equals dmm_instance_rhs on an FP32 instance bit for bit.
#include <mutex>

#include "dmm_pack.h"
#include "dmm_step.cuh"

namespace dmm {
namespace {

constexpr int NA_MAX_VARS = 1 << 15;
constexpr int NA_MAX_CLAUSES = 1 << 16;
constexpr int NA_MAX_SLOTS = 3 * NA_MAX_CLAUSES;
constexpr int NA_MAX_OCC = 1024;  // longest per-variable slot list the sorter handles
constexpr int NA_THREADS = 512;
constexpr int NA_MAX_DEVICES = 64;

struct NaScratch {
  int2 list[NA_MAX_SLOTS];      // slots of the variables with their contributions
  float C[NA_MAX_CLAUSES];      // C_m of each clause
  int32_t cnt[NA_MAX_VARS];     // occurrences (zero between calls)
  int32_t fill[NA_MAX_VARS];    // list cursors: the lists' ends once filled
  // [0] unsatisfied clauses, [1] long lists, [2] bad literals, [3] slots handed out, [4] blocks
  // of the last launch that have left (all zero between calls)
  int32_t counters[8];
};
static_assert(sizeof(NaScratch) < (size_t(22) << 20) / 10, "about 2.1 MB, as documented");

__device__ __align__(256) NaScratch g_na_scratch;

std::mutex g_na_mu;
NaScratch* g_na_addr[NA_MAX_DEVICES] = {nullptr};
int32_t* g_na_flags[NA_MAX_DEVICES] = {nullptr};  // page-locked host memory, four ints

// Canonical sum (tree_sum) of variable v's contributions, by one warp: its d slots, in no
// particular order in the list, are ranked (by shuffles up to 32 of them, else sorted in buf)
// so that the slot of rank j is added to the j mod 32-th partial.
__device__ __forceinline__ float na_sum(const NaScratch* s, int first, int d, int32_t* buf,
                                        int lane) {
  float p = 0.f;
  if (d <= 32) {
    int2 e = make_int2(0x7fffffff, 0);
    if (lane < d) e = __ldcg(s->list + first + lane);
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) rank += __shfl_sync(0xffffffffu, e.x, j) < e.x;
    if (lane < d) buf[rank] = e.y;
    __syncwarp();
    if (lane < d) p = add(0.f, __int_as_float(buf[lane]));
    __syncwarp();
  } else {
    int N = 64;
    while (N < d) N <<= 1;
    int32_t* val = buf + NA_MAX_OCC;
    for (int j = lane; j < N; j += 32) {
      int2 e = make_int2(0x7fffffff, 0);
      if (j < d) e = __ldcg(s->list + first + j);
      buf[j] = e.x;
      val[j] = e.y;
    }
    __syncwarp();
    for (int k = 2; k <= N; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int e = lane; e < N; e += 32) {
          const int q = e ^ j;
          if (q > e) {
            const bool up = (e & k) == 0;
            const int32_t a = buf[e], b = buf[q];
            if (up ? (b < a) : (a < b)) {
              const int32_t t = val[e];
              buf[e] = b;
              buf[q] = a;
              val[e] = val[q];
              val[q] = t;
            }
          }
        }
        __syncwarp();
      }
    for (int j = lane; j < d; j += 32) p = add(p, __int_as_float(val[j]));
    __syncwarp();
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) p = add(p, __shfl_xor_sync(0xffffffffu, p, off));
  return p;
}

// The launches after the first are programmatic dependents: their blocks may start once every block
// of the launch before has started (all of them are on an SM by then, so none waits for room that
// a later launch holds) and wait here until it has ended and its writes are visible.
__device__ __forceinline__ void na_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void na_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Literals in range and occurrence counts.
__global__ void __launch_bounds__(NA_THREADS)
    k_na_count(NaScratch* s, const int32_t* __restrict__ lits, int n, int m) {
  na_next();
  int bad = 0;
  for (int q = blockIdx.x * NA_THREADS + threadIdx.x; q < 3 * m; q += gridDim.x * NA_THREADS) {
    const int l = lits[q];
    if (l == 0 || l > n || l < -n) bad++;
    else atomicAdd(&s->cnt[abs(l) - 1], 1);
  }
  bad = warp_sum_i(bad);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(&s->counters[2], bad);
}

// A range for every list (their order does not matter); over-long lists.
__global__ void __launch_bounds__(NA_THREADS) k_na_lists(NaScratch* s, int n) {
  na_next();
  na_wait();
  const int lane = threadIdx.x & 31;
  const int v = blockIdx.x * NA_THREADS + threadIdx.x;  // (whole warps: the grid covers n)
  const int c = v < n ? s->cnt[v] : 0;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  int first = 0;
  if (lane == 31) first = atomicAdd(&s->counters[3], incl);
  first = __shfl_sync(0xffffffffu, first, 31);
  if (v < n) s->fill[v] = first + incl - c;
  if (c > NA_MAX_OCC) atomicAdd(&s->counters[1], 1);
}

// What the first two launches found: 0 nothing, 1 a check failed, 2 the counts do not add up (they
// were not all zero before the call).
__device__ __forceinline__ int na_fault(const NaScratch* s, int m) {
  const int longs = s->counters[1], bad = s->counters[2], slots = s->counters[3];
  return slots + bad != 3 * m ? 2 : bad || longs ? 1 : 0;
}

__global__ void __launch_bounds__(NA_THREADS)
    k_na_clause(NaScratch* s, const int32_t* __restrict__ lits, int n, int m,
                const float* __restrict__ x, ClauseConsts<float> kc) {
  na_next();
  na_wait();
  if (na_fault(s, m)) return;
  int unsat = 0;
  for (int c = blockIdx.x * NA_THREADS + threadIdx.x; c < m; c += gridDim.x * NA_THREADS) {
    const int l0 = lits[3 * c], l1 = lits[3 * c + 1], l2 = lits[3 * c + 2];
    const int p0 = atomicAdd(&s->fill[abs(l0) - 1], 1), p1 = atomicAdd(&s->fill[abs(l1) - 1], 1),
              p2 = atomicAdd(&s->fill[abs(l2) - 1], 1);
    float u0, u1, u2;
    bool ss;
    const float C = clause3(l0, l1, l2, x[abs(l0) - 1], x[abs(l1) - 1], x[abs(l2) - 1], x[n + c],
                            x[n + m + c], kc, u0, u1, u2, ss);
    s->list[p0] = make_int2(3 * c, __float_as_int(u0));
    s->list[p1] = make_int2(3 * c + 1, __float_as_int(u1));
    s->list[p2] = make_int2(3 * c + 2, __float_as_int(u2));
    s->C[c] = C;
    unsat += !(C < 0.5f);
  }
  unsat = warp_sum_i(unsat);
  if ((threadIdx.x & 31) == 0 && unsat) atomicAdd(&s->counters[0], unsat);
}

// dV of every variable, dXs and dXl of every clause (x may be dxdt: an entry is read by the thread
// that writes it).  The last block to leave reports and clears the counters.  flags (host memory):
// over-long lists, bad literals, counts that do not add up.
__global__ void __launch_bounds__(NA_THREADS)
    k_na_sum(NaScratch* s, int n, int m, const float* x, ClauseConsts<float> kc, float* dxdt,
             int32_t* loc, volatile int32_t* flags) {
  extern __shared__ int32_t na_smem[];  // 2 NA_MAX_OCC per warp
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int gt = blockIdx.x * NA_THREADS + tid, GT = gridDim.x * NA_THREADS;
  na_wait();
  const int fault = na_fault(s, m);
  if (fault) {  // nothing is written to dxdt and loc
    for (int v = gt; v < n; v += GT) s->cnt[v] = 0;
  } else {
    for (int v = blockIdx.x * (NA_THREADS / 32) + w; v < n; v += gridDim.x * (NA_THREADS / 32)) {
      const int d = s->cnt[v], end = s->fill[v];
      const float dv = na_sum(s, end - d, d, na_smem + w * 2 * NA_MAX_OCC, lane);
      if (lane == 0) {
        dxdt[v] = dv;
        s->cnt[v] = 0;
      }
    }
    for (int c = gt; c < m; c += GT) {
      const float xs = clampv(x[n + c], 0.f, 1.f);
      const float C = s->C[c];
      dxdt[n + c] = mul(mul(kc.beta, add(xs, kc.eps)), sub(C, kc.gamma));
      dxdt[n + m + c] = mul(kc.alpha, sub(C, kc.delta));
    }
    if (gt == 0) *loc = s->counters[0];
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&s->counters[4], 1) == (int)gridDim.x - 1) {
      __threadfence();
      flags[0] = s->counters[1];
      flags[1] = s->counters[2];
      flags[2] = fault == 2;
      for (int k = 0; k < 8; k++) s->counters[k] = 0;
      __threadfence_system();
    }
  }
}

}  // namespace
}  // namespace dmm

using namespace dmm;

extern "C" dmm_status dmm_rhs3_f32_noalloc(const int32_t* lits, int32_t n, int32_t m,
                                           const float* x, const dmm_params* p, float* dxdt,
                                           int32_t* loc, void* stream) {
  clear_error();
  if (!lits || !x || !dxdt || !loc || n <= 0 || m < 0) {
    set_error("dmm_rhs3_f32_noalloc: null buffer or bad size");
    return DMM_ERR_ARG;
  }
  if (n > NA_MAX_VARS || m > NA_MAX_CLAUSES) {
    set_error("dmm_rhs3_f32_noalloc: n=%d m=%d exceeds the fixed scratch (at most %d variables "
              "and %d clauses)", n, m, NA_MAX_VARS, NA_MAX_CLAUSES);
    return DMM_ERR_ARG;
  }
  int dev = 0;
  DMM_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= NA_MAX_DEVICES) {
    set_error("dmm_rhs3_f32_noalloc: device %d out of range", dev);
    return DMM_ERR_ARG;
  }
  NaScratch* s = nullptr;
  int32_t* flags = nullptr;
  {
    std::lock_guard<std::mutex> g(g_na_mu);
    if (!g_na_addr[dev]) {
      void* a = nullptr;
      DMM_CUDA(cudaGetSymbolAddress(&a, g_na_scratch));
      void* h = nullptr;
      DMM_CUDA(cudaHostAlloc(&h, 4 * sizeof(int32_t), cudaHostAllocPortable));
      g_na_flags[dev] = static_cast<int32_t*>(h);
      g_na_addr[dev] = static_cast<NaScratch*>(a);
    }
    s = g_na_addr[dev];
    flags = g_na_flags[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  dmm_params d;
  dmm_params_default(&d);
  if (!p) p = &d;
  ClauseConsts<float> kc;
  kc.beta = float(p->beta);
  kc.gamma = float(p->gamma);
  kc.delta = float(p->delta);
  kc.eps = float(p->epsilon);
  kc.zeta = float(p->zeta);
  kc.alpha = float(p->alpha);
  kc.h = 0.f;
  {
    int32_t v = (int32_t)((uint32_t)p->xl_max * (uint32_t)m);  // dynex.cc:2358-2359
    if (v <= 0) v = 0x7fffffff;
    kc.xlmax = float((double)v);
  }
  const int L = 3 * m;
  constexpr int kSmem = (NA_THREADS / 32) * 2 * NA_MAX_OCC * (int)sizeof(int32_t);
  int sms = 0;
  DMM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  DMM_CUDA(allow_smem((const void*)k_na_sum, kSmem));
  // a thread per slot or clause (at most two blocks per SM), a warp per variable in a few rounds
  // (the sorters take half an SM's shared memory each)
  auto blocks = [&](int64_t threads, int most) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((threads + NA_THREADS - 1) / NA_THREADS, most));
  };
  const unsigned g_slots = blocks(L, 2 * sms), g_vars = blocks(n, NA_MAX_VARS / NA_THREADS),
                 g_clauses = blocks(m, 2 * sms), g_sum = blocks(std::max<int64_t>(m, 8 * (int64_t)n), sms);
  volatile int32_t* hf = flags;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(NA_THREADS);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  for (int attempt = 0; attempt < 2; attempt++) {
    hf[0] = hf[1] = hf[2] = 0;
    k_na_count<<<g_slots, NA_THREADS, 0, st>>>(s, lits, n, m);
    DMM_CUDA(cudaGetLastError());
    cfg.gridDim = dim3(g_vars);
    DMM_CUDA(cudaLaunchKernelEx(&cfg, k_na_lists, s, n));
    cfg.gridDim = dim3(g_clauses);
    DMM_CUDA(cudaLaunchKernelEx(&cfg, k_na_clause, s, lits, n, m, x, kc));
    cfg.gridDim = dim3(g_sum);
    cfg.dynamicSmemBytes = kSmem;
    DMM_CUDA(cudaLaunchKernelEx(&cfg, k_na_sum, s, n, m, x, kc, dxdt, loc, hf));
    cfg.dynamicSmemBytes = 0;
    DMM_CUDA(cudaStreamSynchronize(st));
    if (hf[2] == 0) break;
    // the scratch was not as a finished call leaves it
    DMM_CUDA(cudaMemsetAsync(s, 0, sizeof(NaScratch), st));
    DMM_CUDA(cudaStreamSynchronize(st));
    if (attempt == 1) {
      set_error("dmm_rhs3_f32_noalloc: another call used the scratch at the same time");
      return DMM_ERR_CUDA;
    }
  }
  if (hf[1] > 0) {
    set_error("dmm_rhs3_f32_noalloc: %d literals outside [-n, n] or zero", hf[1]);
    return DMM_ERR_LITERAL;
  }
  if (hf[0] > 0) {
    set_error("dmm_rhs3_f32_noalloc: a variable occurs in more than %d literal slots", NA_MAX_OCC);
    return DMM_ERR_ARG;
  }
  return DMM_OK;
}
