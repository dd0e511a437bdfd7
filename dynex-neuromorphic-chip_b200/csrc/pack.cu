// Pack: device arrays, device-built CSR, tile tables and the CUDA-graph step loop.
#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "dmm_admit.cuh"
#include "dmm_cluster.h"
#include "dmm_inst.cuh"
#include "dmm_step.cuh"
#include "dmm_xprep.cuh"
#include "dmm_pack.h"
#include "devmem.h"

namespace dmm {

// ---- errors --------------------------------------------------------------------------------
static thread_local std::string g_err;
void set_error(const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
}
void clear_error() { g_err.clear(); }
const char* last_error() { return g_err.c_str(); }

dmm_status validate_shape(const int32_t* lits, const int64_t* clause_off, int32_t n, int32_t m) {
  if (n <= 0 || m < 0 || clause_off == nullptr) {
    set_error("formula: need n > 0, m >= 0 and clause offsets");
    return DMM_ERR_ARG;
  }
  if (clause_off[0] != 0) {
    set_error("formula: clause_off[0] must be 0");
    return DMM_ERR_ARG;
  }
  const int64_t L = clause_off[m];
  if (L < 0 || L > 0x7fffffffll - 64) {
    set_error("formula: %lld literals outside the 2^31 slot limit", (long long)L);
    return DMM_ERR_ARG;
  }
  if (L > 0 && lits == nullptr) {
    set_error("formula: literals missing");
    return DMM_ERR_ARG;
  }
  return DMM_OK;
}

// Runs f(lo, hi, t) over the chunks t of [0, len) on the helper threads when len is large
// (these passes are bound by memory bandwidth, which one core does not reach); returns the
// number of chunks.
constexpr int kValidateThreads = kPoolHelpers + 1;
constexpr int64_t kValidateChunk = int64_t(1) << 14;  // elements per thread at least
template <class F>
static int host_parallel(int64_t len, F&& f) {
  const int T = (int)std::max<int64_t>(1, std::min<int64_t>(kValidateThreads, len / kValidateChunk));
  const int64_t per = (len + T - 1) / T;
  pool_run(T, [&](int t) { f(t * per, std::min(len, (t + 1) * per), t); });
  return T;
}

dmm_status locate_bad_literal(const int32_t* lits, int64_t len, int32_t n) {
  for (int64_t s = 0; s < len; s++) {
    const int32_t l = lits[s];
    if (l == 0 || l > n || l < -n) {
      set_error("formula: literal %d at position %lld out of range for n=%d", l, (long long)s, n);
      return DMM_ERR_LITERAL;
    }
  }
  return DMM_OK;
}

dmm_status validate_formula(const int32_t* lits, const int64_t* clause_off, int32_t n, int32_t m,
                            bool* k3, bool* may_have_units, bool check_literals) {
  if (n <= 0 || m < 0 || clause_off == nullptr) {
    set_error("formula: need n > 0, m >= 0 and clause offsets");
    return DMM_ERR_ARG;
  }
  if (clause_off[0] != 0) {
    set_error("formula: clause_off[0] must be 0");
    return DMM_ERR_ARG;
  }
  // branch-free passes (they vectorize), split over host threads for large formulas; the
  // slow loops below only locate an error
  int64_t lmin_t[kValidateThreads], lmax_t[kValidateThreads];
  const int nt_c = host_parallel(m, [&](int64_t lo, int64_t hi, int t) {
    int64_t a = INT64_MAX, b = INT64_MIN;
    for (int64_t c = lo; c < hi; c++) {
      const int64_t len = clause_off[c + 1] - clause_off[c];
      a = len < a ? len : a;
      b = len > b ? len : b;
    }
    lmin_t[t] = a;
    lmax_t[t] = b;
  });
  int64_t lmin = INT64_MAX, lmax = INT64_MIN;
  for (int t = 0; t < nt_c; t++) {
    lmin = std::min(lmin, lmin_t[t]);
    lmax = std::max(lmax, lmax_t[t]);
  }
  if (m > 0 && (lmin < 0 || lmax > DMM_MAX_CLAUSE_LITS)) {
    for (int32_t c = 0; c < m; c++) {
      const int64_t len = clause_off[c + 1] - clause_off[c];
      if (len < 0) {
        set_error("formula: clause offsets decrease at clause %d", c);
        return DMM_ERR_ARG;
      }
      if (len > DMM_MAX_CLAUSE_LITS) {
        set_error("CLAUSE %d HAS MORE THAN %d LITERALS", c, DMM_MAX_CLAUSE_LITS);
        return DMM_ERR_CLAUSE_LEN;
      }
    }
  }
  const int64_t L = clause_off[m];
  if (L > 0x7fffffffll - 64) {
    set_error("formula: %lld literals exceed the 2^31 slot limit", (long long)L);
    return DMM_ERR_ARG;
  }
  if (L > 0 && lits == nullptr) {
    set_error("formula: literals missing");
    return DMM_ERR_ARG;
  }
  // -n <= l <= n, l != 0: (unsigned)l + n lies in [0, 2n]
  const uint32_t un = (uint32_t)n, span = 2u * (uint32_t)n;
  uint32_t bad_t[kValidateThreads];
  const int nt_l = host_parallel(check_literals ? L : 0, [&](int64_t lo, int64_t hi, int t) {
    uint32_t bad = 0;
    for (int64_t s = lo; s < hi; s++) {
      const int32_t l = lits[s];
      bad |= (uint32_t)(l == 0) | (uint32_t)((uint32_t)l + un > span);
    }
    bad_t[t] = bad;
  });
  uint32_t bad = 0;
  for (int t = 0; t < nt_l; t++) bad |= bad_t[t];
  if (bad) DMM_TRY(locate_bad_literal(lits, L, n));
  *k3 = m > 0 && lmin == 3 && lmax == 3;
  if (may_have_units) *may_have_units = m > 0 && lmin <= 1;
  return DMM_OK;
}

// ---- range allocator ---------------------------------------------------------------------------
void RangeAlloc::reset(int64_t cap) {
  free_.clear();
  if (cap > 0) free_[0] = cap;
}

int64_t RangeAlloc::alloc(int64_t len) {
  len = round(std::max<int64_t>(len, 1));
  for (auto it = free_.begin(); it != free_.end(); ++it) {
    if (it->second >= len) {
      const int64_t start = it->first, rest = it->second - len;
      free_.erase(it);
      if (rest > 0) free_[start + len] = rest;
      return start;
    }
  }
  return -1;
}

void RangeAlloc::free(int64_t start, int64_t len) {
  len = round(std::max<int64_t>(len, 1));
  auto it = free_.emplace(start, len).first;
  auto nx = std::next(it);
  if (nx != free_.end() && it->first + it->second == nx->first) {
    it->second += nx->second;
    free_.erase(nx);
  }
  if (it != free_.begin()) {
    auto pv = std::prev(it);
    if (pv->first + pv->second == it->first) {
      pv->second += it->second;
      free_.erase(it);
    }
  }
}

int64_t RangeAlloc::largest_free() const {
  int64_t b = 0;
  for (auto& kv : free_) b = std::max(b, kv.second);
  return b;
}

// ---- pack ------------------------------------------------------------------------------------

namespace {
inline int blocks_for(int64_t work, int per = kThreads, int cap = 148 * 16) {
  int64_t b = (work + per - 1) / per;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (int)b;
}
constexpr int kMinClauseTile = 256;  // smallest clause tile (bounds the tile tables)
constexpr int kMinVarTile = 32;      // smallest variable tile
constexpr int kPersistThreads = 1024;  // block size of the cooperative step kernel
// FP64: 512 threads, so that the sorted sums and the clause code fit in registers without
// spilling (measured 74.3 vs 76.4 us per n=100k step with 1024 threads)
constexpr int kPersistThreads64 = 512;
constexpr int kStagedThreads = 1024;  // block size of the staged form
static int persist_threads(dmm_precision prec) {
  return prec == DMM_FP64 ? kPersistThreads64 : kPersistThreads;
}
constexpr int kSlotPad = 8;             // entries past the last slot of vslot and u
constexpr int kXpSmemMax = 220 * 1024;  // dynamic shared memory of the staged form, at most
// ... and of its several-tiles-per-block form: beyond about 195 KB a block takes the largest
// shared-memory carve-out, and the L1 left to the gathers shrinks (measured at 0.4-1.5 million
// variables: every tiling above the cap ran 8-30 % slower than the best one below it)
constexpr int kXpSmemMaxMT = 193 * 1024;  // with the form's ~1.4 KB of static shared memory
constexpr int staged_smem_max(bool mt) { return mt ? kXpSmemMaxMT : kXpSmemMax; }
constexpr int kClusterChunk = 8;        // launches of steps_per_graph steps run() makes one of
constexpr int kStreamSlots = 9000000;   // literals from which the streaming form runs a formula
constexpr int kXpMaxTiles = 1 << 14;    // clause or variable tiles of the staged form, at most
constexpr int kStatusInts = 8;           // ring_tail_d_
constexpr int64_t kDirectCopy = 1 << 13; // doubles the driver's own pageable copies move
constexpr int kMiscInts = 48;            // misc_d_: 192 bytes
constexpr int kMiscLaunch = 16;          // misc_d_ index of the per-launch area (byte 64)
constexpr int kMiscAcc2 = 20;            // misc_d_ index of the StepAcc pair (byte 80)
}  // namespace

int64_t Pack::bytes_per(dmm_precision prec, int64_t n, int64_t m, int64_t slots,
                        bool with_alpha_cm) {
  const int64_t t = prec == DMM_FP64 ? 8 : 4;
  n = RangeAlloc::round(std::max<int64_t>(n, 1));
  m = RangeAlloc::round(std::max<int64_t>(m, 1));
  slots = RangeAlloc::round(std::max<int64_t>(slots, 1));
  // per slot: literal, CSR entry, variable-major position (4 each) and the contribution
  int64_t b = m * (3 * t + 4 + (with_alpha_cm ? t : 0)) + slots * (12 + t) + n * (8 * t + 9);
  b += (m / kMinClauseTile + 1) * (8 + 16) + (n / kMinVarTile + 1) * 16;
  b += sizeof(InstDesc) + sizeof(InstCtrl) + 8;
  return b;
}

Pack::~Pack() {
  if (dev_ >= 0) cudaSetDevice(dev_);
  if (stream_) cudaStreamSynchronize(stream_);
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
  if (graph_) cudaGraphDestroy(graph_);
  void* ptrs[] = {Xs_,      Xl_,        Cp_,      alpha_cm_,   u_,         cand_,
                  coff_,    lit_,       vslot_,   vend_,       fill_,      unit_,
                  epart_,   inst_d_,    ctrl_d_,  ctiles_d_,   vtiles_d_,  ntiles_d_,
                  queue_d_, ring_d_,  ring_tail_d_, scan_tmp_, longv_d_,
                  stage_,   aux_ctiles_d_, aux_vtiles_d_, flush_, live_d_, misc_d_, order_d_,
                  upos_,    trace_};
  for (void* p : ptrs)
    if (p) dev_free(p);
  for (void* p : xbuf_)
    if (p) dev_free(p);
  for (void* p : gbuf_)
    if (p) dev_free(p);
  for (auto& e : ev_)
    if (e) cudaEventDestroy(e);
  for (auto& a : admit_) {
    if (a.host) pinned_free(a.host);
    if (a.dev) dev_free(a.dev);
    if (a.sent) cudaEventDestroy(a.sent);
  }
  for (auto& x : side_) {
    if (x.first) cudaStreamSynchronize(x.first);
    if (x.first) cudaStreamDestroy(x.first);
    if (x.second) cudaEventDestroy(x.second);
  }
  if (pinned_) pinned_free(pinned_);
  if (stream_) cudaStreamDestroy(stream_);
}

dmm_status Pack::init(const PackCaps& caps_in, bool with_alpha_cm, bool fixed_grid) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    set_error("no CUDA device");
    return DMM_ERR_NO_DEVICE;
  }
  if (dev_ < 0 || dev_ >= ndev) {
    set_error("device %d out of range (%d devices)", dev_, ndev);
    return DMM_ERR_ARG;
  }
  DMM_CUDA(cudaSetDevice(dev_));
  DMM_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
  DMM_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev_));
  for (auto& e : ev_) DMM_CUDA(cudaEventCreate(&e));
  with_alpha_cm_ = with_alpha_cm;
  fixed_grid_ = fixed_grid;
  tsize_ = prec_ == DMM_FP64 ? 8 : 4;
  caps_ = caps_in;
  if (caps_.insts < 1) caps_.insts = 1;
  caps_.vars = RangeAlloc::round(caps_.vars) + 32 * (int64_t)caps_.insts;
  caps_.clauses = RangeAlloc::round(caps_.clauses) + 32 * (int64_t)caps_.insts;
  caps_.slots = RangeAlloc::round(caps_.slots) + 32 * (int64_t)caps_.insts;
  const int64_t V = caps_.vars, C = caps_.clauses, S = caps_.slots, I = caps_.insts;
  ctile_cap_ = C / kMinClauseTile + I + 1;
  vtile_cap_ = V / kMinVarTile + I + 1;
  DMM_CUDA(dev_alloc(&Xs_, C * tsize_));
  DMM_CUDA(dev_alloc(&Xl_, C * tsize_));
  DMM_CUDA(dev_alloc(&Cp_, C * tsize_));
  if (with_alpha_cm) DMM_CUDA(dev_alloc(&alpha_cm_, C * tsize_));
  DMM_CUDA(dev_alloc(&coff_, C * 4));
  DMM_CUDA(dev_alloc(&lit_, S * 4));
  // the per-variable lists are read in aligned 16-byte words: padding past the last slot
  DMM_CUDA(dev_alloc(&vslot_, (S + kSlotPad) * 4));
  DMM_CUDA(dev_alloc(&upos_, S * 4));
  DMM_CUDA(dev_alloc(&u_, (S + kSlotPad) * tsize_));
  DMM_CUDA(dev_alloc(&cand_, 2 * kTrials * V * tsize_));
  DMM_CUDA(dev_alloc(&vend_, V * 4));
  DMM_CUDA(dev_alloc(&fill_, V * 4));
  DMM_CUDA(dev_alloc(&unit_, V));
  DMM_CUDA(dev_alloc(&epart_, ctile_cap_ * sizeof(double)));
  DMM_CUDA(dev_alloc(&inst_d_, I * sizeof(InstDesc)));
  DMM_CUDA(dev_alloc(&ctrl_d_, I * sizeof(InstCtrl)));
  DMM_CUDA(dev_alloc(&ctiles_d_, ctile_cap_ * sizeof(Tile)));
  DMM_CUDA(dev_alloc(&vtiles_d_, vtile_cap_ * sizeof(Tile)));
  DMM_CUDA(dev_alloc(&ntiles_d_, 4 * sizeof(int32_t)));
  DMM_CUDA(dev_alloc(&queue_d_, 2 * sizeof(int32_t)));
  DMM_CUDA(dev_alloc(&ring_d_, I * sizeof(int32_t)));
  // status words: [0] finished-ring tail, [2] long lists, [3] bad literals, [4] running
  // formulas, [5] barrier error
  DMM_CUDA(dev_alloc(&ring_tail_d_, kStatusInts * sizeof(int32_t)));
  active_d_ = ring_tail_d_ + 4;
  error_d_ = ring_tail_d_ + 5;
  longv_cap_ = (int32_t)(S / kSortCap + 2);
  DMM_CUDA(dev_alloc(&longv_d_, longv_cap_ * sizeof(int32_t)));
  DMM_CUDA(dev_alloc(&live_d_, I * sizeof(int32_t)));
  DMM_CUDA(dev_alloc(&order_d_, I * sizeof(int32_t)));
  // [0] live formulas, [1] error flag, [3] k_inst queue; bytes 64..191: grid-barrier
  // counter and the two step accumulators of the single-formula form (zeroed per launch)
  DMM_CUDA(dev_alloc(&misc_d_, kMiscInts * sizeof(int32_t)));
  DMM_CUDA(cudaMemsetAsync(misc_d_, 0, kMiscInts * sizeof(int32_t), stream_));
  DMM_CUDA(cudaMemsetAsync(ctrl_d_, 0, I * sizeof(InstCtrl), stream_));
  DMM_CUDA(cudaMemsetAsync(ntiles_d_, 0, 4 * sizeof(int32_t), stream_));
  DMM_CUDA(cudaMemsetAsync(queue_d_, 0, 2 * sizeof(int32_t), stream_));
  DMM_CUDA(cudaMemsetAsync(ring_tail_d_, 0, kStatusInts * sizeof(int32_t), stream_));
  DMM_CUDA(cudaMemsetAsync(cand_, 0, 2 * kTrials * V * tsize_, stream_));
  var_alloc_.reset(V);
  cls_alloc_.reset(C);
  slot_alloc_.reset(S);
  inst_h_.assign(I, InstDesc{});
  live_.assign(I, 0);
  add_serial_.assign(I, 0);
  cl_need_.assign(I, ClusterNeed{});
  tun_ = dmm_tuning{};
  DMM_TRY(set_tuning(&tun_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

dmm_status Pack::set_tuning(const dmm_tuning* t) {
  dmm_tuning n = *t;
  if (n.clause_tile < 0 || (n.clause_tile > 0 && (n.clause_tile % 4 || n.clause_tile < kMinClauseTile))) {
    set_error("clause_tile must be 0 (balanced) or a multiple of 4 that is >= %d", kMinClauseTile);
    return DMM_ERR_ARG;
  }
  if (n.var_tile < 0 || (n.var_tile > 0 && n.var_tile < kMinVarTile)) {
    set_error("var_tile must be 0 (balanced) or >= %d", kMinVarTile);
    return DMM_ERR_ARG;
  }
  if (prec_ == DMM_FP64) {
    if (n.var_group != 0 && n.var_group != 32) {
      set_error("FP64 mode reduces with one warp per variable (var_group 32)");
      return DMM_ERR_ARG;
    }
    n.var_group = 32;
  } else {
    if (n.var_group <= 0) n.var_group = 4;
    if (n.var_group != 1 && n.var_group != 2 && n.var_group != 4 && n.var_group != 8 &&
        n.var_group != 16 && n.var_group != 32) {
      set_error("var_group must be 1, 2, 4, 8, 16 or 32");
      return DMM_ERR_ARG;
    }
  }
  if (n.steps_per_graph <= 0) n.steps_per_graph = 32;
  if (n.steps_per_graph > 4096) n.steps_per_graph = 4096;
  if (n.blocks_per_sm < 0 || n.blocks_per_sm > 32) {
    set_error("blocks_per_sm out of range");
    return DMM_ERR_ARG;
  }
  if (n.l2_policy < 0 || n.l2_policy > 3) {
    set_error("l2_policy must be 0..3 (bit 0: no eviction hints, bit 1: L2 prefetch)");
    return DMM_ERR_ARG;
  }
  if (n.u_layout < 0 || n.u_layout > 2) {
    set_error("u_layout must be 0 (default), 1 (slot-major, no staging) or 2 (variable-major)");
    return DMM_ERR_ARG;
  }
  if (n.launch_mode < 0 || n.launch_mode > 3) {
    set_error("launch_mode must be 0 (auto), 1 (kernel per phase), 2 (cooperative tiles) or "
              "3 (one block per small formula)");
    return DMM_ERR_ARG;
  }
  tun_ = n;
  graph_stale_ = true;
  if (planned()) return commit_tiles();
  return DMM_OK;
}

int32_t Pack::num_live() const {
  int32_t c = 0;
  for (auto l : live_) c += l;
  return c;
}

int32_t Pack::free_insts() const {
  int32_t c = 0;
  for (auto l : live_) c += !l;
  return c;
}

dmm_status Pack::ensure_stage(int64_t doubles) {
  if (doubles <= stage_cap_) return DMM_OK;
  if (stage_) retire(stage_);
  stage_ = nullptr;
  stage_cap_ = 0;
  DMM_CUDA(dev_alloc(&stage_, doubles * sizeof(double)));
  stage_cap_ = doubles;
  return DMM_OK;
}

void Pack::retire(void* p) {
  // the block may still be read by work queued on this pack's stream, and the cache can
  // hand it to another stream at once
  cudaStreamSynchronize(stream_);
  dev_free(p);
}

// Small records travel as kernel arguments: stream-ordered, no host staging, no wait.
__global__ void k_put_desc(InstDesc* dst, InstDesc d) { *dst = d; }
__global__ void k_put_ctrl(InstCtrl* dst, InstCtrl c) { *dst = c; }
// The control record of a restarted formula; one that was not running is counted again.
__global__ void k_restart(InstCtrl* dst, InstCtrl c, int keep_best, int32_t* active) {
  if (dst->done != 0) atomicAdd(active, 1);
  if (keep_best) {
    c.best_loc = dst->best_loc;
    c.best_t = dst->best_t;
  }
  *dst = c;
}

// Signs of V on the device (the control record says which candidate holds it), so that
// one byte per variable crosses to the host: pre from the solving step's V (0 for V == 0;
// flag[0] = 1 when the formula is not solved), post from the current V (+1 / -1).
template <class T>
__global__ void k_signs(const InstCtrl* __restrict__ ctrl, const T* __restrict__ cand,
                        int64_t var_cap, int64_t var0, int n, int8_t* pre, int8_t* post,
                        int32_t* flag) {
  const InstCtrl c = *ctrl;
  if (pre && c.solved_step < 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *flag = 1;
    pre = nullptr;
  }
  const T* vs = cand + (int64_t)(c.sol_set * kTrials + c.sol_k) * var_cap + var0;
  const T* vc = cand + (int64_t)(c.set * kTrials + c.kcur) * var_cap + var0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (pre) {
      const T v = vs[i];
      pre[i] = v > T(0) ? 1 : (v < T(0) ? -1 : 0);
    }
    if (post) post[i] = vc[i] > T(0) ? 1 : -1;
  }
}


dmm_status Pack::upload_desc(int32_t idx) {
  DMM_TRY(flush_adds());
  k_put_desc<<<1, 1, 0, stream_>>>(inst_d_ + idx, inst_h_[idx]);
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

dmm_status Pack::write_ctrl(int32_t idx, const InstCtrl& c) {
  DMM_TRY(flush_adds());
  k_put_ctrl<<<1, 1, 0, stream_>>>(ctrl_d_ + idx, c);
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

__global__ void k_active_add(int32_t* a, int32_t d) { atomicAdd(a, d); }

dmm_status Pack::add_active(int32_t delta) {
  k_active_add<<<1, 1, 0, stream_>>>(active_d_, delta);
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

dmm_status Pack::read_ctrl(int32_t idx, InstCtrl* c) {
  if (!live(idx)) {
    set_error("instance %d is not live", idx);
    return DMM_ERR_ARG;
  }
  DMM_TRY(flush_adds());
  DMM_CUDA(cudaMemcpyAsync(c, ctrl_d_ + idx, sizeof(InstCtrl), cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

dmm_status Pack::read_ctrls(std::vector<InstCtrl>* out) {
  DMM_TRY(flush_adds());
  out->resize(caps_.insts);
  DMM_CUDA(cudaMemcpyAsync(out->data(), ctrl_d_, caps_.insts * sizeof(InstCtrl),
                           cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

static dmm_status scan_inclusive(int32_t* a, int64_t len, int32_t* tmp, cudaStream_t s) {
  constexpr int per = kThreads * 8;
  const int64_t nb = (len + per - 1) / per;
  if (nb <= 1) {
    k_scan_block<<<1, kThreads, 0, s>>>(a, (int)len, nullptr);
    DMM_CUDA(cudaGetLastError());
    return DMM_OK;
  }
  k_scan_block<<<(unsigned)nb, kThreads, 0, s>>>(a, (int)len, tmp);
  DMM_CUDA(cudaGetLastError());
  DMM_TRY(scan_inclusive(tmp, nb, tmp + nb, s));
  k_scan_add<<<(unsigned)nb, kThreads, 0, s>>>(a, (int)len, tmp);
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

dmm_status Pack::build_csr(const InstDesc& I, const int32_t* lits_host) {
  const int n = I.n, L = I.nslots;
  int32_t* vend = vend_ + I.var0;
  int32_t* fill = fill_ + I.var0;
  const int32_t* lit = lit_ + I.slot0;
  int32_t* vsl = vslot_ + I.slot0;
  DMM_CUDA(cudaMemsetAsync(vend, 0, (size_t)n * 4, stream_));
  if (L > 0) {
    k_count<<<blocks_for(L), kThreads, 0, stream_>>>(lit, L, n, vend, ring_tail_d_ + 3);
    DMM_CUDA(cudaGetLastError());
  }
  const int64_t need = n / (kThreads * 8) + 64;
  if (need > scan_tmp_cap_) {
    if (scan_tmp_) retire(scan_tmp_);
    scan_tmp_ = nullptr;
    DMM_CUDA(dev_alloc(&scan_tmp_, need * 2 * sizeof(int32_t)));
    scan_tmp_cap_ = need;
  }
  DMM_TRY(scan_inclusive(vend, n, scan_tmp_, stream_));
  k_fill_start<<<blocks_for(n), kThreads, 0, stream_>>>(vend, n, fill);
  DMM_CUDA(cudaGetLastError());
  if (L > 0) {
    k_scatter<<<blocks_for(L), kThreads, 0, stream_>>>(lit, L, n, fill, vsl);
    DMM_CUDA(cudaGetLastError());
  }
  // lists longer than the shared-memory sorter are appended to longv_d_ (count at
  // ring_tail_d_[2]) and sorted by resolve_long_lists() before the CSR is first used, so
  // that adding a formula needs no host synchronization
  const size_t smem = (kThreads / 32) * kSortCap * sizeof(int32_t);
  k_sort_lists<<<blocks_for(n, kThreads / 32), kThreads, smem, stream_>>>(
      vend, n, vsl, longv_d_, ring_tail_d_ + 2, (int32_t)I.var0, longv_cap_);
  DMM_CUDA(cudaGetLastError());
  long_pending_ = true;
  if (L > 0) {
    // variable-major position of every slot (the inverse of the sorted CSR)
    k_invert<<<blocks_for(L), kThreads, 0, stream_>>>(vsl, L, upos_ + I.slot0);
    DMM_CUDA(cudaGetLastError());
  }
  (void)lits_host;
  return DMM_OK;
}

dmm_status Pack::resolve_long_lists() {
  DMM_TRY(flush_adds());
  if (!long_pending_) return DMM_OK;
  int32_t counts[2] = {0, 0};  // long lists, literals the CSR build found out of range
  DMM_CUDA(cudaMemcpyAsync(counts, ring_tail_d_ + 2, sizeof counts, cudaMemcpyDeviceToHost,
                           stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  const int32_t nlong = counts[0];
  if (counts[1] > 0) {
    // a formula admitted with device_literal_check holds a bad literal: name it as the host
    // check would, then leave the counters for the caller to discard the pack
    for (int32_t i = 0; i < (int32_t)live_.size(); i++) {
      if (!live_[i]) continue;
      const InstDesc& I = inst_h_[i];
      std::vector<int32_t> h(I.nslots);
      DMM_CUDA(cudaMemcpy(h.data(), lit_ + I.slot0, (size_t)I.nslots * 4, cudaMemcpyDeviceToHost));
      DMM_TRY(locate_bad_literal(h.data(), I.nslots, I.n));
    }
    set_error("formula: %d literals out of range", counts[1]);
    return DMM_ERR_LITERAL;
  }
  if (nlong > 0) {
    // sorted on the host (setup only); an entry whose formula was removed meanwhile is
    // skipped, one whose range a later formula took is sorted again (harmless).  Past the
    // list's capacity (formulas with long lists added and removed repeatedly before a
    // commit) every long list of every live formula is taken.
    std::vector<int32_t> ids;
    if (nlong <= longv_cap_) {
      ids.resize(nlong);
      DMM_CUDA(cudaMemcpy(ids.data(), longv_d_, nlong * 4, cudaMemcpyDeviceToHost));
    } else {
      for (int32_t i = 0; i < (int32_t)live_.size(); i++) {
        if (!live_[i]) continue;
        const InstDesc& I = inst_h_[i];
        std::vector<int32_t> ends(I.n);
        DMM_CUDA(cudaMemcpy(ends.data(), vend_ + I.var0, (size_t)I.n * 4, cudaMemcpyDeviceToHost));
        for (int32_t v = 0; v < I.n; v++)
          if (ends[v] - (v > 0 ? ends[v - 1] : 0) > kSortCap) ids.push_back((int32_t)I.var0 + v);
      }
    }
    std::vector<int32_t> redo;
    std::vector<int32_t> seg;
    for (int32_t g : ids) {
      int32_t owner = -1;
      for (int32_t i = 0; i < (int32_t)live_.size(); i++)
        if (live_[i] && g >= inst_h_[i].var0 && g < inst_h_[i].var0 + inst_h_[i].n) owner = i;
      if (owner < 0) continue;
      const InstDesc& I = inst_h_[owner];
      const int32_t v = g - (int32_t)I.var0;
      int32_t e[2] = {0, 0};
      if (v > 0)
        DMM_CUDA(cudaMemcpy(e, vend_ + I.var0 + v - 1, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost));
      else
        DMM_CUDA(cudaMemcpy(e + 1, vend_ + I.var0, sizeof(int32_t), cudaMemcpyDeviceToHost));
      int32_t* vsl = vslot_ + I.slot0;
      seg.resize(e[1] - e[0]);
      DMM_CUDA(cudaMemcpy(seg.data(), vsl + e[0], seg.size() * 4, cudaMemcpyDeviceToHost));
      std::sort(seg.begin(), seg.end());
      DMM_CUDA(cudaMemcpy(vsl + e[0], seg.data(), seg.size() * 4, cudaMemcpyHostToDevice));
      if (std::find(redo.begin(), redo.end(), owner) == redo.end()) redo.push_back(owner);
    }
    for (int32_t i : redo) {
      const InstDesc& I = inst_h_[i];
      k_invert<<<blocks_for(I.nslots), kThreads, 0, stream_>>>(vslot_ + I.slot0, I.nslots,
                                                               upos_ + I.slot0);
      DMM_CUDA(cudaGetLastError());
    }
    DMM_CUDA(cudaMemsetAsync(ring_tail_d_ + 2, 0, sizeof(int32_t), stream_));
  }
  long_pending_ = false;
  return DMM_OK;
}

static double effective_xl_max(int32_t factor, int32_t m) {
  int32_t v = (int32_t)((uint32_t)factor * (uint32_t)m);  // dynex.cc:2358 in int arithmetic
  if (v <= 0) v = 0x7fffffff;
  return (double)v;
}

static void fill_params(InstDesc& I, const dmm_params* p) {
  dmm_params d;
  dmm_params_default(&d);
  if (!p) p = &d;
  I.alpha = p->alpha;
  I.beta = p->beta;
  I.gamma = p->gamma;
  I.delta = p->delta;
  I.eps = p->epsilon;
  I.zeta = p->zeta;
  I.xl_max = effective_xl_max(p->xl_max, I.m);
}

// Copies from pageable host memory have read their source when cudaMemcpyAsync returns;
// from page-locked memory they run later, so a call that copies from a caller's
// page-locked buffer waits for its stream before returning (the caller may reuse it).
static bool page_locked(const void* p) {
  if (!p) return false;
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;  // unknown: treat as page-locked
  }
  return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

template <class T>
static dmm_status upload_alpha(T* dst, const double* a, int32_t m, cudaStream_t s) {
  std::vector<T> h(m);
  for (int32_t i = 0; i < m; i++) h[i] = T(a[i]);
  DMM_CUDA(cudaMemcpyAsync(dst, h.data(), (size_t)m * sizeof(T), cudaMemcpyHostToDevice, s));
  DMM_CUDA(cudaStreamSynchronize(s));
  return DMM_OK;
}

// Bytes of the records at the start of a block.
int64_t Pack::admit_head() const {
  return (std::min<int64_t>(kAdmitRecs, caps_.insts) * (int64_t)sizeof(AdmitRec) + 15) & ~int64_t(15);
}

dmm_status Pack::stage_add(const InstDesc& I, int32_t idx, const int32_t* lits,
                           const int64_t* clause_off, bool units, const double* x0, bool* done) {
  *done = false;
  const int64_t n = I.n, m = I.m, L = I.nslots;
  auto al = [](int64_t b) { return (b + 15) & ~int64_t(15); };
  const int64_t b_lit = al(4 * L), b_coff = I.k3 ? 0 : al(4 * m), b_unit = units ? al(n) : 0,
                b_x = al((n + 2 * m) * (int64_t)tsize_);
  // a block holds what the pack can, up to kAdmitBytes: a batch of two small formulas takes no
  // 16 MB of device and page-locked memory for them
  const int64_t recs = std::min<int64_t>(kAdmitRecs, caps_.insts), head = admit_head();
  const int64_t cap = std::min<int64_t>(
      kAdmitBytes, head + 4 * caps_.slots + 4 * caps_.clauses + caps_.vars +
                       (int64_t)tsize_ * (caps_.vars + 2 * caps_.clauses) + 64 * recs);
  if (n > kAdmitVars || L > kAdmitSlots || head + b_lit + b_coff + b_unit + b_x > cap)
    return DMM_OK;
  if (admit_[admit_cur_].count == recs ||
      head + admit_[admit_cur_].used + b_lit + b_coff + b_unit + b_x > cap)
    DMM_TRY(flush_adds());
  AdmitBlock& A = admit_[admit_cur_];
  if (!A.host) {
    void *h = nullptr, *dv = nullptr;
    cudaError_t e = pinned_alloc(&h, cap);
    if (e == cudaSuccess) e = dev_alloc(&dv, cap);
    if (e == cudaErrorMemoryAllocation) {  // formulas are added one by one without the blocks
      cudaGetLastError();
      pinned_free(h);
      admit_off_ = true;
      return DMM_OK;
    }
    A.host = static_cast<unsigned char*>(h);
    A.dev = static_cast<unsigned char*>(dv);
    DMM_CUDA(e);
    DMM_CUDA(cudaEventCreateWithFlags(&A.sent, cudaEventDisableTiming));
  }
  if (A.busy) {  // its previous contents are still on their way
    DMM_CUDA(cudaEventSynchronize(A.sent));
    A.busy = false;
  }
  AdmitRec R{};
  R.I = I;
  R.c = running_ctrl(I, 0.0, 0);
  R.idx = idx;
  int64_t at = head + A.used;
  R.lit = at;
  unsigned char* const lit_at = A.host + at;
  at += b_lit;
  R.coff = R.unit = -1;
  if (!I.k3) {
    R.coff = at;
    int32_t* o = reinterpret_cast<int32_t*>(A.host + at);
    for (int64_t c = 0; c < m; c++) o[c] = (int32_t)clause_off[c];
    at += b_coff;
  }
  if (units) {
    R.unit = at;
    int8_t* u = reinterpret_cast<int8_t*>(A.host + at);
    std::memset(u, 0, (size_t)n);
    for (int64_t c = 0; c < m; c++)
      if (clause_off[c + 1] - clause_off[c] == 1) {
        const int32_t l = lits[clause_off[c]];
        u[std::abs(l) - 1] = l > 0 ? 1 : -1;
      }
    at += b_unit;
  }
  R.x = at;
  unsigned char* const x_at = A.host + at;
  at += b_x;
  // literals and state, in parts of both
  const int parts = pool_parts(4 * L + 8 * (n + 2 * m));
  pool_run(parts, [&](int i) {
    const int64_t N = n + 2 * m;
    const int64_t l0 = L * i / parts, l1 = L * (i + 1) / parts, e0 = N * i / parts,
                  e1 = N * (i + 1) / parts;
    std::memcpy(lit_at + 4 * l0, lits + l0, (size_t)(l1 - l0) * 4);
    if (prec_ == DMM_FP64) {
      std::memcpy(x_at + 8 * e0, x0 + e0, (size_t)(e1 - e0) * 8);
    } else {
      float* o = reinterpret_cast<float*>(x_at);
      for (int64_t e = e0; e < e1; e++) o[e] = (float)x0[e];
    }
  });
  std::memcpy(A.host + (int64_t)A.count * sizeof(AdmitRec), &R, sizeof R);
  A.count++;
  A.used = at - head;
  *done = true;
  return DMM_OK;
}

dmm_status Pack::flush_adds() {
  AdmitBlock& A = admit_[admit_cur_];
  if (A.count == 0) return DMM_OK;
  const int64_t head = admit_head();
  const int count = A.count;
  const int64_t used = A.used;
  A.count = 0;
  A.used = 0;
  DMM_CUDA(cudaMemcpyAsync(A.dev, A.host, (size_t)count * sizeof(AdmitRec), cudaMemcpyHostToDevice,
                           stream_));
  DMM_CUDA(cudaMemcpyAsync(A.dev + head, A.host + head, (size_t)used, cudaMemcpyHostToDevice, stream_));
  const int smem = (kAdmitVars + (kAdmitThreads / 32) * kSortCap) * 4;
  const AdmitRec* recs = reinterpret_cast<const AdmitRec*>(A.dev);
  if (prec_ == DMM_FP64) {
    DMM_CUDA(allow_smem((const void*)k_admit<double>, smem));
    k_admit<double><<<count, kAdmitThreads, smem, stream_>>>(
        recs, A.dev, inst_d_, ctrl_d_, lit_, vslot_, upos_, vend_, coff_, unit_,
        static_cast<double*>(cand_), static_cast<double*>(Xs_), static_cast<double*>(Xl_), active_d_,
        longv_d_, ring_tail_d_ + 2, longv_cap_);
  } else {
    DMM_CUDA(allow_smem((const void*)k_admit<float>, smem));
    k_admit<float><<<count, kAdmitThreads, smem, stream_>>>(
        recs, A.dev, inst_d_, ctrl_d_, lit_, vslot_, upos_, vend_, coff_, unit_,
        static_cast<float*>(cand_), static_cast<float*>(Xs_), static_cast<float*>(Xl_), active_d_,
        longv_d_, ring_tail_d_ + 2, longv_cap_);
  }
  DMM_CUDA(cudaGetLastError());
  DMM_CUDA(cudaEventRecord(A.sent, stream_));
  A.busy = true;
  admit_cur_ ^= 1;
  long_pending_ = true;
  return DMM_OK;
}

dmm_status Pack::add(const int32_t* lits, const int64_t* clause_off, int32_t n, int32_t m,
                     const dmm_params* p, const double* alpha_cm, int32_t max_steps,
                     int32_t* idx_out, const double* x0, bool device_literal_check) {
  DMM_TRY(validate_shape(lits, clause_off, n, m));
  if (alpha_cm && !with_alpha_cm_) {
    set_error("this pack was created without per-clause alpha storage");
    return DMM_ERR_ARG;
  }
  DMM_CUDA(cudaSetDevice(dev_));
  int32_t idx = -1;
  for (int32_t i = 0; i < (int32_t)live_.size(); i++)
    if (!live_[i]) {
      idx = i;
      break;
    }
  if (idx < 0) {
    set_error("pack is full (%d instances)", caps_.insts);
    return DMM_ERR_BUDGET;
  }
  const int64_t L = clause_off[m];
  const int64_t var0 = var_alloc_.alloc(n);
  const int64_t cls0 = var0 < 0 ? -1 : cls_alloc_.alloc(m);
  const int64_t slot0 = cls0 < 0 ? -1 : slot_alloc_.alloc(L);
  if (var0 < 0 || cls0 < 0 || slot0 < 0) {
    if (var0 >= 0) var_alloc_.free(var0, n);
    if (cls0 >= 0) cls_alloc_.free(cls0, m);
    set_error("pack capacity exhausted (n=%d m=%d literals=%lld)", n, m, (long long)L);
    return DMM_ERR_BUDGET;
  }
  // small formulas with an initial state are laid aside and unpacked many at a time
  if (x0 && !alpha_cm && !device_literal_check && !admit_off_ && n <= kAdmitVars && L <= kAdmitSlots) {
    bool k3 = false, units = true, done = false;
    dmm_status st = validate_formula(lits, clause_off, n, m, &k3, &units, true);
    InstDesc I{};
    I.n = n;
    I.m = m;
    I.var0 = var0;
    I.cls0 = cls0;
    I.slot0 = slot0;
    I.nslots = (int32_t)L;
    I.k3 = k3 ? 1 : 0;
    I.max_steps = max_steps;
    fill_params(I, p);
    if (st == DMM_OK) st = stage_add(I, idx, lits, clause_off, units, x0, &done);
    if (st != DMM_OK) {
      var_alloc_.free(var0, n);
      cls_alloc_.free(cls0, m);
      slot_alloc_.free(slot0, L);
      return st;
    }
    if (done) {
      inst_h_[idx] = I;
      live_[idx] = 1;
      add_serial_[idx] = ++add_counter_;
      if (!fixed_grid_) graph_stale_ = true;
      *idx_out = idx;
      return DMM_OK;
    }
  }
  // the literal upload runs while the host checks the clauses (and literals)
  if (L > 0)
    DMM_CUDA(cudaMemcpyAsync(lit_ + slot0, lits, (size_t)L * 4, cudaMemcpyHostToDevice, stream_));
  InstDesc I{};
  I.n = n;
  I.m = m;
  I.var0 = var0;
  I.cls0 = cls0;
  I.slot0 = slot0;
  I.nslots = (int32_t)L;
  // with the literals checked on the device the occurrence lists need nothing from the
  // host pass: they build while the host checks the clause offsets
  if (device_literal_check) DMM_TRY(build_csr(I, lits));
  bool k3 = false, units = true;
  const dmm_status vst =
      validate_formula(lits, clause_off, n, m, &k3, &units, !device_literal_check);
  if (vst != DMM_OK) {
    cudaStreamSynchronize(stream_);
    var_alloc_.free(var0, n);
    cls_alloc_.free(cls0, m);
    slot_alloc_.free(slot0, L);
    return vst;
  }
  I.k3 = k3 ? 1 : 0;
  I.has_alpha_cm = alpha_cm ? 1 : 0;
  I.max_steps = max_steps;
  fill_params(I, p);
  std::vector<int32_t> coff_local;
  if (!k3 && m > 0) {
    coff_local.resize(m);
    for (int32_t c = 0; c < m; c++) coff_local[c] = (int32_t)clause_off[c];
    DMM_CUDA(cudaMemcpyAsync(coff_ + cls0, coff_local.data(), (size_t)m * 4,
                             cudaMemcpyHostToDevice, stream_));
  }
  // unit clauses (dynex.cc:2459-2469: the last unit clause of a variable wins)
  if (units) {
    unit_h_.assign(n, 0);
    for (int32_t c = 0; c < m; c++)
      if (clause_off[c + 1] - clause_off[c] == 1) {
        const int32_t l = lits[clause_off[c]];
        if (l == 0 || l > n || l < -n) continue;  // unchecked literal: the device check reports it
        unit_h_[std::abs(l) - 1] = l > 0 ? 1 : -1;
      }
    DMM_CUDA(cudaMemcpyAsync(unit_ + var0, unit_h_.data(), n, cudaMemcpyHostToDevice, stream_));
  } else {
    DMM_CUDA(cudaMemsetAsync(unit_ + var0, 0, n, stream_));
  }
  if (alpha_cm) {
    if (prec_ == DMM_FP64)
      DMM_TRY(upload_alpha(static_cast<double*>(alpha_cm_) + cls0, alpha_cm, m, stream_));
    else
      DMM_TRY(upload_alpha(static_cast<float*>(alpha_cm_) + cls0, alpha_cm, m, stream_));
  }
  if (!device_literal_check) DMM_TRY(build_csr(I, lits));
  inst_h_[idx] = I;
  live_[idx] = 1;
  add_serial_[idx] = ++add_counter_;
  DMM_TRY(upload_desc(idx));
  InstCtrl c{};
  c.done = DMM_CANCELLED;  // not runnable until a state is set
  c.best_loc = m;
  c.loc = m;
  c.solved_step = -1;
  c.solved_t = -1.0;
  c.h_state = 0.125;
  if (x0) {
    // runnable at once: the state set_state would upload, without reading the control
    // record back (it is the one written here)
    const dmm_status st = upload_state(I, x0);
    if (st != DMM_OK) {
      write_ctrl(idx, c);
      var_alloc_.free(var0, n);
      cls_alloc_.free(cls0, m);
      slot_alloc_.free(slot0, L);
      live_[idx] = 0;
      return st;
    }
    DMM_TRY(write_ctrl(idx, running_ctrl(I, 0.0, 0)));
    DMM_TRY(add_active(+1));
  } else {
    DMM_TRY(write_ctrl(idx, c));
  }
  if (!fixed_grid_) graph_stale_ = true;
  if (page_locked(lits) || page_locked(x0)) DMM_CUDA(cudaStreamSynchronize(stream_));
  *idx_out = idx;
  return DMM_OK;
}

dmm_status Pack::remove(int32_t idx) {
  if (!live(idx)) {
    set_error("instance %d is not live", idx);
    return DMM_ERR_ARG;
  }
  InstCtrl c;
  DMM_TRY(read_ctrl(idx, &c));
  if (c.done == 0) {
    DMM_TRY(add_active(-1));
    c.done = DMM_CANCELLED;
    DMM_TRY(write_ctrl(idx, c));
  }
  const InstDesc& I = inst_h_[idx];
  var_alloc_.free(I.var0, I.n);
  cls_alloc_.free(I.cls0, I.m);
  slot_alloc_.free(I.slot0, I.nslots);
  live_[idx] = 0;
  if (!fixed_grid_) graph_stale_ = true;
  return DMM_OK;
}

dmm_status Pack::set_params(int32_t idx, const dmm_params* p, const double* alpha_cm) {
  if (!live(idx)) return DMM_ERR_ARG;
  if (alpha_cm && !with_alpha_cm_) {
    set_error("this pack was created without per-clause alpha storage");
    return DMM_ERR_ARG;
  }
  InstDesc& I = inst_h_[idx];
  fill_params(I, p);
  I.has_alpha_cm = alpha_cm ? 1 : 0;
  if (alpha_cm) {
    if (prec_ == DMM_FP64)
      DMM_TRY(upload_alpha(static_cast<double*>(alpha_cm_) + I.cls0, alpha_cm, I.m, stream_));
    else
      DMM_TRY(upload_alpha(static_cast<float*>(alpha_cm_) + I.cls0, alpha_cm, I.m, stream_));
  }
  DMM_TRY(upload_desc(idx));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

dmm_status Pack::set_max_steps(int32_t idx, int32_t max_steps) {
  if (!live(idx)) return DMM_ERR_ARG;
  inst_h_[idx].max_steps = max_steps;
  DMM_TRY(upload_desc(idx));
  return DMM_OK;
}

dmm_status Pack::set_state(int32_t idx, const double* x) {
  return set_state_at(idx, x, 0.0, 0, false);
}

dmm_status Pack::set_state_at(int32_t idx, const double* x, double t, int32_t step,
                              bool keep_best) {
  if (!live(idx) || !x || step < 0) {
    set_error("set_state: bad instance or null state");
    return DMM_ERR_ARG;
  }
  const InstDesc& I = inst_h_[idx];
  DMM_TRY(flush_adds());
  DMM_TRY(upload_state(I, x));
  k_restart<<<1, 1, 0, stream_>>>(ctrl_d_ + idx, running_ctrl(I, t, step), keep_best ? 1 : 0,
                                  active_d_);
  DMM_CUDA(cudaGetLastError());
  if (page_locked(x)) DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

dmm_status Pack::pinned() {
  if (!pinned_) DMM_CUDA(pinned_alloc(&pinned_, 4096));
  return DMM_OK;
}

dmm_status Pack::upload_doubles(double* dst, const double* src, int64_t count) {
  if (count <= kDirectCopy || page_locked(src))
    DMM_CUDA(cudaMemcpyAsync(dst, src, count * sizeof(double), cudaMemcpyHostToDevice, stream_));
  else
    DMM_CUDA(XferLease()->upload<double>(dst, src, count, stream_));
  return DMM_OK;
}

template <class T>
dmm_status Pack::download_state(double* dst, const T* src, int64_t count) {
  if (sizeof(T) == 8 && (count <= kDirectCopy || page_locked(dst))) {
    DMM_CUDA(cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyDeviceToHost, stream_));
    DMM_CUDA(cudaStreamSynchronize(stream_));
  } else {
    DMM_CUDA(XferLease()->download<T>(dst, src, count, stream_));
  }
  return DMM_OK;
}

dmm_status Pack::upload_state(const InstDesc& I, const double* x) {
  const int64_t n = I.n, m = I.m, N = n + 2 * m;
  if (N > kDirectCopy && !page_locked(x)) {  // rounded on the host, straight to its place
    XferLease xfer;
    if (prec_ == DMM_FP64) {
      DMM_CUDA(xfer->upload<double>(static_cast<double*>(cand_) + I.var0, x, n, stream_));
      DMM_CUDA(xfer->upload<double>(static_cast<double*>(Xs_) + I.cls0, x + n, m, stream_));
      DMM_CUDA(xfer->upload<double>(static_cast<double*>(Xl_) + I.cls0, x + n + m, m, stream_));
    } else {
      DMM_CUDA(xfer->upload<float>(static_cast<float*>(cand_) + I.var0, x, n, stream_));
      DMM_CUDA(xfer->upload<float>(static_cast<float*>(Xs_) + I.cls0, x + n, m, stream_));
      DMM_CUDA(xfer->upload<float>(static_cast<float*>(Xl_) + I.cls0, x + n + m, m, stream_));
    }
    return DMM_OK;
  }
  DMM_TRY(ensure_stage(N));
  DMM_CUDA(cudaMemcpyAsync(stage_, x, N * sizeof(double), cudaMemcpyHostToDevice, stream_));
  if (prec_ == DMM_FP64) {
    double* V = static_cast<double*>(cand_) + I.var0;
    k_set_state<double><<<blocks_for(N), kThreads, 0, stream_>>>(
        stage_, I.n, I.m, V, static_cast<double*>(Xs_) + I.cls0, static_cast<double*>(Xl_) + I.cls0);
  } else {
    float* V = static_cast<float*>(cand_) + I.var0;
    k_set_state<float><<<blocks_for(N), kThreads, 0, stream_>>>(
        stage_, I.n, I.m, V, static_cast<float*>(Xs_) + I.cls0, static_cast<float*>(Xl_) + I.cls0);
  }
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

InstCtrl Pack::running_ctrl(const InstDesc& I, double t, int32_t step) {
  InstCtrl c{};
  c.done = 0;
  c.step = step;
  c.t = t;
  c.loc = I.m;
  c.best_loc = I.m;
  c.best_t = 0.0;
  c.solved_step = -1;
  c.solved_t = -1.0;
  c.h_state = 0.125;
  return c;
}

dmm_status Pack::get_state(int32_t idx, double* x, double* t) {
  if (!live(idx)) return DMM_ERR_ARG;
  DMM_TRY(flush_adds());
  const InstDesc& I = inst_h_[idx];
  const int64_t N = (int64_t)I.n + 2 * (int64_t)I.m;
  DMM_TRY(ensure_stage(N));
  DMM_TRY(pinned());
  InstCtrl* c = reinterpret_cast<InstCtrl*>(pinned_ + 64);
  if (t) DMM_CUDA(cudaMemcpyAsync(c, ctrl_d_ + idx, sizeof(InstCtrl), cudaMemcpyDeviceToHost, stream_));
  if (prec_ == DMM_FP64) {
    k_get_state<double><<<blocks_for(N), kThreads, 0, stream_>>>(
        inst_d_, ctrl_d_, idx, static_cast<double*>(cand_), caps_.vars, static_cast<double*>(Xs_),
        static_cast<double*>(Xl_), static_cast<double*>(Cp_), static_cast<double*>(alpha_cm_), stage_);
    DMM_CUDA(cudaGetLastError());
    if (x) DMM_TRY(download_state(x, stage_, N));
  } else {
    float* out = reinterpret_cast<float*>(stage_);
    k_get_state<float><<<blocks_for(N), kThreads, 0, stream_>>>(
        inst_d_, ctrl_d_, idx, static_cast<float*>(cand_), caps_.vars, static_cast<float*>(Xs_),
        static_cast<float*>(Xl_), static_cast<float*>(Cp_), static_cast<float*>(alpha_cm_), out);
    DMM_CUDA(cudaGetLastError());
    if (x) DMM_TRY(download_state(x, out, N));
  }
  if (!x) DMM_CUDA(cudaStreamSynchronize(stream_));
  if (t) *t = c->t;
  return DMM_OK;
}

template <class T>
void Pack::fill_view(void* vv) const {
  PackView<T>& v = *static_cast<PackView<T>*>(vv);
  v.Xs = static_cast<T*>(Xs_);
  v.Xl = static_cast<T*>(Xl_);
  v.Cp = static_cast<T*>(Cp_);
  v.alpha_cm = static_cast<const T*>(alpha_cm_);
  v.coff = coff_;
  v.lit = lit_;
  v.u = static_cast<T*>(u_);
  v.vslot = vslot_;
  v.vend = vend_;
  v.cand = static_cast<T*>(cand_);
  v.var_cap = caps_.vars;
  v.unit = unit_;
  v.epart = epart_;
  v.inst = inst_d_;
  v.ctrl = ctrl_d_;
  v.ctiles = use_aux_ ? aux_ctiles_d_ : ctiles_d_;
  v.vtiles = use_aux_ ? aux_vtiles_d_ : vtiles_d_;
  v.ntiles = use_aux_ ? ntiles_d_ + 2 : ntiles_d_;
  v.queue = queue_d_;
  v.active = active_d_;
  v.ring = ring_d_;
  v.ring_tail = ring_tail_d_;
  v.ring_cap = caps_.insts;
  v.live = live_d_;
  v.live0 = live0_;
  v.nlive = misc_d_;
  v.acc2 = reinterpret_cast<StepAcc*>(misc_d_ + kMiscAcc2);
  // tile paths: slot-major unless asked (measured faster there); the one-block-per-formula
  // kernel switches to variable-major by default in launch_inst
  v.upos = tun_.u_layout == 2 ? upos_ : nullptr;
  v.xdlist = xp_active_ ? static_cast<const int32_t*>(xbuf_[kXpDlist]) : nullptr;
  v.xdoff = static_cast<const int32_t*>(xbuf_[kXpDoff]);
  v.xllit = static_cast<const int16_t*>(xbuf_[kXpLlit]);
  v.xspos = static_cast<const uint16_t*>(xbuf_[kXpSpos]);
  v.ux = static_cast<T*>(xbuf_[kXpUx]);
  v.xubase = static_cast<const int32_t*>(xbuf_[kXpUbase]);
  v.xboff = static_cast<const int32_t*>(xbuf_[kXpBoff]);
  v.xsrc8 = static_cast<const int32_t*>(xbuf_[kXpSrc8]);
  v.xdst = static_cast<const uint16_t*>(xbuf_[kXpDst]);
  v.xsv_cap = xsv_cap_;
  v.xbk_cap = xbk_cap_;
  v.xtv_cap = xtv_cap_;
  v.xst_cap = xst_cap_;
  v.xl2_plain = tun_.l2_policy & 1;
  v.xprefetch = (tun_.l2_policy & 2) != 0;
  v.barrier_extra = barrier_extra_;
  v.trace = trace_on_ ? trace_ : nullptr;
  v.trace_steps = trace_on_ ? trace_steps_ : 0;
}

dmm_status Pack::enqueue_clause() {
  if (prec_ == DMM_FP64) {
    PackView<double> v;
    fill_view<double>(&v);
    k_clause<double, false><<<grid_c_, kThreads, 0, stream_>>>(v);
  } else {
    PackView<float> v;
    fill_view<float>(&v);
    k_clause<float, true><<<grid_c_, kThreads, 0, stream_>>>(v);
  }
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

template <int MODE>
static void launch_var_f32(int G, int grid, cudaStream_t s, const PackView<float>& v, double* dv) {
  switch (G) {
    case 1: k_var<float, 1, false, MODE><<<grid, kThreads, 0, s>>>(v, dv); break;
    case 2: k_var<float, 2, false, MODE><<<grid, kThreads, 0, s>>>(v, dv); break;
    case 4: k_var<float, 4, false, MODE><<<grid, kThreads, 0, s>>>(v, dv); break;
    case 8: k_var<float, 8, false, MODE><<<grid, kThreads, 0, s>>>(v, dv); break;
    case 16: k_var<float, 16, false, MODE><<<grid, kThreads, 0, s>>>(v, dv); break;
    default: k_var<float, 32, false, MODE><<<grid, kThreads, 0, s>>>(v, dv); break;
  }
}

dmm_status Pack::enqueue_var(bool rhs_only, void* dv_out) {
  double* dv = static_cast<double*>(dv_out);
  if (prec_ == DMM_FP64) {
    PackView<double> v;
    fill_view<double>(&v);
    if (rhs_only)
      k_var<double, 32, true, 1><<<grid_v_, kThreads, 0, stream_>>>(v, dv);
    else
      k_var<double, 32, true, 0><<<grid_v_, kThreads, 0, stream_>>>(v, dv);
  } else {
    PackView<float> v;
    fill_view<float>(&v);
    if (rhs_only)
      launch_var_f32<1>(tun_.var_group, grid_v_, stream_, v, dv);
    else
      launch_var_f32<0>(tun_.var_group, grid_v_, stream_, v, dv);
  }
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

dmm_status Pack::enqueue_step(bool rhs_only, void* dv_out) {
  DMM_TRY(enqueue_clause());
  DMM_TRY(enqueue_var(rhs_only, dv_out));
  return DMM_OK;
}

// Blocks of a kernel that an SM holds at once, 0 when it cannot hold one: a cooperative launch
// would be refused.  cap: the kernel's largest dynamic shared memory (allow_smem)
static int resident_blocks(const void* fn, int threads, size_t smem, int cap) {
  int b = 0;
  if (allow_smem(fn, cap) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return b;
}

static int occupancy_blocks(const void* fn, int threads) {
  int b = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, threads, 0) != cudaSuccess) {
    cudaGetLastError();
    b = 4;
  }
  return std::max(1, b);
}

// ONE: single-formula form
template <bool ONE>
static const void* persist_fn_x(dmm_precision prec, int G) {
  if (prec == DMM_FP64)
    return (const void*)k_persist<double, 32, true, false, kPersistThreads64, ONE>;
  switch (G) {
    case 1: return (const void*)k_persist<float, 1, false, true, kPersistThreads, ONE>;
    case 2: return (const void*)k_persist<float, 2, false, true, kPersistThreads, ONE>;
    case 4: return (const void*)k_persist<float, 4, false, true, kPersistThreads, ONE>;
    case 8: return (const void*)k_persist<float, 8, false, true, kPersistThreads, ONE>;
    case 16: return (const void*)k_persist<float, 16, false, true, kPersistThreads, ONE>;
    default: return (const void*)k_persist<float, 32, false, true, kPersistThreads, ONE>;
  }
}

// the staged form (FP32, single formula); mt: several tiles per block
template <bool MT>
static const void* staged_fn_x(int G) {
  switch (G) {
    case 1: return (const void*)k_staged<1, kStagedThreads, MT>;
    case 2: return (const void*)k_staged<2, kStagedThreads, MT>;
    case 4: return (const void*)k_staged<4, kStagedThreads, MT>;
    case 8: return (const void*)k_staged<8, kStagedThreads, MT>;
    case 16: return (const void*)k_staged<16, kStagedThreads, MT>;
    default: return (const void*)k_staged<32, kStagedThreads, MT>;
  }
}
static const void* staged_fn(int G, bool mt) {
  return mt ? staged_fn_x<true>(G) : staged_fn_x<false>(G);
}

// Estimated microseconds per step, fitted to single formulas of 500 to 30,000 variables at 4.3
// and 8 clauses per variable: the cluster form by a block's clauses (FP32 3.1 us at 250 and
// 4.8 at 1,000; FP64 4.7 and 9.9), in waves when the clusters do not all fit at once (blocks of a
// cluster share a GPC: few clusters of 16 are resident together; 16 formulas of n = 8,000 at 4.3,
// FP32: 28.2 us in clusters of 16, 26.8 in the tile forms, 15.8 in the resident grid form); the
// resident grid form by a block's share of the clauses (FP32 5.1 us at 54, 9.8 at 1,600; FP64
// 7.5 and 15.9).  The two meet at about 18,000 clauses (FP32) and 13,000 (FP64) for one formula.
// Clauses of other lengths have their own fits, at 3.5 and 6.6 clauses per variable (cluster
// FP32 4.2 us at 206 and 7.2 at 825, FP64 6.1 and, at 619, 9.5; grid FP32 6.2 at 67 and 11.8 at
// 1,338, FP64 9.2 and 17.0): a warp of the cluster form waits for its longest clause, the grid
// form orders them.  These meet at about 10,000 and 9,400 clauses (cluster / grid at 13,200:
// FP32 7.2 / 6.3; at 10,500: FP64 10.6 / 8.8).
double Pack::cluster_step_us() const {
  const bool fp64 = prec_ == DMM_FP64;
  double blocks = 0, full = 0, most = 0;
  for (const ClusterLaunch& L : clusters_) {
    blocks += (double)L.R * L.count;
    full += (double)L.count / L.resident;
    const double us = L.general ? (fp64 ? 4.2 + 8.2e-3 * L.caps.tc : 2.6 + 5.6e-3 * L.caps.tc)
                                : (fp64 ? 3.6 + 5.0e-3 * L.caps.tc : 2.6 + 2.2e-3 * L.caps.tc);
    most = std::max(most, us);
  }
  return std::ceil(std::max(blocks / sms_, full)) * most;
}

double Pack::grid_step_us(const std::vector<int32_t>& list) const {
  if ((int)list.size() > sms_) return 1e9;
  const bool fp64 = prec_ == DMM_FP64;
  double total = 0, most = 0;
  bool general = false;
  for (int32_t i : list) {
    total += inst_h_[i].m;
    most = std::max(most, (double)inst_h_[i].m);
    general |= inst_h_[i].k3 == 0;
  }
  const double share = std::max(total / sms_, most / (sms_ - (double)list.size() + 1));
  return general ? (fp64 ? 8.6 + 6.3e-3 * share : 5.9 + 4.3e-3 * share)
                 : (fp64 ? 7.0 + 5.2e-3 * share : 4.9 + 3.2e-3 * share);
}

// The formulas of `all` that are not among `some`.
std::vector<int32_t> Pack::without(const std::vector<int32_t>& all,
                                   const std::vector<int32_t>& some) const {
  std::vector<char> taken(live_.size(), 0);
  for (int32_t i : some) taken[i] = 1;
  std::vector<int32_t> rest;
  for (int32_t i : all)
    if (!taken[i]) rest.push_back(i);
  return rest;
}

// Estimated microseconds per step of several formulas in the tile forms, fitted to some 560 batches
// of 2 to 148 formulas of 50 to 400,000 variables at 4.3 and 8 clauses per variable (error 6 to 7 %),
// other clause lengths at 6.6 (7 %): waves of clause and variable tiles, and what they hold.
double Pack::tile_step_us(const std::vector<int32_t>& list) const {
  const bool fp64 = prec_ == DMM_FP64;
  const int block = persist_threads(prec_);
  double ct = 0, vt = 0, m = 0;
  bool general = false;
  for (int32_t i : list) {
    ct += (inst_h_[i].m + 4 * block - 1) / (4 * block);
    vt += (inst_h_[i].n + block - 1) / block;
    m += 1e-6 * inst_h_[i].m;
    general |= inst_h_[i].k3 == 0;
  }
  ct /= sms_;
  vt /= sms_;
  if (list.empty()) return 0.0;
  // (one formula: its tiles are balanced over the grid)
  if (list.size() == 1)
    return general ? (fp64 ? 13 + 94 * m : 11 + 66 * m) : (fp64 ? 9 + 50 * m : 8 + 39 * m);
  const double c = 0.01 * (double)list.size(), cw = std::ceil(ct), vw = std::ceil(vt);
  if (general)
    return fp64 ? 2.2 + 12.7 * cw + 17.5 * vw + 53.8 * m - 23.2 * c
                : 7.9 + 14.2 * cw + 15.1 * vw + 35.9 * m - 15.3 * c;
  return fp64 ? -0.6 + 5.6 * cw + 13.0 * vw + 4.5 * ct - 12.2 * vt + 35.1 * m - 7.4 * c
              : 7.0 + 5.7 * cw + 12.9 * vw + 14.1 * ct - 10.2 * vt + 1.9 * m - 11.1 * c;
}

// Whether several formulas `all` run faster when `groups` (the formulas `list`) take the resident
// grid form and the others the tile forms after it, than all together in the tile forms: the grid
// form's step is that of its most loaded block, and the launch for the others comes on top.  The
// former by the largest share of the clauses and the tiles of a block, fitted to the same batches
// (error 10 to 13 %).  Of 413 such batches 24 were 3 to 30 % slower with the grid form wherever
// tables could be built, 3 are where this says so (us per step, grid form / tile forms: four of
// n = 60,000, FP64 at 4.3 clauses per variable, 91 / 84; 60 of 100 to 10,000, FP32, mixed lengths,
// 115 / 88; 16 of 500 to 20,000, FP32 at 8, 18 / 43).
bool Pack::grid_pays(const std::vector<int32_t>& all, const std::vector<int32_t>& list,
                     const std::vector<GridGroup>& groups) const {
  const bool fp64 = prec_ == DMM_FP64;
  double share = 0, tiles = 0;
  bool general = false;
  for (const GridGroup& g : groups) {
    share = std::max(share, 1e-3 * g.TC * g.kc);
    tiles = std::max(tiles, (double)(g.kc + g.kv));
    general |= g.k3 == 0;
  }
  const double grid = general ? (fp64 ? 2.4 + 8.7 * share + 4.7 * tiles : -13.3 + 6.3 * share + 9.0 * tiles)
                              : (fp64 ? 2.9 + 4.3 * share + 3.7 * tiles : -3.4 + 2.0 * share + 6.0 * tiles);
  return grid + tile_step_us(without(all, list)) < tile_step_us(all);
}

dmm_status Pack::grid_buffer(int which, int64_t bytes) {
  bytes = std::max<int64_t>(bytes, 16);
  if (bytes <= gbuf_cap_[which]) return DMM_OK;
  if (gbuf_[which]) retire(gbuf_[which]);
  gbuf_[which] = nullptr;
  gbuf_cap_[which] = 0;
  DMM_CUDA(dev_alloc(&gbuf_[which], bytes));
  gbuf_cap_[which] = bytes;
  return DMM_OK;
}

// Places a group's part of each table array.
void Pack::grid_place(GridGroup* g, GridSizes* z) const {
  const int kw = 16 / (int)tsize_;
  g->o_pair = z->pair;
  g->o_blk = z->blks;
  g->o_ct = z->ct;
  g->o_vt = z->vt;
  g->o_list = z->lst;
  g->o_slot = z->slot;
  g->o_ux = z->ux;
  g->o_word = z->word;
  g->o_row = z->row;
  g->o_push = z->push;
  g->o_bb = z->bb;
  g->o_var = z->var;
  g->o_cls = z->cls;
  const int64_t pairs = (int64_t)g->nct * g->nvt, Ls = RangeAlloc::round(g->L);
  const int64_t uxn = RangeAlloc::round(g->L + (g->pad - 1) * pairs + 32);
  z->pair += pairs;
  z->blks += std::max(g->NL, g->B) + 1;
  z->ct += std::max(g->nct, g->B) + 1;
  z->vt += g->nvt + 1;
  const int64_t chunks = (int64_t)g->NL * g->B;  // each padded to whole words
  const int64_t ent = RangeAlloc::round(std::min<int64_t>(g->L, (int64_t)g->NL * g->n) +
                                        (kw - 1) * chunks + 4 * g->NL);
  z->lst += ent;
  z->slot += Ls;
  z->ux += uxn;
  z->word += uxn / kw;
  z->row += (int64_t)g->nvt * g->TVr * 32;
  z->push += ent / kw + 32;
  z->bb += (int64_t)g->NL * (g->B + 1);
  z->var += RangeAlloc::round(g->n);
  z->cls += RangeAlloc::round(g->m);
  z->max_n = std::max(z->max_n, g->n);
  z->max_nct = std::max(z->max_nct, g->nct);
  z->max_nvt = std::max(z->max_nvt, g->nvt);
  z->max_rows = std::max(z->max_rows, g->nvt + g->B);
}

// Gives the tables back after an allocation failed, so that the forms that need none (or less)
// can run.
void Pack::drop_grid_tables() {
  cudaGetLastError();
  clear_error();
  for (int q = 0; q < kGrBufs; q++) {
    if (gbuf_[q]) retire(gbuf_[q]);
    gbuf_[q] = nullptr;
    gbuf_cap_[q] = 0;
  }
}

// Allocates and builds the tables (map: group of every variable list; nblocks: blocks of the
// launch); out: what grid_build reports per group.
dmm_status Pack::grid_tables(const std::vector<GridGroup>& groups, const std::vector<int32_t>& map,
                             int nblocks, const GridSizes& z, bool stream, GridTables* tables,
                             std::vector<int32_t>* out) {
  const int T = (int)tsize_, copies = stream ? 1 : 2;
  const int64_t G = (int64_t)groups.size();
  int64_t bytes[kGrBufs] = {};
  bytes[kGrGroups] = G * (int64_t)sizeof(GridGroup);
  bytes[kGrBlk] = (int64_t)map.size() * 4;
  bytes[kGrDlist] = z.lst * 4;
  bytes[kGrDinfo] = z.blks * 8;
  bytes[kGrLlit] = z.slot * 2;
  bytes[kGrSpos] = z.slot * 2;
  bytes[kGrWdst] = z.word * 4;
  bytes[kGrWoff] = z.ct * 4;
  bytes[kGrBoff] = z.vt * 4;
  bytes[kGrRows] = z.row * 2;
  bytes[kGrIdx] = z.slot * 2;
  const int kw = 16 / T;
  bytes[kGrSinfo] = z.blks * 8;
  bytes[kGrIds] = z.push * kw * 2;
  bytes[kGrSdst] = z.push * 4;
  bytes[kGrDlp] = bytes[kGrPoff] = z.bb * 4;
  const bool ordered = prec_ == DMM_FP64 && !stream;
  if (ordered) bytes[kGrPos] = bytes[kGrPerm] = z.var * 2;
  bool general = false;
  for (const GridGroup& g : groups) general |= !stream && g.k3 == 0;
  if (general) bytes[kGrCord] = z.cls * 2;
  bytes[kGrUx] = copies * z.ux * T;
  bytes[kGrInbox] = copies * z.lst * T;
  bytes[kGrCnt] = bytes[kGrSb] = bytes[kGrBt] = z.pair * 4;
  bytes[kGrSt] = z.ct * 4;
  bytes[kGrDcnt] = z.blks * 4;
  bytes[kGrDlo] = z.bb * 4;
  bytes[kGrOut] = G * kGridOut * 4;
  bytes[kGrSync] = G * kGridSyncBytes;
  bytes[kGrEpart] = (int64_t)nblocks * 16;
  bytes[kGrBtot] = z.vt * 4;
  bytes[kGrPtot] = z.blks * 4;
  if (stream) bytes[kGrDv] = caps_.vars * T;
  for (int q = 0; q < kGrBufs; q++)
    if (bytes[q] > 0) DMM_TRY(grid_buffer(q, bytes[q]));
  GridTables t{};
  t.dlist = static_cast<int32_t*>(gbuf_[kGrDlist]);
  t.dinfo = static_cast<int2*>(gbuf_[kGrDinfo]);
  t.llit = static_cast<int16_t*>(gbuf_[kGrLlit]);
  t.spos = static_cast<uint16_t*>(gbuf_[kGrSpos]);
  t.wdst = static_cast<uint32_t*>(gbuf_[kGrWdst]);
  t.woff = static_cast<int32_t*>(gbuf_[kGrWoff]);
  t.boff = static_cast<int32_t*>(gbuf_[kGrBoff]);
  t.rows = static_cast<uint16_t*>(gbuf_[kGrRows]);
  t.idx = static_cast<uint16_t*>(gbuf_[kGrIdx]);
  t.sinfo = static_cast<int2*>(gbuf_[kGrSinfo]);
  t.ids = static_cast<uint16_t*>(gbuf_[kGrIds]);
  t.sdst = static_cast<uint32_t*>(gbuf_[kGrSdst]);
  t.pos = ordered ? static_cast<uint16_t*>(gbuf_[kGrPos]) : nullptr;
  t.cord = general ? static_cast<uint16_t*>(gbuf_[kGrCord]) : nullptr;
  t.perm = ordered ? static_cast<uint16_t*>(gbuf_[kGrPerm]) : nullptr;
  t.dlp = static_cast<int32_t*>(gbuf_[kGrDlp]);
  t.poff = static_cast<int32_t*>(gbuf_[kGrPoff]);
  t.ux = gbuf_[kGrUx];
  t.inbox = gbuf_[kGrInbox];
  t.ux_len = z.ux;
  t.inbox_len = z.lst;
  t.cnt = static_cast<int32_t*>(gbuf_[kGrCnt]);
  t.sb = static_cast<int32_t*>(gbuf_[kGrSb]);
  t.bt = static_cast<int32_t*>(gbuf_[kGrBt]);
  t.st = static_cast<int32_t*>(gbuf_[kGrSt]);
  t.dcnt = static_cast<int32_t*>(gbuf_[kGrDcnt]);
  t.dlo = static_cast<int32_t*>(gbuf_[kGrDlo]);
  t.btot = static_cast<int32_t*>(gbuf_[kGrBtot]);
  t.ptot = static_cast<int32_t*>(gbuf_[kGrPtot]);
  t.out = static_cast<int32_t*>(gbuf_[kGrOut]);
  DMM_CUDA(cudaMemcpyAsync(gbuf_[kGrGroups], groups.data(), (size_t)bytes[kGrGroups],
                           cudaMemcpyHostToDevice, stream_));
  DMM_CUDA(cudaMemcpyAsync(gbuf_[kGrBlk], map.data(), (size_t)bytes[kGrBlk], cudaMemcpyHostToDevice,
                           stream_));
  DMM_CUDA(cudaMemsetAsync(t.rows, 0, (size_t)bytes[kGrRows], stream_));
  DMM_CUDA(grid_build(static_cast<const GridGroup*>(gbuf_[kGrGroups]),
                      static_cast<const int32_t*>(gbuf_[kGrBlk]), (int)G, (int)map.size(), z.max_n,
                      z.max_nct, z.max_nvt, z.max_rows, lit_, upos_, vend_, coff_, t, prec_ == DMM_FP64, stream_));
  out->resize((size_t)(G * kGridOut));
  DMM_CUDA(cudaMemcpyAsync(out->data(), t.out, (size_t)bytes[kGrOut], cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  *tables = t;
  return DMM_OK;
}

dmm_status Pack::plan_stream(int32_t idx, bool* ok) {
  *ok = false;
  const InstDesc& I = inst_h_[idx];
  // chunks of whole 32-byte sectors: a sector written by two blocks in halves is filled from
  // memory when the buckets exceed the L2
  constexpr int kw = 4, pad = 8;
  const int B = sms_;
  if (I.m <= 0 || I.nslots <= 0) return DMM_OK;
  int kc_min = 1, kv_min = 1;
  for (int round = 0; round < 4; round++) {
    // fewest tiles per block whose lists, areas and buckets fit
    const double n = I.n, L = I.nslots;
    int kc = 0, kv = 0;
    for (int sum = kc_min + kv_min; sum <= 128 && !kc; sum++)
      for (int c = kc_min; c <= sum - kv_min && !kc; c++) {
        const int v = sum - c;
        const double Lt = L / ((double)B * c);
        const double dl = n * (1.0 - std::exp(-Lt / n)) * 1.02 + 0.5 * kw * B + 16;
        const double st = Lt * 1.02 + 0.5 * pad * B * v + 64;
        const double bk = L / ((double)B * v) * 1.06 + 0.5 * pad * B * c + 64;
        const double tv = n / B + 8 * v;
        if (dl > kGridMaxDistinct || st > 65000 || bk > 65000 || tv > 65000) continue;
        if (stream_shape((int)dl, (int)st, (int)bk, (int)tv).total > kStreamSmemMax) continue;
        kc = c;
        kv = v;
      }
    if (!kc) return DMM_OK;
    GridGroup g{};
    g.inst = idx;
    g.B = B;
    g.kc = kc;
    g.kv = kv;
    g.n = I.n;
    g.m = I.m;
    g.L = I.nslots;
    g.k3 = I.k3;
    g.var0 = I.var0;
    g.cls0 = I.cls0;
    g.slot0 = I.slot0;
    g.TC = ((I.m + B * kc - 1) / (B * kc) + 3) & ~3;
    g.TV = ((I.n + B * kv - 1) / (B * kv) + 3) & ~3;
    g.TVr = (g.TV + 31) & ~31;
    g.nct = B * kc;
    g.nvt = B * kv;
    g.lt = 1;
    g.pad = pad;
    g.NL = g.nct;
    GridSizes z;
    grid_place(&g, &z);
    if (z.ux > INT32_MAX / 2 || z.row > INT32_MAX || z.pair > (int64_t(1) << 26)) return DMM_OK;
    const std::vector<uint64_t> key{~0ull, add_serial_[idx], ((uint64_t)kc << 32) | (uint64_t)kv};
    if (key == gr_key_) {
      *ok = true;
      return DMM_OK;
    }
    gr_key_.clear();
    const std::vector<GridGroup> groups{g};
    const std::vector<int32_t> map((size_t)g.NL, 0);
    GridTables t{};
    std::vector<int32_t> out;
    const dmm_status st = grid_tables(groups, map, B, z, true, &t, &out);
    if (st == DMM_ERR_NOMEM) {
      drop_grid_tables();
      return DMM_OK;
    }
    DMM_TRY(st);
    const StreamLayout lay = stream_shape(out[1], out[2], out[3], g.TV * g.kv);
    if (out[0] == 3 || (out[0] == 0 && lay.total > kStreamSmemMax && out[3] > out[2])) {
      kv_min = kv + 1;
      continue;
    }
    if (out[0] != 0 || lay.total > kStreamSmemMax) {
      kc_min = kc + 1;
      continue;
    }
    stream_general_ = I.k3 == 0;
    if (resident_blocks(stream_kernel(stream_general_), kStreamThreads, lay.total, kStreamSmemMax) < 1)
      return DMM_OK;
    stream_layout_ = lay;
    gr_tables_ = t;
    gr_key_ = key;
    *ok = true;
    return DMM_OK;
  }
  return DMM_OK;
}

dmm_status Pack::launch_stream(int32_t nsteps) {
  PackView<float> view;
  fill_view<float>(&view);
  unsigned int* bar = reinterpret_cast<unsigned int*>(misc_d_ + kMiscLaunch);
  if (!launch_area_clean_)
    DMM_CUDA(cudaMemsetAsync(bar, 0, kLaunchAreaInts * sizeof(int32_t), stream_));
  launch_area_clean_ = true;
  const void* fn = stream_kernel(stream_general_);
  DMM_CUDA(allow_smem(fn, kStreamSmemMax));
  const void* groups = gbuf_[kGrGroups];
  void* dv = gbuf_[kGrDv];
  void* epart = gbuf_[kGrEpart];
  int* err = error_d_;
  void* args[] = {&view, &gr_tables_, &groups, &stream_layout_, &dv, &nsteps, &bar, &epart, &err};
  DMM_CUDA(cudaLaunchCooperativeKernel(fn, dim3((unsigned)sms_), dim3(kStreamThreads), args,
                                       (size_t)stream_layout_.total, stream_));
  return DMM_OK;
}

dmm_status Pack::plan_grid(const std::vector<int32_t>& cand, std::vector<int32_t>* taken) {
  taken->clear();
  gr_groups_.clear();
  const bool fp64 = prec_ == DMM_FP64;
  const int T = (int)tsize_, kw = 16 / T;
  std::vector<int32_t> list;
  for (int32_t i : cand)
    if (inst_h_[i].m > 0 && inst_h_[i].nslots > 0) list.push_back(i);
  // rounds: the tilings are estimates, corrected by what a build reports
  std::vector<int> kc_min(live_.size(), 1), kv_min(live_.size(), 1);
  for (int round = 0; round < 4; round++) {
    if (list.empty() || (int)list.size() > sms_) return DMM_OK;
    // the SMs shared out by literal count, at least one block each
    double total = 0;
    for (int32_t i : list) total += inst_h_[i].nslots;
    std::vector<int> B(list.size());
    int used = 0;
    for (size_t k = 0; k < list.size(); k++) {
      B[k] = std::max(1, (int)(inst_h_[list[k]].nslots / total * sms_));
      used += B[k];
    }
    while (used != sms_) {  // take from, or give to, the formula with least / most per block
      size_t at = 0;
      for (size_t k = 1; k < list.size(); k++) {
        const double a = inst_h_[list[k]].nslots / (double)B[k],
                     c = inst_h_[list[at]].nslots / (double)B[at];
        if (used > sms_ ? (B[at] == 1 || (B[k] > 1 && a < c)) : a > c) at = k;
      }
      if (used > sms_ && B[at] == 1) return DMM_OK;
      B[at] += used > sms_ ? -1 : 1;
      used += used > sms_ ? -1 : 1;
    }
    std::vector<GridGroup> groups;
    std::vector<int32_t> blk, next;
    GridSizes z;
    bool general = false;
    for (size_t k = 0; k < list.size(); k++) {
      const InstDesc& I = inst_h_[list[k]];
      GridGroup g{};
      g.inst = list[k];
      g.blk0 = (int32_t)blk.size();
      g.B = B[k];
      g.n = I.n;
      g.m = I.m;
      g.L = I.nslots;
      g.k3 = I.k3;
      g.var0 = I.var0;
      g.cls0 = I.cls0;
      g.slot0 = I.slot0;
      // fewest tiles per block whose areas fit beside the block's voltages
      const double n = I.n, L = I.nslots;
      const double distinct = n * (1.0 - std::exp(-L / (B[k] * n))) * 1.02 + 0.5 * kw * B[k] + 16;
      bool fits = false;
      for (int sum = 2; sum <= kGridMaxTiles && !fits; sum++)
        for (int kc = (sum + 1) / 2; kc < sum && !fits; kc++) {
          const int kv = sum - kc;
          if (kc < kc_min[list[k]] || kv < kv_min[list[k]] || kv > kc) continue;
          const double stage = L / (B[k] * kc) * 1.02 + 0.5 * kw * B[k] * kv + 64;
          const double bucket = L / (B[k] * kv) * 1.06 + 0.5 * kw * B[k] * kc + 64;
          const double tvb = n / B[k] + 8 * kv;
          const double smem = T * distinct + T * std::max(stage, bucket) + tvb * (2 * T + 9) +
                              8 * B[k] + (fp64 ? 16384 : 0) + 2048;
          if (distinct > kGridMaxDistinct || stage > 65000 || bucket > 65000 ||
              smem > kGridSmemMax || B[k] * kv > 1024 || B[k] * kc > 1024)
            continue;
          g.kc = kc;
          g.kv = kv;
          fits = true;
        }
      // one large formula: the staged and tile forms are faster once a block's share is large
      // (n at 8 clauses per variable, us per step against them: FP32 50,000 12.5 / 13.4, 70,000
      // 16.9 / 15.5; FP64 70,000 31.6 / 32.5, 100,000, with two tiles per block, 58 / 44)
      if (list.size() == 1 && ((!fp64 && I.k3 && L / B[k] > 9000) || (fp64 && g.kc + g.kv > 2)))
        fits = false;
      if (!fits) continue;
      g.TC = ((I.m + g.B * g.kc - 1) / (g.B * g.kc) + 3) & ~3;
      g.TV = ((I.n + g.B * g.kv - 1) / (g.B * g.kv) + 3) & ~3;
      g.TVr = (g.TV + 31) & ~31;
      g.nct = g.B * g.kc;
      g.nvt = g.B * g.kv;
      g.lt = g.kc;
      g.pad = kw;
      g.NL = g.B;
      g.list0 = g.blk0;
      grid_place(&g, &z);
      general |= I.k3 == 0;
      for (int b = 0; b < g.B; b++) blk.push_back((int32_t)groups.size());
      groups.push_back(g);
      next.push_back(list[k]);
    }
    if (next.size() != list.size()) {  // share the SMs among those that fit
      list = next;
      continue;
    }
    if (z.ux > INT32_MAX / 2 || z.row > INT32_MAX / 2) return DMM_OK;
    if (cand.size() > 1 && !grid_pays(cand, list, groups)) return DMM_OK;
    // (the tables of the same formulas in the same tiles are still valid: only this function
    // writes them, and a live formula's device arrays do not change)
    std::vector<uint64_t> key;
    for (const GridGroup& g : groups) {
      key.push_back(add_serial_[g.inst]);
      key.push_back(((uint64_t)g.B << 40) | ((uint64_t)g.kc << 20) | (uint64_t)g.kv);
    }
    if (key == gr_key_) {
      gr_groups_ = groups;
      *taken = list;
      return DMM_OK;
    }
    gr_key_.clear();
    GridTables t{};
    std::vector<int32_t> out;
    const dmm_status st = grid_tables(groups, blk, (int)blk.size(), z, false, &t, &out);
    if (st == DMM_ERR_NOMEM) {
      drop_grid_tables();
      return DMM_OK;
    }
    DMM_TRY(st);
    // what the tables need; a formula whose tiles came out too large gets more of them
    GridCaps caps{};
    bool again = false;
    for (size_t k = 0; k < groups.size(); k++) {
      const int32_t* o = &out[k * kGridOut];
      const GridGroup& g = groups[k];
      if (o[0] == 1) {
        list.erase(list.begin() + (long)k);
        again = true;
        break;
      }
      GridCaps one{o[1], o[2], o[3], g.TV * g.kv, g.B, g.TC * g.kc, o[5], o[6],
                   g.kv * g.TVr * 32, o[7], o[4]};
      if (o[0] == 2 || o[0] == 3 || grid_smem(one, fp64, g.k3 == 0, 0) > kGridSmemMax) {
        if (o[0] == 2 || (o[0] == 0 && one.st > one.bk)) kc_min[g.inst] = g.kc + 1;
        else kv_min[g.inst] = g.kv + 1, kc_min[g.inst] = std::max(g.kc, g.kv + 1);
        again = true;
      }
      caps.dl = std::max(caps.dl, one.dl);
      caps.st = std::max(caps.st, one.st);
      caps.bk = std::max(caps.bk, one.bk);
      caps.tv = std::max(caps.tv, one.tv);
      caps.B = std::max(caps.B, one.B);
      caps.tc = std::max(caps.tc, one.tc);
      caps.ts = std::max(caps.ts, one.ts);
      caps.wd = std::max(caps.wd, one.wd);
      caps.row = std::max(caps.row, one.row);
      caps.csr = std::max(caps.csr, one.csr);
      caps.snd = std::max(caps.snd, one.snd);
    }
    if (again) continue;
    if (grid_smem(caps, fp64, general, 0) > kGridSmemMax) {
      // formulas whose maxima do not fit together: the one with the largest areas goes elsewhere
      size_t at = 0;
      for (size_t k = 1; k < groups.size(); k++)
        if (inst_h_[groups[k].inst].nslots > inst_h_[groups[at].inst].nslots) at = k;
      list.erase(list.begin() + (long)at);
      continue;
    }
    gr_resident_ = 2;
    while (gr_resident_ > 0 && grid_smem(caps, fp64, general, gr_resident_) > kGridSmemMax)
      gr_resident_--;
    gr_layout_ = grid_shape(caps, fp64, general, gr_resident_);
    const void* fn = grid_kernel(fp64, general, gr_resident_);
    if (resident_blocks(fn, fp64 ? kGridThreads64 : kGridThreads, gr_layout_.total, kGridSmemMax) < 1)
      return DMM_OK;
    gr_general_ = general;
    gr_tables_ = t;
    gr_blocks_ = (int32_t)blk.size();
    gr_key_ = key;
    gr_clean_ = false;
    gr_groups_ = groups;
    *taken = list;
    return DMM_OK;
  }
  return DMM_OK;
}

dmm_status Pack::launch_grid(int32_t nsteps) {
  const bool fp64 = prec_ == DMM_FP64;
  PackView<float> vf;
  PackView<double> vd;
  void* view;
  if (fp64) {
    fill_view<double>(&vd);
    view = &vd;
  } else {
    fill_view<float>(&vf);
    view = &vf;
  }
  void* sync = gbuf_[kGrSync];
  if (!gr_clean_) {
    DMM_CUDA(cudaMemsetAsync(sync, 0, gr_groups_.size() * kGridSyncBytes, stream_));
    DMM_CUDA(grid_unset(gr_tables_, fp64, stream_));
  }
  gr_clean_ = true;
  const void* fn = grid_kernel(fp64, gr_general_, gr_resident_);
  DMM_CUDA(allow_smem(fn, kGridSmemMax));
  const void* groups = gbuf_[kGrGroups];
  const void* blk = gbuf_[kGrBlk];
  void* epart = gbuf_[kGrEpart];
  int* err = error_d_;
  void* args[] = {view, &gr_tables_, &groups, &blk, &gr_layout_, &nsteps, &sync, &epart, &err};
  DMM_CUDA(cudaLaunchCooperativeKernel(fn, dim3((unsigned)gr_blocks_),
                                       dim3(fp64 ? kGridThreads64 : kGridThreads), args,
                                       (size_t)gr_layout_.total, stream_));
  return DMM_OK;
}

const void* Pack::persist_fn() const {
  if (xp_active_) return staged_fn(tun_.var_group, xp_mt_);
  if (one_active_) return persist_fn_x<true>(prec_, tun_.var_group);
  return persist_fn_x<false>(prec_, tun_.var_group);
}

// Tables of the staged form (dmm_xpose.cuh) for formula idx with clause tiles of TC and
// variable tiles of TV, built on the device (dmm_xprep.cuh); mt: the several-tiles-per-block
// form (the tile lists must hold that tiling).  Leaves *ok false (and the plain tile code in
// use) when the formula or its tiles do not fit the form's 16-bit indices or shared memory.
dmm_status Pack::prepare_xpose(int32_t idx, int TC, int TV, bool mt, bool* ok) {
  *ok = false;
  const InstDesc& I = inst_h_[idx];
  if (prec_ != DMM_FP32 || !I.k3) return DMM_OK;
  // the tables of the same formula at the same place with the same tiles are still valid
  // (only this function writes them, and a live formula's device arrays do not change)
  const XpKey key{idx, I.var0, I.slot0, I.n, I.m, TC, TV, tun_.var_group, mt, add_serial_[idx]};
  if (xp_key_valid_ && key == xp_key_) {
    *ok = true;
    return DMM_OK;
  }
  xp_key_valid_ = false;
  const int m = I.m, n = I.n, L = I.nslots;
  const int nct = (m + TC - 1) / TC, nvt = (n + TV - 1) / TV;
  if (nct <= 0 || nvt <= 0) return DMM_OK;
  if (!mt && (nct > grid_p_ || nvt > grid_p_)) return DMM_OK;
  if (nct > kXpMaxTiles || nvt > kXpMaxTiles) return DMM_OK;
  const int W = (n + 31) / 32;
  const int RW = std::min(W, kXpRangeWords);
  const int smem_k = (nvt + 2 * RW) * 4;
  if (smem_k > kXpSmemMax) return DMM_OK;
  const int64_t pairs = (int64_t)nct * nvt;
  const int64_t ux_cap = (int64_t)L + 8 * pairs;  // sector padding: < 8 per chunk
  if (ux_cap > INT32_MAX / 2) return DMM_OK;
  // scratch: cnt, sb, bt (pairs each), st, dcnt (nct each), btot (nvt), out (8)
  const int64_t scratch_ints = 3 * pairs + 2 * (int64_t)nct + nvt + 8;
  const int64_t bytes[kXpBufs] = {
      ((int64_t)L + 4 * nct) * 4,  // dlist
      2 * (int64_t)nct * 4,        // doff
      (int64_t)L * 2,              // llit
      (int64_t)L * 2,              // spos
      ux_cap * 4,                  // ux
      ((int64_t)nct + 1) * 4,      // ubase
      ((int64_t)nvt + 1) * 4,      // boff
      (ux_cap / 8 + 1) * 4,        // src8
      ux_cap * 2,                  // dst
      scratch_ints * 4};           // scratch
  for (int i = 0; i < kXpBufs; i++) {
    const int64_t want = std::max<int64_t>(bytes[i], 16);
    if (want > xbuf_cap_[i]) {
      if (xbuf_[i]) retire(xbuf_[i]);
      xbuf_[i] = nullptr;
      xbuf_cap_[i] = 0;
      DMM_CUDA(dev_alloc(&xbuf_[i], want));
      xbuf_cap_[i] = want;
    }
  }
  int* scr = static_cast<int*>(xbuf_[kXpScratch]);
  int* cnt = scr;
  int* sb = cnt + pairs;
  int* bt = sb + pairs;
  int* st = bt + pairs;
  int* dcnt = st + nct;
  int* btot = dcnt + nct;
  int* out = btot + nvt;
  auto* dlist = static_cast<int32_t*>(xbuf_[kXpDlist]);
  auto* doff = static_cast<int32_t*>(xbuf_[kXpDoff]);
  auto* llit = static_cast<int16_t*>(xbuf_[kXpLlit]);
  auto* spos = static_cast<uint16_t*>(xbuf_[kXpSpos]);
  auto* ubase = static_cast<int32_t*>(xbuf_[kXpUbase]);
  auto* boff = static_cast<int32_t*>(xbuf_[kXpBoff]);
  auto* src8 = static_cast<int32_t*>(xbuf_[kXpSrc8]);
  auto* dst = static_cast<uint16_t*>(xbuf_[kXpDst]);
  const int32_t* lit = lit_ + I.slot0;
  const int32_t* upos = upos_ + I.slot0;
  const int32_t* vend = vend_ + I.var0;
  DMM_CUDA(cudaMemsetAsync(dlist, 0, bytes[kXpDlist], stream_));
  DMM_CUDA(cudaMemsetAsync(dst, 0xFF, bytes[kXpDst], stream_));
  DMM_CUDA(allow_smem((const void*)k_xp_count<kXprepThreads>, kXpSmemMax));
  DMM_CUDA(allow_smem((const void*)k_xp_fill<kXprepThreads>, kXpSmemMax));
  k_xp_count<kXprepThreads><<<nct, kXprepThreads, smem_k, stream_>>>(lit, L, TC, TV, nvt, n, RW,
                                                                     cnt, sb, st, dcnt, spos);
  k_xp_scan<kXprepThreads><<<1, kXprepThreads, 0, stream_>>>(nct, nvt, cnt, st, dcnt, ubase,
                                                             doff, bt, boff, btot, out);
  k_xp_fill<kXprepThreads><<<nct, kXprepThreads, smem_k, stream_>>>(
      lit, upos, vend, L, TC, TV, nct, nvt, n, RW, sb, ubase, doff, bt, boff, dlist, llit, spos,
      dst, src8);
  DMM_CUDA(cudaGetLastError());
  int h[8];
  DMM_CUDA(cudaMemcpyAsync(h, out, sizeof h, cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  if (h[0] != 0) return DMM_OK;
  const int sv_cap = std::max(h[1], 4);
  const int st_cap = std::max(h[6], 8);
  const int bk_cap = mt ? std::max(h[7], 8) : std::max(h[2], 8);
  const int smem = mt ? xp_layout_mt(sv_cap, st_cap, bk_cap, TV).total
                      : xp_layout(sv_cap, bk_cap, TV).total;
  if (smem > staged_smem_max(mt)) return DMM_OK;
  if (resident_blocks(staged_fn(tun_.var_group, mt), kStagedThreads, smem, staged_smem_max(mt)) * sms_ !=
      grid_p_)
    return DMM_OK;
  xsv_cap_ = sv_cap;
  xst_cap_ = st_cap;
  xbk_cap_ = bk_cap;
  xtv_cap_ = TV;
  xsmem_ = smem;
  xp_mt_ = mt;
  xp_key_ = key;
  xp_key_valid_ = true;
  *ok = true;
  return DMM_OK;
}

// Tile lists of the single live formula idx (the only entries of the tables).
dmm_status Pack::set_tiles(int32_t idx, int TC, int TV) {
  InstDesc& I = inst_h_[idx];
  ctiles_h_.clear();
  vtiles_h_.clear();
  I.ctile0 = 0;
  for (int32_t b = 0; b < I.m; b += TC) ctiles_h_.push_back(Tile{idx, b, std::min(TC, I.m - b), 0});
  I.nctile = (int32_t)ctiles_h_.size();
  I.vtile0 = 0;
  for (int32_t b = 0; b < I.n; b += TV) vtiles_h_.push_back(Tile{idx, b, std::min(TV, I.n - b), 0});
  I.nvtile = (int32_t)vtiles_h_.size();
  if ((int64_t)ctiles_h_.size() > ctile_cap_ || (int64_t)vtiles_h_.size() > vtile_cap_) {
    set_error("tile tables overflow");
    return DMM_ERR_BUDGET;
  }
  return upload_desc(idx);
}

// The several-tiles-per-block staged form: k_c clause tiles and k_v variable tiles per block
// (tile counts multiples of the grid, so that every block has the same number).  Candidate
// tilings whose estimated shared memory fits are ordered by an estimate of their step time
// (a fixed cost per tile a block visits, plus the bytes of the tiles' variable lists and of
// the chunk padding at the measured HBM rate); the first one whose tables build and fit is
// kept.  Leaves *ok false, with the tile lists in an unspecified state, when none fits.
dmm_status Pack::prepare_xpose_mt(int32_t idx, bool* ok) {
  *ok = false;
  const InstDesc& I = inst_h_[idx];
  if (prec_ != DMM_FP32 || !I.k3) return DMM_OK;
  const double n = I.n, m = I.m;
  const int grid = grid_p_;
  struct Cand {
    int TC, TV;
    double cost;
  };
  std::vector<Cand> cands;
  for (int kc = 1; kc <= 64; kc++) {
    const int TC = (int)(((int64_t)std::ceil(m / (kc * (double)grid)) + 3) & ~int64_t(3));
    if (TC < kMinClauseTile) break;
    const double nct = std::ceil(m / TC);
    const double distinct = n * (1.0 - std::exp(-3.0 * TC / n));
    for (int kv = 1; kv <= 64; kv++) {
      const int TV = (int)(((int64_t)std::ceil(n / (kv * (double)grid)) + 3) & ~int64_t(3));
      if (TV < kMinVarTile) break;
      const double nvt = std::ceil(n / TV);
      const double stage = 3.0 * TC + 3.5 * nvt;
      const double bucket = 3.0 * m / nvt * 1.08 + 3.5 * nct;
      if (distinct > 30000 || stage > 60000 || bucket > 60000) continue;
      const double smem = 4.0 * std::max(distinct * 1.03 + stage, bucket) + 0.5 * bucket +
                          9.0 * TV + 4096;
      if (smem > kXpSmemMaxMT + 7 * 1024) continue;  // the estimate runs up to ~6 KB high
      const double bytes = 4.0 * distinct * nct + 8.0 * 3.5 * nct * nvt;
      cands.push_back({TC, TV, 2.0 * (kc + kv) + bytes / 6.0e6});
    }
  }
  std::sort(cands.begin(), cands.end(), [](const Cand& a, const Cand& b) { return a.cost < b.cost; });
  for (size_t k = 0; k < cands.size() && k < 8; k++) {
    DMM_TRY(set_tiles(idx, cands[k].TC, cands[k].TV));
    DMM_TRY(prepare_xpose(idx, cands[k].TC, cands[k].TV, true, ok));
    if (*ok) return DMM_OK;
  }
  return DMM_OK;
}

dmm_status Pack::commit_tiles() {
  DMM_TRY(resolve_long_lists());
  stream_active_ = false;
  short_ = ShortPlan::none;
  ctiles_h_.clear();
  vtiles_h_.clear();
  std::vector<int32_t> live_list;
  // formulas that one block integrates alone (FP32, V and dV fit in shared memory): used
  // when there are enough of them to fill the GPU (auto) or when forced (launch_mode 3)
  std::vector<int32_t> small_list, cluster_list;
  {
    std::vector<int32_t> eligible, others;
    for (int32_t i = 0; i < (int32_t)live_.size(); i++) {
      if (!live_[i]) continue;
      const bool ok = prec_ == DMM_FP32 && inst_h_[i].n <= kInstVCap &&
                      (tun_.launch_mode == 0 || tun_.launch_mode == 3);
      (ok ? eligible : others).push_back(i);
    }
    const bool use_small = tun_.launch_mode == 3 || (int64_t)eligible.size() >= sms_;
    if (use_small) {
      small_list = eligible;
    } else {
      others.insert(others.end(), eligible.begin(), eligible.end());
      std::sort(others.begin(), others.end());
    }
    // with the launch shape left open, the cluster form takes the formulas that fit it and the
    // resident grid form the others, or the latter takes all of them when the estimated step
    // is shorter (the server's formulas change between launches: no tables are built for them)
    clusters_.clear();
    gr_groups_.clear();
    const bool open_shape = tun_.launch_mode == 0 && tun_.u_layout == 0 && tun_.clause_tile == 0 &&
                            tun_.var_tile == 0;
    if (open_shape && !no_cluster_) DMM_TRY(plan_clusters(others, &cluster_list));
    if (open_shape && !no_grid_ && !fixed_grid_) {
      const std::vector<int32_t> rest = without(others, cluster_list);
      if (!cluster_list.empty() &&
          grid_step_us(others) < cluster_step_us() + (rest.empty() ? 0.0 : grid_step_us(rest))) {
        clusters_.clear();
        cluster_list.clear();
      }
      std::vector<int32_t> grid_list;
      DMM_TRY(plan_grid(without(others, cluster_list), &grid_list));
      cluster_list.insert(cluster_list.end(), grid_list.begin(), grid_list.end());
    }
    others = without(others, cluster_list);
    live_list = others;
    std::stable_sort(small_list.begin(), small_list.end(),
                     [&](int32_t a, int32_t b) { return inst_h_[a].m > inst_h_[b].m; });
  }
  n_small_ = (int32_t)small_list.size();
  small_list.insert(small_list.end(), cluster_list.begin(), cluster_list.end());
  for (int32_t i : small_list) {
    inst_h_[i].ctile0 = inst_h_[i].nctile = inst_h_[i].vtile0 = inst_h_[i].nvtile = 0;
    DMM_TRY(upload_desc(i));
  }
  if (!small_list.empty())
    DMM_CUDA(cudaMemcpyAsync(order_d_, small_list.data(), small_list.size() * sizeof(int32_t),
                             cudaMemcpyHostToDevice, stream_));
  for (auto& c : clusters_) c.first += n_small_;
  return plan_tiles(live_list, small_list.empty());
}

dmm_status Pack::plan_tiles(const std::vector<int32_t>& live_list, bool alone) {
  xp_active_ = false;
  one_active_ = false;
  // grids
  int bc, bv;
  if (prec_ == DMM_FP64) {
    bc = occupancy_blocks((const void*)k_clause<double, false>, kThreads);
    bv = occupancy_blocks((const void*)k_var<double, 32, true, 0>, kThreads);
  } else {
    bc = occupancy_blocks((const void*)k_clause<float, true>, kThreads);
    bv = occupancy_blocks((const void*)k_var<float, 8, false, 0>, kThreads);
  }
  if (tun_.blocks_per_sm > 0) {
    bc = std::min(bc, tun_.blocks_per_sm);
    bv = std::min(bv, tun_.blocks_per_sm);
  }
  grid_p_ = occupancy_blocks(persist_fn(), persist_threads(prec_)) * sms_;
  const bool coop = tun_.launch_mode != 1;
  const int block = coop ? persist_threads(prec_) : kThreads;
  const int64_t spread = coop ? grid_p_ : (int64_t)bc * sms_;
  // tile sizes: balanced over the grid for a single instance, else fixed
  int TC = tun_.clause_tile, TV = tun_.var_tile;
  if (TC == 0) {
    TC = 4 * block;
    if (live_list.size() == 1) {
      const int64_t m = inst_h_[live_list[0]].m;
      TC = (int)std::max<int64_t>(kMinClauseTile, ((m + spread - 1) / spread + 3) & ~int64_t(3));
    }
  }
  if (TV == 0) {
    TV = block;
    if (live_list.size() == 1) {
      const int64_t n = inst_h_[live_list[0]].n;
      // a multiple of 4 (not of a warp) so that every block gets a variable tile
      TV = (int)std::max<int64_t>(kMinVarTile, ((n + spread - 1) / spread + 3) & ~int64_t(3));
    }
  }
  for (int32_t i : live_list) {
    InstDesc& I = inst_h_[i];
    I.ctile0 = (int32_t)ctiles_h_.size();
    for (int32_t b = 0; b < I.m; b += TC) ctiles_h_.push_back(Tile{i, b, std::min(TC, I.m - b), 0});
    I.nctile = (int32_t)ctiles_h_.size() - I.ctile0;
    I.vtile0 = (int32_t)vtiles_h_.size();
    for (int32_t b = 0; b < I.n; b += TV) vtiles_h_.push_back(Tile{i, b, std::min(TV, I.n - b), 0});
    I.nvtile = (int32_t)vtiles_h_.size() - I.vtile0;
    DMM_TRY(upload_desc(i));
  }
  if ((int64_t)ctiles_h_.size() > ctile_cap_ || (int64_t)vtiles_h_.size() > vtile_cap_) {
    set_error("tile tables overflow");
    return DMM_ERR_BUDGET;
  }
  // one formula on the cooperative path: two grid barriers per step; FP32 with the
  // default layout and tiles: the staged form when it fits
  one_active_ = coop && live_list.size() == 1 && alone;
  if (one_active_ && tun_.u_layout == 0 && tun_.clause_tile == 0 && tun_.var_tile == 0) {
    const int32_t one = live_list[0];
    if (prec_ == DMM_FP32) DMM_TRY(prepare_xpose(one, TC, TV, false, &xp_active_));
    // too large for one tile per block: the streaming form (tiles in turn), else several staged
    // tiles per block, else the tiles above
    // (FP32 from 9 million literals on: below, and in FP64, where the sorted sums bound the
    // step, its third barrier costs more than the gathers it saves; dmm_stream.cuh)
    if (!xp_active_ && tun_.launch_mode == 0 && !fixed_grid_ && !no_grid_ && prec_ == DMM_FP32 &&
        inst_h_[one].nslots >= kStreamSlots)
      DMM_TRY(plan_stream(one, &stream_active_));
    if (!xp_active_ && !stream_active_ && prec_ == DMM_FP32) {
      DMM_TRY(prepare_xpose_mt(one, &xp_active_));
      if (!xp_active_) DMM_TRY(set_tiles(one, TC, TV));
    }
  }
  if (!ctiles_h_.empty())
    DMM_CUDA(cudaMemcpyAsync(ctiles_d_, ctiles_h_.data(), ctiles_h_.size() * sizeof(Tile),
                             cudaMemcpyHostToDevice, stream_));
  if (!vtiles_h_.empty())
    DMM_CUDA(cudaMemcpyAsync(vtiles_d_, vtiles_h_.data(), vtiles_h_.size() * sizeof(Tile),
                             cudaMemcpyHostToDevice, stream_));
  live0_ = live_list.size() == 1 ? live_list[0] : -1;
  if (!live_list.empty())
    DMM_CUDA(cudaMemcpyAsync(live_d_, live_list.data(), live_list.size() * sizeof(int32_t),
                             cudaMemcpyHostToDevice, stream_));
  int32_t nt[2] = {(int32_t)ctiles_h_.size(), (int32_t)vtiles_h_.size()};
  int32_t nl = (int32_t)live_list.size();
  DMM_CUDA(cudaMemcpyAsync(ntiles_d_, nt, sizeof nt, cudaMemcpyHostToDevice, stream_));
  DMM_CUDA(cudaMemcpyAsync(misc_d_, &nl, sizeof nl, cudaMemcpyHostToDevice, stream_));
  const int gc = bc * sms_, gv = bv * sms_;
  const int new_c = fixed_grid_ ? gc : std::max(1, std::min<int>(gc, nt[0]));
  const int new_v = fixed_grid_ ? gv : std::max(1, std::min<int>(gv, nt[1]));
  if (new_c != grid_c_ || new_v != grid_v_) graph_stale_ = true;
  grid_c_ = new_c;
  grid_v_ = new_v;
  if (!fixed_grid_) graph_stale_ = true;
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

// Launches of up to this many steps leave a formula of the cluster or resident grid form to the
// tile forms: those forms bring the formula and their tables into shared memory when a launch
// starts, which only the following steps win back.  us per call of step(k), resident or cluster
// / tile forms: FP32 at 8 clauses of three literals per variable, n = 2,000 (cluster) k = 1
// 108 / 102, 4 118 / 126; 20,000 k = 1 116 / 100, 4 143 / 128, 16 237 / 238; 50,000 k = 4
// 166 / 145, 16 312 / 304, 32 503 / 515; FP64 at 4.3, 50,000 k = 1 130 / 106, 4 171 / 161, 16
// 332 / 381; clauses of 1 to 8 literals FP32 n = 30,000 k = 1 124 / 109, 4 156 / 174.
int32_t Pack::short_steps() const {
  if (fixed_grid_ || tun_.launch_mode == 1 || !ctiles_h_.empty() || !vtiles_h_.empty() ||
      n_small_ > 0)
    return 0;
  if (gr_groups_.empty() && clusters_.size() == 1 && clusters_[0].count == 1) {
    const int32_t m = clusters_[0].R * clusters_[0].caps.tc;
    return clusters_[0].general || m < 8600 ? 0 : m / 5000;
  }
  if (gr_groups_.size() != 1 || !clusters_.empty()) return 0;
  return gr_general_ ? 2 : 2 + gr_groups_[0].m / (prec_ == DMM_FP64 ? 100000 : 20000);
}

dmm_status Pack::plan_short() {
  if (short_ != ShortPlan::none) return DMM_OK;
  short_ = ShortPlan::refused;
  int32_t one = -1, count = 0;
  for (int32_t i = 0; i < (int32_t)live_.size(); i++)
    if (live_[i]) {
      one = i;
      count++;
    }
  if (count != 1) return DMM_OK;
  no_grid_ = true;  // the streaming form's tables share the resident grid form's memory
  const dmm_status st = plan_tiles({one}, true);
  no_grid_ = false;
  // the committed forms stay as they are: these tiles are launched by short launches alone
  ctiles_h_.clear();
  vtiles_h_.clear();
  if (st == DMM_ERR_NOMEM) {
    clear_error();
    xp_active_ = one_active_ = false;
    return DMM_OK;
  }
  DMM_TRY(st);
  short_ = ShortPlan::ready;
  return DMM_OK;
}

dmm_status Pack::launch_persist(int32_t nsteps) {
  PackView<float> vf;
  PackView<double> vd;
  void* view;
  if (prec_ == DMM_FP64) {
    fill_view<double>(&vd);
    view = &vd;
  } else {
    fill_view<float>(&vf);
    view = &vf;
  }
  static_assert(kMiscAcc2 * 4 + 2 * sizeof(StepAcc) <= kMiscInts * 4, "misc area");
  static_assert(kMiscInts - kMiscLaunch == kLaunchAreaInts, "launch area");
  unsigned int* bar = reinterpret_cast<unsigned int*>(misc_d_ + kMiscLaunch);
  int* err = error_d_;
  // a completed launch leaves its area zeroed (leave_launch); after an error or before the
  // first launch it is zeroed here
  if (!launch_area_clean_)
    DMM_CUDA(cudaMemsetAsync(bar, 0, kLaunchAreaInts * sizeof(int32_t), stream_));
  launch_area_clean_ = true;
  void* args[] = {view, &nsteps, &bar, &err};
  const size_t smem = xp_active_ ? (size_t)xsmem_ : 0;
  if (smem) DMM_CUDA(allow_smem(persist_fn(), staged_smem_max(xp_mt_)));
  const int block = xp_active_ ? kStagedThreads : persist_threads(prec_);
  DMM_CUDA(cudaLaunchCooperativeKernel(persist_fn(), dim3(grid_p_), dim3(block), args, smem,
                                       stream_));
  return DMM_OK;
}

dmm_status Pack::plan_clusters(const std::vector<int32_t>& cand, std::vector<int32_t>* taken) {
  taken->clear();
  const bool fp64 = prec_ == DMM_FP64;
  const int ts = (int)tsize_;
  std::vector<int32_t> list, fresh;
  for (int32_t i : cand) {
    const InstDesc& I = inst_h_[i];
    if (I.n > kClusterMaxVars || 2 * (int64_t)ts * I.n > kClusterSmemMax ||
        3 * (int64_t)ts * I.m / kClusterMax > kClusterSmemMax)
      continue;
    list.push_back(i);
    if (cl_need_[i].serial != add_serial_[i]) fresh.push_back(i);
  }
  if (list.empty()) return DMM_OK;
  if (!fresh.empty()) {
    const int64_t need = 2 * kClusterSizes * (int64_t)fresh.size();
    DMM_TRY(ensure_stage(need));
    DMM_CUDA(cudaMemcpyAsync(order_d_, fresh.data(), fresh.size() * sizeof(int32_t),
                             cudaMemcpyHostToDevice, stream_));
    DMM_CUDA(cluster_need(inst_d_, order_d_, (int)fresh.size(), vend_, coff_,
                          reinterpret_cast<int2*>(stage_), stream_));
    std::vector<int2> h(fresh.size() * kClusterSizes);
    DMM_CUDA(cudaMemcpyAsync(h.data(), stage_, h.size() * sizeof(int2), cudaMemcpyDeviceToHost,
                             stream_));
    DMM_CUDA(cudaStreamSynchronize(stream_));
    for (size_t f = 0; f < fresh.size(); f++) {
      ClusterNeed& q = cl_need_[fresh[f]];
      q.serial = add_serial_[fresh[f]];
      for (int r = 0; r < kClusterSizes; r++) {
        q.bk[r] = h[f * kClusterSizes + r].x;
        q.ts[r] = h[f * kClusterSizes + r].y;
      }
    }
  }
  // Cluster size: the SMs shared out evenly over the formulas (one formula: 16 blocks, the
  // fastest size from n = 500 on and within 6 % of the best below), or the next larger size
  // that holds the formula.  Formulas of one size and clause kind share a launch.
  int q0 = kClusterSizes - 1;
  while (q0 > 0 && ((int64_t)list.size() << q0) > sms_) q0--;
  // With more formulas than SMs (FP64: the FP32 ones run one block each) the clusters run in many
  // waves, and few of 16 blocks are resident at once: formulas that need them are faster in the
  // tile forms (200 formulas, clauses each, blocks, us per step against them: 8,600, 8, 101 / 130;
  // 12,000, 8, 137 / 177; 12,900, 16, 218 / 194; 16,000, 16, 255 / 219).
  const int sizes = (int)list.size() > sms_ ? kClusterSizes - 1 : kClusterSizes;
  std::vector<std::vector<int32_t>> member;
  for (int32_t i : list) {
    const InstDesc& I = inst_h_[i];
    for (int q = q0; q < sizes; q++) {
      const bool general = I.k3 == 0;
      size_t g = 0;
      while (g < clusters_.size() && (clusters_[g].R != 1 << q || clusters_[g].general != general)) g++;
      ClusterLaunch L;
      if (g < clusters_.size()) L = clusters_[g];
      L.R = 1 << q;
      L.general = general;
      L.caps.n = std::max(L.caps.n, I.n);
      L.caps.tc = std::max(L.caps.tc, cluster_tc(I.m, L.R));
      L.caps.ts = std::max(L.caps.ts, cl_need_[i].ts[q]);
      L.caps.tv = std::max(L.caps.tv, cluster_tv(I.n, L.R));
      L.caps.bk = std::max(L.caps.bk, cl_need_[i].bk[q]);
      L.smem = cluster_smem(L.caps, fp64, general);
      if (L.smem > kClusterSmemMax) continue;
      if (g == clusters_.size()) {
        ClusterLaunch one = L;  // the device must be able to hold such a cluster
        one.count = 1;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        DMM_TRY(cluster_config(one, &cfg, &at));
        int act = 0;
        if (cudaOccupancyMaxActiveClusters(&act, cluster_kernel(fp64, general), &cfg) !=
                cudaSuccess || act < 1) {
          cudaGetLastError();
          continue;
        }
        L.resident = act;
        clusters_.push_back(L);
        member.emplace_back();
      }
      L.count++;
      clusters_[g] = L;
      member[g].push_back(i);
      break;
    }
  }
  // the launches of large clusters first: they take longest
  std::vector<size_t> by(clusters_.size());
  for (size_t g = 0; g < by.size(); g++) by[g] = g;
  std::stable_sort(by.begin(), by.end(),
                   [&](size_t a, size_t b) { return clusters_[a].R > clusters_[b].R; });
  std::vector<ClusterLaunch> sorted;
  for (size_t g : by) {
    clusters_[g].first = (int32_t)taken->size();
    sorted.push_back(clusters_[g]);
    taken->insert(taken->end(), member[g].begin(), member[g].end());
  }
  clusters_ = sorted;
  return DMM_OK;
}

// Launch parameters of a cluster launch; sets the kernel's attributes (per device, cheap).
dmm_status Pack::cluster_config(const ClusterLaunch& L, cudaLaunchConfig_t* cfg,
                                cudaLaunchAttribute* at) {
  const bool fp64 = prec_ == DMM_FP64;
  const void* fn = cluster_kernel(fp64, L.general);
  DMM_CUDA(allow_smem(fn, kClusterSmemMax));
  if (L.R > 8) DMM_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  *cfg = cudaLaunchConfig_t{};
  *at = cudaLaunchAttribute{};
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)L.R;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg->gridDim = dim3((unsigned)(L.count * L.R));
  cfg->blockDim = dim3((unsigned)cluster_threads(L.caps, fp64));
  cfg->dynamicSmemBytes = (size_t)L.smem;
  cfg->stream = stream_;
  cfg->attrs = at;
  cfg->numAttrs = 1;
  return DMM_OK;
}

dmm_status Pack::launch_cluster(int32_t nsteps) {
  const bool fp64 = prec_ == DMM_FP64;
  PackView<float> vf;
  PackView<double> vd;
  void* view;
  if (fp64) {
    fill_view<double>(&vd);
    vd.upos = upos_;
    view = &vd;
  } else {
    fill_view<float>(&vf);
    vf.upos = upos_;
    view = &vf;
  }
  // launches of different cluster sizes run side by side: the first on the pack's stream,
  // the others on streams forked from it and joined again
  const size_t G = clusters_.size();
  if (G > 1) {
    while (side_.size() + 1 < G) {
      cudaStream_t s = nullptr;
      cudaEvent_t e = nullptr;
      DMM_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      side_.push_back({s, e});
      DMM_CUDA(cudaStreamCreateWithFlags(&side_.back().first, cudaStreamNonBlocking));
    }
    DMM_CUDA(cudaEventRecord(ev_[3], stream_));
  }
  dmm_status st = DMM_OK;
  for (size_t g = 0; g < G && st == DMM_OK; g++) {
    const ClusterLaunch& L = clusters_[g];
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    DMM_TRY(cluster_config(L, &cfg, &at));
    const int32_t* order = order_d_ + L.first;
    ClusterCaps caps = L.caps;
    void* args[] = {view, &order, &nsteps, &caps};
    if (g > 0) {
      cfg.stream = side_[g - 1].first;
      DMM_CUDA(cudaStreamWaitEvent(cfg.stream, ev_[3], 0));
    }
    DMM_CUDA(cudaLaunchKernelExC(&cfg, cluster_kernel(fp64, L.general), args));
    if (g > 0) {
      DMM_CUDA(cudaEventRecord(side_[g - 1].second, cfg.stream));
      DMM_CUDA(cudaStreamWaitEvent(stream_, side_[g - 1].second, 0));
    }
  }
  return st;
}

template <int G>
static dmm_status launch_inst_g(const PackView<float>& v, const int32_t* order, int count,
                                int nsteps, int* queue, int grid, cudaStream_t s) {
  // function attributes are per device: set it on the current one (a cheap driver call)
  DMM_CUDA(allow_smem((const void*)k_inst<G>, (int)kInstSmem));
  k_inst<G><<<grid, kInstThreads, kInstSmem, s>>>(v, order, count, nsteps, queue);
  DMM_CUDA(cudaGetLastError());
  return DMM_OK;
}

dmm_status Pack::launch_inst(int32_t nsteps) {
  PackView<float> v;
  fill_view<float>(&v);
  // variable-major contributions by default here: scattered into shared memory, then read
  // contiguously per variable (measured 1.5x faster than gathering through the CSR)
  v.upos = tun_.u_layout == 1 ? nullptr : upos_;
  int* queue = misc_d_ + 3;
  DMM_CUDA(cudaMemsetAsync(queue, 0, sizeof(int32_t), stream_));
  const int grid = std::max(1, std::min(sms_, (int)n_small_));
  switch (tun_.var_group) {
    case 1: return launch_inst_g<1>(v, order_d_, n_small_, nsteps, queue, grid, stream_);
    case 2: return launch_inst_g<2>(v, order_d_, n_small_, nsteps, queue, grid, stream_);
    case 4: return launch_inst_g<4>(v, order_d_, n_small_, nsteps, queue, grid, stream_);
    case 8: return launch_inst_g<8>(v, order_d_, n_small_, nsteps, queue, grid, stream_);
    case 16: return launch_inst_g<16>(v, order_d_, n_small_, nsteps, queue, grid, stream_);
    default: return launch_inst_g<32>(v, order_d_, n_small_, nsteps, queue, grid, stream_);
  }
}

dmm_status Pack::check_error() {
  int32_t e = 0;
  DMM_CUDA(cudaMemcpyAsync(&e, error_d_, sizeof(int32_t), cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  if (e) {
    launch_area_clean_ = false;
    gr_clean_ = false;
    DMM_CUDA(cudaMemsetAsync(error_d_, 0, sizeof(int32_t), stream_));  // reported once
    DMM_CUDA(cudaStreamSynchronize(stream_));
    set_error("grid barrier wait gave up in the cooperative step kernel");
    return DMM_ERR_CUDA;
  }
  return DMM_OK;
}

// Commits the grid-wide forms for the scope of a call that traces or tests their barriers, or
// (tiles) the forms over the tile tables, when other forms run some of the pack's formulas.
struct Pack::TileForms {
  Pack& p;
  const bool on;
  dmm_status st = DMM_OK;
  TileForms(Pack& pack, bool tiles)
      : p(pack), on(!pack.clusters_.empty() || (tiles && !pack.gr_groups_.empty())) {
    if (!on) return;
    p.no_cluster_ = true;
    p.no_grid_ = tiles;
    st = p.commit_tiles();
  }
  ~TileForms() {
    p.no_cluster_ = p.no_grid_ = false;
    if (on) p.commit_tiles();
  }
};

dmm_status Pack::test_barrier_timeout() {
  DMM_CUDA(cudaSetDevice(dev_));
  TileForms tile_forms(*this, false);
  DMM_TRY(tile_forms.st);
  if (tun_.launch_mode == 1 || (ctiles_h_.empty() && vtiles_h_.empty() && gr_groups_.empty())) {
    set_error("the barrier test needs the cooperative launch of tile-path formulas");
    return DMM_ERR_STATE;
  }
  barrier_extra_ = 1;
  const dmm_status st = gr_groups_.empty() ? launch_tiles(1) : launch_grid(1);
  barrier_extra_ = 0;
  DMM_TRY(st);
  // a run has its next launch queued before it sees the error: the forms that check for one
  // must leave the state and the control record alone
  if (!gr_groups_.empty()) DMM_TRY(launch_grid(1));
  else if (stream_active_) DMM_TRY(launch_stream(1));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return check_error();
}

dmm_status Pack::capture(int32_t steps) {
  if (graph_exec_) {
    DMM_CUDA(cudaGraphExecDestroy(graph_exec_));
    graph_exec_ = nullptr;
  }
  if (graph_) {
    DMM_CUDA(cudaGraphDestroy(graph_));
    graph_ = nullptr;
  }
  DMM_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
  dmm_status st = DMM_OK;
  for (int32_t s = 0; s < steps && st == DMM_OK; s++) st = enqueue_step(false, nullptr);
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(stream_, &g);
  if (st != DMM_OK) {
    if (g) cudaGraphDestroy(g);
    return st;
  }
  DMM_CUDA(e);
  graph_ = g;
  DMM_CUDA(cudaGraphInstantiate(&graph_exec_, graph_, 0));
  graph_steps_ = steps;
  graph_stale_ = false;
  return DMM_OK;
}

dmm_status Pack::launch_steps(int32_t nsteps) {
  DMM_CUDA(cudaSetDevice(dev_));
  if (!planned()) return DMM_OK;
  const int32_t S = tun_.steps_per_graph;
  if (nsteps <= short_steps()) {
    DMM_TRY(plan_short());
    if (short_ == ShortPlan::ready) return nsteps > 0 ? launch_persist(nsteps) : DMM_OK;
  }
  if (tun_.launch_mode != 1) {
    // cluster launches alone take all the steps at once: their steps are a few microseconds,
    // and a launch's prologue costs about as much as two of them
    const bool clusters_only = cluster_only();
    while (nsteps > 0) {
      const int32_t k = clusters_only ? nsteps : std::min(nsteps, S);
      if (!ctiles_h_.empty() || !vtiles_h_.empty()) DMM_TRY(launch_tiles(k));
      if (n_small_ > 0) DMM_TRY(launch_inst(k));
      if (!gr_groups_.empty()) DMM_TRY(launch_grid(k));
      if (!clusters_.empty()) DMM_TRY(launch_cluster(k));
      nsteps -= k;
    }
    return DMM_OK;
  }
  while (nsteps >= S) {
    if (graph_stale_ || graph_steps_ != S || !graph_exec_) DMM_TRY(capture(S));
    DMM_CUDA(cudaGraphLaunch(graph_exec_, stream_));
    nsteps -= S;
  }
  for (int32_t s = 0; s < nsteps; s++) DMM_TRY(enqueue_step(false, nullptr));
  return DMM_OK;
}

dmm_status Pack::ensure_flush(int64_t flush_bytes) {
  if (flush_bytes > flush_cap_) {
    if (flush_) retire(flush_);
    flush_ = nullptr;
    DMM_CUDA(dev_alloc(&flush_, flush_bytes));
    flush_cap_ = flush_bytes;
  }
  return DMM_OK;
}

dmm_status Pack::time_steps_flushed(int32_t nsteps, int64_t flush_bytes, double* ms) {
  DMM_CUDA(cudaSetDevice(dev_));
  DMM_TRY(ensure_flush(flush_bytes));
  double total = 0.0;
  for (int32_t s = 0; s < nsteps; s++) {
    if (flush_bytes > 0) {
      k_flush<<<sms_ * 4, kThreads, 0, stream_>>>(static_cast<int4*>(flush_), flush_bytes / 16, s);
      DMM_CUDA(cudaGetLastError());
    }
    DMM_CUDA(cudaEventRecord(ev_[0], stream_));
    DMM_TRY(launch_steps(1));
    DMM_CUDA(cudaEventRecord(ev_[1], stream_));
    DMM_CUDA(cudaEventSynchronize(ev_[1]));
    float a = 0;
    DMM_CUDA(cudaEventElapsedTime(&a, ev_[0], ev_[1]));
    total += a;
  }
  *ms = total;
  return check_error();
}

dmm_status Pack::preload_kernels() {
  DMM_CUDA(cudaSetDevice(dev_));
  const int G = tun_.var_group;
  std::vector<const void*> fns = {
      persist_fn_x<false>(prec_, G), (const void*)k_count, (const void*)k_scan_block,
      (const void*)k_scan_add, (const void*)k_fill_start, (const void*)k_scatter,
      (const void*)k_sort_lists, (const void*)k_invert, (const void*)k_active_add,
      (const void*)k_put_desc,   (const void*)k_put_ctrl};
  if (prec_ == DMM_FP64) {
    fns.push_back((const void*)k_set_state<double>);
    fns.push_back((const void*)k_get_state<double>);
    fns.push_back((const void*)k_signs<double>);
    fns.push_back((const void*)k_signs_all<double>);
    fns.push_back((const void*)k_admit<double>);
    fns.push_back(persist_fn_x<true>(prec_, G));
  } else {
    fns.push_back((const void*)k_set_state<float>);
    fns.push_back((const void*)k_get_state<float>);
    fns.push_back((const void*)k_signs<float>);
    fns.push_back((const void*)k_signs_all<float>);
    fns.push_back((const void*)k_admit<float>);
    fns.push_back(persist_fn_x<true>(prec_, G));
    fns.push_back(staged_fn(G, false));
    fns.push_back(staged_fn(G, true));
    fns.push_back((const void*)k_xp_count<kXprepThreads>);
    fns.push_back((const void*)k_xp_scan<kXprepThreads>);
    fns.push_back((const void*)k_xp_fill<kXprepThreads>);
    switch (G) {
      case 1: fns.push_back((const void*)k_inst<1>); break;
      case 2: fns.push_back((const void*)k_inst<2>); break;
      case 4: fns.push_back((const void*)k_inst<4>); break;
      case 8: fns.push_back((const void*)k_inst<8>); break;
      case 16: fns.push_back((const void*)k_inst<16>); break;
      default: fns.push_back((const void*)k_inst<32>); break;
    }
  }
  fns.push_back(cluster_kernel(prec_ == DMM_FP64, false));
  fns.push_back(cluster_kernel(prec_ == DMM_FP64, true));
  grid_functions(prec_ == DMM_FP64, &fns);
  if (prec_ == DMM_FP32) {
    fns.push_back(stream_kernel(false));
    fns.push_back(stream_kernel(true));
  }
  for (const void* f : fns) {
    cudaFuncAttributes a;
    DMM_CUDA(cudaFuncGetAttributes(&a, f));
  }
  return DMM_OK;
}

int Pack::launch_form() const {
  if (tun_.launch_mode == 1) return 1;
  if (ctiles_h_.empty() && vtiles_h_.empty() && n_small_ > 0) return 5;
  if (ctiles_h_.empty() && vtiles_h_.empty() && !clusters_.empty())
    return prec_ == DMM_FP32 && !clusters_[0].general ? 4 : 3;
  if (ctiles_h_.empty() && vtiles_h_.empty() && gr_groups_.size() == 1)
    return prec_ == DMM_FP32 && !gr_general_ ? 4 : 3;
  if (xp_active_) return xp_mt_ ? 6 : 4;
  if (stream_active_) return !stream_general_ ? 6 : 3;
  if (one_active_) return 3;
  return 2;
}

int Pack::step_kernel() const {
  if (tun_.launch_mode != 1 && ctiles_h_.empty() && vtiles_h_.empty() && n_small_ == 0) {
    if (!clusters_.empty()) return 7;
    if (!gr_groups_.empty()) return 8;
  }
  return tun_.launch_mode != 1 && stream_active_ ? 9 : launch_form();
}

dmm_status Pack::trace_phases(int32_t nsteps, double* out) {
  DMM_CUDA(cudaSetDevice(dev_));
  TileForms tile_forms(*this, false);
  DMM_TRY(tile_forms.st);
  if (tun_.launch_mode == 1 || n_small_ > 0 || nsteps <= 0) {
    set_error("phase tracing needs the cooperative launch of tile-path formulas");
    return DMM_ERR_STATE;
  }
  constexpr int K = kTraceK;
  const bool grid = !gr_groups_.empty();
  const int G = grid ? gr_blocks_ : stream_active_ ? sms_ : grid_p_;
  const int64_t half = (int64_t)nsteps * K * G;
  // timer stamps, clock counts, then every block's entry and exit times (trace_launch)
  const int64_t need = 2 * half + 2 * G;
  if (need > trace_cap_) {
    if (trace_) retire(trace_);
    trace_ = nullptr;
    DMM_CUDA(dev_alloc(&trace_, need * sizeof(long long)));
    trace_cap_ = need;
  }
  DMM_CUDA(cudaMemsetAsync(trace_, 0, need * sizeof(long long), stream_));
  trace_on_ = true;
  trace_steps_ = nsteps;
  dmm_status st = grid ? launch_grid(nsteps) : launch_tiles(nsteps);  // one launch: trace step s = launch step s
  trace_on_ = false;
  DMM_TRY(st);
  std::vector<long long> h(need);
  DMM_CUDA(cudaMemcpyAsync(h.data(), trace_, need * sizeof(long long), cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  DMM_TRY(check_error());
  auto at = [&](int64_t s, int k, int b) { return h[(s * K + k) * G + b]; };
  double mean[K] = {}, mx[K] = {};
  int used = 0;
  // a step counts when every block stamped its start and the next step's start exists
  for (int32_t s = 0; s + 1 < nsteps; s++) {
    bool ok = true;
    for (int b = 0; b < G && ok; b++) ok = at(s, 0, b) != 0 && at(s + 1, 0, b) != 0;
    if (!ok) break;
    double sm[K] = {}, smx[K] = {};
    for (int b = 0; b < G; b++) {
      long long pts[K + 1];
      for (int k = 0; k < K; k++) {
        const long long v = at(s, k, b);
        pts[k] = v != 0 ? v : pts[k - 1];  // a block without a tile of the phase
      }
      pts[K] = at(s + 1, 0, b);
      for (int k = 0; k < K; k++) {
        const double d = (double)(pts[k + 1] - pts[k]);
        sm[k] += d;
        smx[k] = std::max(smx[k], d);
      }
    }
    for (int k = 0; k < K; k++) {
      mean[k] += sm[k] / G;
      mx[k] += smx[k];
    }
    used++;
  }
  for (int k = 0; k < K; k++) {
    out[2 * k] = used ? mean[k] / used / 1000.0 : 0.0;  // microseconds
    out[2 * k + 1] = used ? mx[k] / used / 1000.0 : 0.0;
  }
  // SM clock of block 0 over the traced steps
  out[2 * K] = 0.0;
  if (used > 0) {
    const long long t0 = at(0, 0, 0), t1 = at(used, 0, 0);
    const long long c0 = h[half + 0], c1 = h[half + (int64_t)used * K * G];
    if (t1 > t0) out[2 * K] = (double)(c1 - c0) / (double)(t1 - t0) * 1000.0;  // MHz
  }
  // launch entry to the first step, last step's end to exit (forms that stamp them)
  out[2 * K + 1] = out[2 * K + 2] = 0.0;
  for (int b = 0; b < G; b++) {
    const long long in = h[2 * half + b], ex = h[2 * half + G + b];
    if (in == 0 || ex == 0 || at(0, 0, b) == 0) continue;
    int32_t last = nsteps - 1;
    while (last > 0 && at(last, K - 1, b) == 0) last--;
    out[2 * K + 1] += (double)(at(0, 0, b) - in) / G / 1000.0;
    if (at(last, K - 1, b) != 0) out[2 * K + 2] += (double)(ex - at(last, K - 1, b)) / G / 1000.0;
  }
  return DMM_OK;
}

dmm_status Pack::profile_steps(int32_t nsteps, int64_t flush_bytes, StepTimes* t) {
  DMM_CUDA(cudaSetDevice(dev_));
  TileForms tile_forms(*this, true);
  DMM_TRY(tile_forms.st);
  if (flush_bytes > flush_cap_) {
    if (flush_) retire(flush_);
    flush_ = nullptr;
    DMM_CUDA(dev_alloc(&flush_, flush_bytes));
    flush_cap_ = flush_bytes;
  }
  for (int32_t s = 0; s < nsteps; s++) {
    if (flush_bytes > 0) {
      k_flush<<<sms_ * 4, kThreads, 0, stream_>>>(static_cast<int4*>(flush_), flush_bytes / 16, s);
      DMM_CUDA(cudaGetLastError());
    }
    DMM_CUDA(cudaEventRecord(ev_[0], stream_));
    DMM_TRY(enqueue_clause());
    DMM_CUDA(cudaEventRecord(ev_[1], stream_));
    DMM_TRY(enqueue_var(false, nullptr));
    DMM_CUDA(cudaEventRecord(ev_[2], stream_));
    DMM_CUDA(cudaEventSynchronize(ev_[2]));
    float a = 0, b = 0;
    DMM_CUDA(cudaEventElapsedTime(&a, ev_[0], ev_[1]));
    DMM_CUDA(cudaEventElapsedTime(&b, ev_[1], ev_[2]));
    t->clause_ms += a;
    t->var_ms += b;
    t->step_ms += a + b;
    t->launches += 2;
  }
  return DMM_OK;
}

dmm_status Pack::read_active(int32_t* active) {
  DMM_TRY(flush_adds());
  DMM_CUDA(cudaMemcpyAsync(active, active_d_, sizeof(int32_t), cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

dmm_status Pack::run(double wall_s, int64_t* steps_launched, bool* timed_out,
                     int32_t stop_after) {
  DMM_CUDA(cudaSetDevice(dev_));
  *timed_out = false;
  if (steps_launched) *steps_launched = 0;
  DMM_TRY(pinned());
  DMM_TRY(flush_adds());
  const auto t0 = std::chrono::steady_clock::now();
  auto elapsed = [&]() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  };
  // status words before the run and after each chunk of steps (two in turn)
  auto status = [&](int slot) { return pinned_ + 8 * slot; };
  auto fetch = [&](int slot) -> dmm_status {
    DMM_CUDA(cudaMemcpyAsync(status(slot), ring_tail_d_, kStatusInts * sizeof(int32_t),
                             cudaMemcpyDeviceToHost, stream_));
    return DMM_OK;
  };
  DMM_TRY(fetch(2));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  const int32_t tail0 = status(2)[0];
  if (status(2)[4] <= 0) return DMM_OK;
  const int32_t S = tun_.steps_per_graph * (cluster_only() ? kClusterChunk : 1);
  auto chunk = [&](int slot) -> dmm_status {
    DMM_TRY(launch_steps(S));
    DMM_TRY(fetch(slot));
    DMM_CUDA(cudaEventRecord(ev_[slot], stream_));
    if (steps_launched) *steps_launched += S;
    return DMM_OK;
  };
  int cur = 0;
  DMM_TRY(chunk(cur));
  for (;;) {
    const int nxt = cur ^ 1;
    DMM_TRY(chunk(nxt));
    DMM_CUDA(cudaEventSynchronize(ev_[cur]));
    if (status(cur)[4] <= 0 || status(cur)[5] != 0) break;
    if (stop_after > 0 && status(cur)[0] - tail0 >= stop_after) break;
    if (wall_s > 0 && elapsed() > wall_s) {
      *timed_out = true;
      break;
    }
    cur = nxt;
  }
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return status(cur ^ 1)[5] ? check_error() : DMM_OK;
}

dmm_status Pack::resume(int32_t idx) {
  InstCtrl c;
  DMM_TRY(read_ctrl(idx, &c));
  if (c.done != DMM_STEP_LIMIT) return DMM_OK;
  c.done = 0;
  DMM_TRY(add_active(+1));
  DMM_TRY(write_ctrl(idx, c));
  return DMM_OK;
}

dmm_status Pack::drain_finished(std::vector<int32_t>* out) {
  out->clear();
  int32_t tail = 0;
  DMM_CUDA(cudaMemcpyAsync(&tail, ring_tail_d_, sizeof(int32_t), cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  if (tail == ring_read_) return DMM_OK;
  std::vector<int32_t> ring(caps_.insts);
  DMM_CUDA(cudaMemcpy(ring.data(), ring_d_, caps_.insts * sizeof(int32_t), cudaMemcpyDeviceToHost));
  for (int32_t p = ring_read_; p < tail; p++) out->push_back(ring[p % caps_.insts]);
  ring_read_ = tail;
  return DMM_OK;
}

dmm_status Pack::stop(int32_t idx, int32_t status) {
  InstCtrl c;
  DMM_TRY(read_ctrl(idx, &c));
  if (c.done != 0) return DMM_OK;
  c.done = status;
  DMM_TRY(add_active(-1));
  DMM_TRY(write_ctrl(idx, c));
  return DMM_OK;
}

dmm_status Pack::sync() {
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return check_error();
}

dmm_status Pack::rhs(int32_t idx, const double* x, double* dxdt, int32_t* loc, double* energy) {
  if (!live(idx) || !x || !dxdt) return DMM_ERR_ARG;
  DMM_TRY(resolve_long_lists());
  DMM_TRY(set_state(idx, x));
  const InstDesc& I = inst_h_[idx];
  const int64_t N = (int64_t)I.n + 2 * (int64_t)I.m;
  DMM_TRY(ensure_stage(N));
  // tiles of this instance only
  std::vector<Tile> ct, vt;
  // the right-hand side runs the kernel-per-phase form with its own fixed tiles
  const int TC = 4 * kThreads, TV = kThreads;
  for (int32_t b = 0; b < I.m; b += TC) ct.push_back(Tile{idx, b, std::min(TC, I.m - b), 0});
  for (int32_t b = 0; b < I.n; b += TV) vt.push_back(Tile{idx, b, std::min(TV, I.n - b), 0});
  const int64_t need = std::max<int64_t>(std::max(ct.size(), vt.size()), 1);
  if (need > aux_cap_) {
    if (aux_ctiles_d_) retire(aux_ctiles_d_);
    if (aux_vtiles_d_) retire(aux_vtiles_d_);
    aux_ctiles_d_ = aux_vtiles_d_ = nullptr;
    DMM_CUDA(dev_alloc(&aux_ctiles_d_, need * sizeof(Tile)));
    DMM_CUDA(dev_alloc(&aux_vtiles_d_, need * sizeof(Tile)));
    aux_cap_ = need;
  }
  if (!ct.empty())
    DMM_CUDA(cudaMemcpyAsync(aux_ctiles_d_, ct.data(), ct.size() * sizeof(Tile),
                             cudaMemcpyHostToDevice, stream_));
  DMM_CUDA(cudaMemcpyAsync(aux_vtiles_d_, vt.data(), vt.size() * sizeof(Tile),
                           cudaMemcpyHostToDevice, stream_));
  int32_t nt[2] = {(int32_t)ct.size(), (int32_t)vt.size()};
  DMM_CUDA(cudaMemcpyAsync(ntiles_d_ + 2, nt, sizeof nt, cudaMemcpyHostToDevice, stream_));
  // the finalize of a right-hand side reads the epart of the auxiliary tiles
  InstDesc Iaux = I;
  Iaux.ctile0 = 0;
  Iaux.nctile = nt[0];
  DMM_CUDA(cudaMemcpyAsync(inst_d_ + idx, &Iaux, sizeof(InstDesc), cudaMemcpyHostToDevice, stream_));
  const int gc = grid_c_, gv = grid_v_;
  grid_c_ = std::max(1, std::min(nt[0], sms_ * 8));
  grid_v_ = std::max(1, std::min(nt[1], sms_ * 8));
  use_aux_ = true;
  dmm_status st = enqueue_step(true, stage_);
  use_aux_ = false;
  grid_c_ = gc;
  grid_v_ = gv;
  DMM_TRY(st);
  if (prec_ == DMM_FP64)
    k_clause_dx<double><<<blocks_for(I.m), kThreads, 0, stream_>>>(
        inst_d_, idx, static_cast<double*>(Xs_), static_cast<double*>(Cp_),
        static_cast<double*>(alpha_cm_), stage_);
  else
    k_clause_dx<float><<<blocks_for(I.m), kThreads, 0, stream_>>>(
        inst_d_, idx, static_cast<float*>(Xs_), static_cast<float*>(Cp_),
        static_cast<float*>(alpha_cm_), stage_);
  DMM_CUDA(cudaGetLastError());
  k_rhs_finish<<<1, kThreads, 0, stream_>>>(inst_d_, ctrl_d_, idx, epart_);
  DMM_CUDA(cudaGetLastError());
  DMM_TRY(upload_desc(idx));
  InstCtrl c;
  DMM_TRY(pinned());
  DMM_CUDA(cudaMemcpyAsync(pinned_ + 64, ctrl_d_ + idx, sizeof(InstCtrl), cudaMemcpyDeviceToHost,
                           stream_));
  DMM_TRY(download_state(dxdt, stage_, N));
  std::memcpy(&c, pinned_ + 64, sizeof c);
  if (loc) *loc = c.loc;
  if (energy) *energy = c.energy;
  return DMM_OK;
}

dmm_status Pack::dostep(int32_t idx, const double* x, const double* dxdt, double h, double* xo) {
  if (!live(idx) || !x || !dxdt || !xo) return DMM_ERR_ARG;
  DMM_TRY(flush_adds());
  const InstDesc& I = inst_h_[idx];
  const int64_t N = (int64_t)I.n + 2 * (int64_t)I.m;
  DMM_TRY(ensure_stage(3 * N));
  DMM_TRY(upload_doubles(stage_, x, N));
  DMM_TRY(upload_doubles(stage_ + N, dxdt, N));
  if (prec_ == DMM_FP64)
    k_dostep<double><<<blocks_for(N), kThreads, 0, stream_>>>(inst_d_, idx, unit_, stage_,
                                                              stage_ + N, h, stage_ + 2 * N);
  else
    k_dostep<float><<<blocks_for(N), kThreads, 0, stream_>>>(inst_d_, idx, unit_, stage_,
                                                             stage_ + N, h, stage_ + 2 * N);
  DMM_CUDA(cudaGetLastError());
  return download_state(xo, stage_ + 2 * N, N);
}

dmm_status Pack::assignments(const std::vector<int32_t>& idx, std::vector<int8_t>* out) {
  DMM_TRY(flush_adds());
  std::vector<int64_t> off(idx.size());
  int64_t total = 0;
  for (size_t k = 0; k < idx.size(); k++) {
    if (!live(idx[k])) return DMM_ERR_ARG;
    off[k] = total;
    total += inst_h_[idx[k]].n;
  }
  out->resize((size_t)total);
  if (idx.empty()) return DMM_OK;
  // [offsets | indices | signs] in the staging buffer
  const int64_t o_idx = (int64_t)idx.size() * 8, o_out = o_idx + (((int64_t)idx.size() * 4 + 15) & ~15);
  DMM_TRY(ensure_stage((o_out + total + 7) / 8));
  unsigned char* base = reinterpret_cast<unsigned char*>(stage_);
  DMM_CUDA(cudaMemcpyAsync(base, off.data(), off.size() * 8, cudaMemcpyHostToDevice, stream_));
  DMM_CUDA(cudaMemcpyAsync(base + o_idx, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice, stream_));
  int8_t* dst = reinterpret_cast<int8_t*>(base + o_out);
  const auto* di = reinterpret_cast<const int32_t*>(base + o_idx);
  const auto* doff = reinterpret_cast<const int64_t*>(base);
  int32_t most = 1;
  for (int32_t i : idx) most = std::max(most, inst_h_[i].n);
  const dim3 grid((unsigned)idx.size(), (unsigned)std::min((most + 4 * kThreads - 1) / (4 * kThreads), 64));
  if (prec_ == DMM_FP64)
    k_signs_all<double><<<grid, kThreads, 0, stream_>>>(
        inst_d_, ctrl_d_, di, doff, static_cast<const double*>(cand_), caps_.vars, dst);
  else
    k_signs_all<float><<<grid, kThreads, 0, stream_>>>(
        inst_d_, ctrl_d_, di, doff, static_cast<const float*>(cand_), caps_.vars, dst);
  DMM_CUDA(cudaGetLastError());
  DMM_CUDA(cudaMemcpyAsync(out->data(), dst, (size_t)total, cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  return DMM_OK;
}

dmm_status Pack::assignment(int32_t idx, int8_t* pre, int8_t* post) {
  if (!live(idx)) return DMM_ERR_ARG;
  DMM_TRY(flush_adds());
  if (!pre && !post) return DMM_OK;
  const InstDesc& I = inst_h_[idx];
  // [flag | pre (n) | post (n)] in the staging buffer
  DMM_TRY(ensure_stage(1 + (2 * (int64_t)I.n + 7) / 8));
  int32_t* flag = reinterpret_cast<int32_t*>(stage_);
  int8_t* dpre = reinterpret_cast<int8_t*>(stage_) + 8;
  int8_t* dpost = dpre + I.n;
  DMM_CUDA(cudaMemsetAsync(flag, 0, sizeof(int32_t), stream_));
  if (prec_ == DMM_FP64)
    k_signs<double><<<blocks_for(I.n), kThreads, 0, stream_>>>(
        ctrl_d_ + idx, static_cast<const double*>(cand_), caps_.vars, I.var0, I.n,
        pre ? dpre : nullptr, post ? dpost : nullptr, flag);
  else
    k_signs<float><<<blocks_for(I.n), kThreads, 0, stream_>>>(
        ctrl_d_ + idx, static_cast<const float*>(cand_), caps_.vars, I.var0, I.n,
        pre ? dpre : nullptr, post ? dpost : nullptr, flag);
  DMM_CUDA(cudaGetLastError());
  int32_t not_solved = 0;
  DMM_CUDA(cudaMemcpyAsync(&not_solved, flag, sizeof(int32_t), cudaMemcpyDeviceToHost, stream_));
  if (pre) DMM_CUDA(cudaMemcpyAsync(pre, dpre, I.n, cudaMemcpyDeviceToHost, stream_));
  if (post) DMM_CUDA(cudaMemcpyAsync(post, dpost, I.n, cudaMemcpyDeviceToHost, stream_));
  DMM_CUDA(cudaStreamSynchronize(stream_));
  if (pre && not_solved) {
    set_error("instance %d is not solved", idx);
    return DMM_ERR_STATE;
  }
  return DMM_OK;
}

}  // namespace dmm
