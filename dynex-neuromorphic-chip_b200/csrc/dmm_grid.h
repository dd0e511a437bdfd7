// Host interface of the resident grid form (dmm_grid.cuh, dmm_gridprep.cuh, grid.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "dmm_device.cuh"

namespace dmm {

constexpr int kGridThreads = 512;    // block size
constexpr int kGridThreads64 = 512;  // ... in FP64 (the sorted sums' registers)
constexpr int kGridSmemMax = 222 * 1024;  // dynamic shared memory, at most
constexpr int kGridMaxTiles = 24;         // clause or variable tiles of a block
constexpr int kGridMaxDistinct = 32767;   // 16-bit tile-local literals

// One formula of a launch: B blocks of the grid from blk0 on, each with kc clause tiles of TC
// clauses and kv variable tiles of TV variables.  The o_* are where its part of each shared
// table array starts (elements).
struct GridGroup {
  int32_t inst, blk0, B, kc, kv, TC, TV, TVr;  // TVr: TV rounded up to 32 (table rows)
  int32_t nct, nvt;                            // B * kc, B * kv
  int32_t lt, NL, list0;                       // clause tiles per variable list, lists, first one
  int32_t pad;                                 // entries that chunks of ux are padded to
  int32_t n, m, L, k3;
  int64_t var0, cls0, slot0;
  int64_t o_pair, o_blk, o_ct, o_vt, o_list, o_slot, o_ux, o_word, o_row, o_push, o_bb, o_var,
      o_cls;
};

// Table arrays of all groups.
struct GridTables {
  // built at commit, read by the steps
  int32_t* dlist;   // [o_list] distinct variables of each list, ascending; the part of every
                    // owning block is padded to whole 16-byte words of voltages (with -1)
  int2* dinfo;      // [o_blk + l] start and count of list l in dlist and in the inbox
  int16_t* llit;    // [o_slot + s] list-local literal, +-(1 + place in the list)
  uint16_t* spos;   // [o_slot + s] place in the tile's staging area
  uint32_t* wdst;   // [o_word + w] 16-byte word of ux each staging word goes to
  int32_t* woff;    // [o_ct + t] first staging word of each clause tile (nct + 1 of them)
  int32_t* boff;    // [o_vt + v] start of each variable tile's bucket in ux (nvt + 1)
  uint16_t* rows;   // [o_row] bucket places of each variable's first 32 contributions
  uint16_t* idx;    // [o_slot + j] bucket place of the contribution in CSR position j
  // FP64: variables of a tile in order of falling list length (null: in their own order)
  uint16_t* pos;    // [o_var + v] place of variable v in its tile
  uint16_t* perm;   // [o_var + tile TV + place] variable of the tile
  // general clauses: those of a tile in order of falling length (null: all have three literals)
  uint16_t* cord;   // [o_cls + tile TC + place] clause of the tile
  int2* sinfo;      // [o_blk + b] start and count of block b's send words
  uint16_t* ids;    // [(o_push + word) kw] block-local variables of a send word
  uint32_t* sdst;   // [o_push + word] inbox word it goes to
  // exchanged within a step, each twice (steps of even and odd number): unset entries hold a
  // value no arithmetic gives
  void* ux;         // [2 o_ux] contributions, bucket after bucket
  void* inbox;      // [2 o_list] dV of each block's distinct variables
  int64_t ux_len, inbox_len;  // elements of one copy
  // scratch of the build
  int32_t *cnt, *sb, *bt;       // [o_pair]
  int32_t *st, *dcnt;           // [o_ct], [o_blk]
  int32_t *dlo, *dlp, *poff;    // [o_bb]: variables below a block, padded; chunk's send words
  int32_t *btot, *ptot;         // [o_vt], [o_blk]
  int32_t* out;                 // [8 x group]
};

// Results of the build, per group: [0] 0 ok, else which limit failed; [1] largest distinct
// list, [2] largest staging area, [3] largest bucket, [4] largest send list (words), [5]
// largest literal-slot count of a block.
constexpr int kGridOut = 8;

struct GridCaps {
  int dl;      // distinct variables of a block (a multiple of 4)
  int st, bk;  // staging entries, bucket entries
  int tv;      // variables of a block
  int B;       // blocks of a group
  // resident tables: clauses, slots, staging words, table rows, CSR entries, sends of a block
  int tc, ts, wd, row, csr, snd;
};

constexpr int kGridSyncBytes = 256;  // per group
// Byte offsets of a block's dynamic shared memory.
struct GridLayout {
  int sv, raw, cur, dv, vend, unit, rank;
  int xs, xl, cp, lit, spos, off, ord, wdst, row, csr, snd, total;
};

// resident: 0 no tables in shared memory, 1 those of the variable phase, 2 all and the clause
// memories
GridLayout grid_shape(const GridCaps& c, bool fp64, bool general, int resident);
inline int grid_smem(const GridCaps& c, bool fp64, bool general, int resident) {
  return grid_shape(c, fp64, general, resident).total;
}
const void* grid_kernel(bool fp64, bool general, int resident);
// The kernels of the form in one precision, its table build included.
void grid_functions(bool fp64, std::vector<const void*>* out);
// Queues the marking of all exchange entries as unset.
cudaError_t grid_unset(const GridTables& t, bool fp64, cudaStream_t s);
// Queues the table build of all groups (list_group: group of every list).
cudaError_t grid_build(const GridGroup* groups, const int32_t* list_group, int ngroups,
                       int nlists, int max_n, int max_nct, int max_nvt, int max_rows, const int32_t* lit,
                       const int32_t* upos, const int32_t* vend, const int32_t* coff,
                       const GridTables& t, bool fp64, cudaStream_t s);

// ---- streaming form (dmm_stream.cuh), FP32
constexpr int kStreamThreads = 1024;  // block size
constexpr int kStreamSmemMax = 222 * 1024;
struct StreamLayout {
  int v0, v1, stage;  // A: two voltage lists (one in use, one arriving), staging area
  int b0, b1;         // B: two buckets, each behind one padding word
  int total;          // C: the block's voltages, from 0
};
StreamLayout stream_shape(int dl, int st, int bk, int tv);
const void* stream_kernel(bool general);

}  // namespace dmm
