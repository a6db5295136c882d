// Column kernels: products in which every channel of the output has its own pair of input columns -- the diagonal
// product, and the full product when x has one channel (the spherical harmonics of a first layer).  With "column" =
// (cell, channel) both are
//
//   r_l[m] (+)= sum_{m1} C_l[m1, m-m1] x_l1[m1] y_l2[m-m1]
//   G[m1,m2] = sum_l C_l[m1,m2] g_l[m1+m2];   xg[m1] += G conj(y[m2]);   yg[m2] += G conj(x[m1])
//
// and a lane that owns a column needs nothing from any other lane.
//
// Organisation.  A warp owns 32 lanes of columns (two adjacent channels per lane where alignment allows, else one) and
// walks the (l1,l2) pairs; the part with the smaller l is the pair's "a" side, the other its "b" side.  The rows of the
// b part at work, and their gradients, sit in shared memory in slots that belong to the lane; up to eleven a rows (a
// block) and their gradients sit in registers.  The pair is walked by output row m: entry i of a step multiplies a[i]
// with b[m - m1(i)].  The gradients of the b rows that a step touches are a window of registers that moves by one row per
// step (the body is instantiated per block size, so everything in registers is indexed statically); a row is added to its
// slot when it leaves the window.  There are no atomics in shared memory and no shuffles, no barriers within a chunk of the
// walk (below), and one read-modify-write per row and block instead of one per band entry.
// Everything a warp reads from global memory -- b rows, a rows, the gradient rows g -- arrives through one stream of rows
// (cp.async, 8 or 16 bytes per lane) in a ring of kColRing rows, whose order is the order of use: taking k rows requests
// the k rows that come kColRing later, so the bytes in flight do not depend on how short the steps are.  What the warps
// of a block share is the walk itself: a chunk (row addresses, step records, coefficients) is copied to shared memory one chunk ahead.
// Gradient rows are added to global memory with red.  Unless an operand is broadcast over cells (stride 0) a row belongs to
// one lane of one block, so the sums have one order and gradients are bitwise repeatable.  Calls with few columns split the
// walk over blocks; in the backward by gradient rows ("owned": the blocks of a cluster walk everything that is added to the
// rows of their group, in which either part of a pair may be the larger one, and sum at the end in the order of their ranks).
// Diagonal products of more than 16 channels and one-channel x with more than 32, which no other kernel sums in one order,
// may instead split by pairs, and then several blocks add to a row.
// Why this form: diag_bwd_cell_kernel spends its time in four shared-memory atomics (compare-and-swap loops) per band
// entry, which a lane that owns its column does not need.  Measured, backward of the diagonal product: maxl 8 x 128
// channels, batch 2048 10.5 -> 4.7 ms; maxl 6 x 33, batch 4000 4.3 -> 1.0 ms; maxl 3 x 12, batch 500 49 -> 29 us (forward 32 ->
// 15 us).  At maxl 8 the backward holds two warps per scheduler -- 242 registers a thread and 25.6 KB of shared memory a warp
// both end there -- and issues in 43 % of its cycles: 494 k warp instructions per 64 columns, whose largest stalls are
// fixed-latency dependencies (1.3 cycles per issue) and shared memory (0.7).  The forward issues in 32 %: 345 k
// instructions, dependencies 1.5, shared memory 1.3, instruction fetch of the unrolled bodies 1.1; its instances spill 84 to
// 168 bytes a thread at 168, 128 and 128 registers, which its block sizes impose.
#pragma once
#include "plan.h"

namespace gelib_b200 {

constexpr int kColRing = 16;                    // rows in flight per warp (a power of two)
constexpr int kColMaxNl = 10;                   // output l per step; pairs with more are walked twice
constexpr int kColMaxLa = 8;                    // largest l of an a side
constexpr int kColBlockBwd = 11;                // a rows per block, backward (registers: a and its gradient, the window)
constexpr int kColBlockFwd = 17;                // a rows per block, forward
constexpr int kColChunkBytes = 13312;           // capacity of a chunk buffer
constexpr int kColMaxSmem = 232448;
constexpr int kColSumRows = 48;                 // gradient rows that the blocks of a cluster sum (owned walks)
constexpr int kColSlots = 3 * kMaxParts;        // x parts, y parts, r (g) parts
constexpr int kColFixedSmem = 16 * kColSlots + 2 * kColChunkBytes;  // part table, chunk buffers

// Output l that a step of nl is worked on with (zero coefficients beyond nl): the body of a step is instantiated per block
// size and for each of these numbers.  With both gradients the bodies are long and fetching them is what costs most, so
// large blocks have two instances, 6 and 10, that stay in the instruction cache: maxl 8 x 128 channels, batch 2048 5.9 ms
// with 2, 4, .. 10, 4.8 ms with 6 and 10, 5.3 ms with 10 alone.  With one gradient, or
// forward, the added multiply-adds cost more than that: one-channel x, maxl 4 x 32, 30000 cells 1.33 against 1.45 ms;
// forward, maxl 8 x 128 3.8 against 4.3 ms.
constexpr int col_nl_padded(int nl, int kb, bool both) { return !both || kb < 6 ? (nl + 1) / 2 * 2 : nl <= 6 ? 6 : 10; }

// Row (slot, v) of a lane: base + v * unit + cell * cell_stride + (lane of the cell) * ch_stride, all in bytes.
struct ColPart {
  float* base;
  unsigned unit, cell_stride;
};

struct ColArgs {
  ColPart part[kColSlots];         // x: 0.., y: kMaxParts.., r or g: 2 kMaxParts..  (v = row for x, y; complex offset for r)
  ColPart grad[2 * kMaxParts];     // xg: 0.., yg: kMaxParts..  (v = row)
  unsigned ch_stride[3];           // bytes between lanes of x, y, r: 8 per column, or 0 for an operand of one channel
  unsigned n, nlanes;              // lanes per cell (channels / columns per lane), lanes in all
  int b_rows;                      // rows of the largest b part
  int accumulate;                  // forward: add to r instead of storing
  const int4* blob;
  const int* chunks;               // per run {first chunk, number of chunks, first record of the ring prologue, list of the
                                   // rows that its group sums}, then per chunk {offset, size} in int4 units
  int nsplits;                     // runs
  int cluster, sum_rows;           // owned walks: blocks that sum rows together, rows of a lane's sums
};

struct ColPlan {
  DevicePlan* dev;
  int max_block;  // a rows of the largest block
  int cpl;        // columns per lane
  bool owned;     // backward with few columns: the walk is cut by gradient rows
  int warps;      // of a block, for an owned walk
  bool plan_others;  // first use of a signature that goes to other kernels at other batch sizes: they should plan it too
};

// Bits of a segment record.
enum { kColFirstOfB = 1, kColLastOfB = 2, kColLastOfChunk = 4, kColLast = 8, kColDrain = 16, kColHalf1 = 32 };

// Warps per block, at most `most`: an SM holds one block, so when one wave of blocks is enough its warps are spread over
// all SMs instead of filling some of them.
inline int col_block_warps(unsigned warps, int splits, int most) {
  const long long total = (long long)warps * splits;
  if (total >= 148LL * most) return most;
  const long long nw = (total + 147) / 148;
  return (int)(nw < 2 ? 2 : nw);
}

// False when the view's cells are no arithmetic progression or a stride does not fit.
bool col_fill_part(const PartView& p, const CellGrid& cg, long long extra_floats, bool rows, ColPart* out);

// One-channel x: whether the kernels of cg_narrow.cu / cg_narrow1_bwd.cu are faster than the column kernels, which take cpl
// columns per lane; max_la: largest min(l1, l2).
bool narrow_wins(bool backward, int cpl, int n, int max_la, long long cells);

// Returns false when the call is not one the column kernels take; otherwise fills args and
// plan (plan->dev == nullptr on a CUDA error).
bool col_setup(const VecCall& c, bool backward, ColArgs* a, ColPlan* plan);

}  // namespace gelib_b200
