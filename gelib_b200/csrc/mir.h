// Mirrored-row and row-pair kernels: products in which every channel of the output has its own pair of input columns (column =
// (cell, channel), see col.h).  Forward (mir_fwd.cu), at every batch except for types of a handful of items on many columns:
//
//   r_l[m] (+)= sum_{m1} C_l[m1, m-m1] x_l1[m1] y_l2[m-m1],     C_l[-m1,-m2] = (-1)^(l1+l2-l) C_l[m1,m2]
//
// An item is a pair (l1,l2), up to kMirMaxNl output l and the two output rows m and -m, which share their coefficients up
// to that sign: band entry i multiplies x[i] y[m-i] and x[-i] y[-(m-i)], and one coefficient serves both.  In row 0 the two
// products are entries of the same row: entries i >= 0 are walked, the two sums are added at the end, and the coefficient of
// entry 0, which meets itself, is halved.
// The inner loop runs over the band with every operand in shared memory and is instantiated per number of output l only, so the
// code is small, nothing is padded to a block size, and nothing is computed outside the band.
// The gradient of y for a one-channel x (mir_bwd.cu), on a full chip and where it measured faster, walks items of two
// neighbouring rows in the same manner.
#pragma once
#include "col.h"

namespace gelib_b200 {

constexpr int kMirMaxNl = 8;  // output l per item
constexpr int kMirMaxL = 8;          // the smaller l of a pair

struct MirArgs {
  ColPart x[kMaxParts], y[kMaxParts], r[kMaxParts];  // r: base with the call's channel offset
  unsigned char xl[kMaxParts], yl[kMaxParts];
  int nx, ny, nr;
  int xrows, yrows;      // staged rows
  unsigned n, ncols;     // channels of a cell, columns in all
  int one_channel;       // x has one channel, y more
  int xcells;            // most cells that the columns of a block touch
  int item_bytes;        // largest item
  int accumulate;
  const int4* items;     // per item {header, records, coefficients}
  const int2* dir;       // per item {first int4, int4 units}
  int nitems;
};

// Gradient of y.
struct MirBwdArgs {
  ColPart x[kMaxParts], yg[kMaxParts], g[kMaxParts];
  unsigned char xl[kMaxParts];
  int nx, nr;
  int y_rows;            // most rows of a y part
  int ring_bytes;        // of the item tables in shared memory
  unsigned n, ncols;     // channels of a cell, columns in all
  int xcells;            // most cells that the columns of a warp touch
  const int4* items;     // per item {header, records, coefficients}
  const int2* dir;       // per item {first int4, int4 units | place in the ring << 8}
  int nitems;
};
// Flags of a backward item: only row m has the first entry, only row m + 1 the last; a row m alone; first and last of an l2;
// last of a pair.
enum { kMirPrologue = 1, kMirEpilogue = 2, kMirSingle = 4, kMirFirstOfB = 8, kMirLastOfB = 16, kMirLastOfPair = 32 };
constexpr int kMirTwoLevels = 6;  // most output l of an item for which the sums of a pair are kept apart

#ifdef __CUDACC__
namespace mir {
__device__ __forceinline__ uint32_t sptr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
}  // namespace mir
#endif

}  // namespace gelib_b200
