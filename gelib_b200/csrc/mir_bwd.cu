// Gradient of y in the product with a one-channel x that needs no gradient itself (a first layer on spherical harmonics), for
// calls that fill the chip:
//
//   H[m1,m2][n2] = sum_l C_l[m1,m2] g_l[m1+m2][n2]  (every output l of the pair (l1,l2) at once);   yg[m2] += H conj(x[m1])
//
// A lane owns a column (cell, n2), a warp is a block: warps are independent, and as many as fit share an SM.  A warp walks the
// items -- a pair, the rows m and m + 1, every output l -- in the order of l2, whose gradient rows it keeps in shared memory,
// one slot per lane, until the last item of that l2.  Entry i of row m and entry i of row m + 1 share x[i], and what entry i of
// row m adds to, yg[m-i], is what row m + 1 adds to at entry i + 1: the sum passes on in a register and a slot is read and
// written once for two products.  Where only one of the rows has an entry (the ends of the bands) only that one is worked on.
// The loop is instantiated per number of output l.  While it works on an item a warp loads the g rows of the next into
// registers, asks those of the one after into the L2, and copies the tables of the third (cp.async).
//
// Measured, a million columns, against cg_narrow1_bwd_kernel: maxl 6 x 16 5.05 -> 4.33 ms, maxl 6 x 32 4.87 -> 4.28; against the column
// kernel: maxl 3 x 9 1.10 -> .77, maxl 5 x 16 3.02 -> 2.73 (row_pairs_from).  Bound by issue and latency: 106 k warp instructions per 32
// columns at maxl 6, of which the band loops are 40 %, issued in 58 % of the cycles.  Measured on maxl 6 x 16, 65536 cells, 4580 us: without the request into the L2
// 5310, at 16 warps instead of 20 4970, at 24, which spills, 5420; two columns per lane (187 registers, 11 warps) 6790.
#include <algorithm>
#include <cstring>
#include <map>

#include "f32x2.h"
#include "mir.h"

namespace gelib_b200 {
namespace mir {

constexpr int kPitch = 256;  // bytes of a row of the warp's 32 columns

// Where an item stands: entry i of the band meets x[i] and the slot of yg[m - i].
struct Band {
  const float4* cf;  // coefficients of row m, then of row m + 1
  const unsigned char* x;
  unsigned char* yg;
};

// Band entry i of rows m (R0) and m + 1 (R1).  acc: what yg[m + 1 - i] has got from row m; on return it belongs to yg[m - i].
template <int NL, bool R0, bool R1>
__device__ __forceinline__ void entry(Band& B, int xpitch, const f32x2* g0, const f32x2* g1, float2& acc) {
  constexpr int P = (2 * NL + 3) / 4;
  f32x2 q[4 * P];
#pragma unroll
  for (int k = 0; k < P; k++) {
    const float4 v = B.cf[k];
    q[4 * k] = pack2(v.x, v.x);
    q[4 * k + 1] = pack2(v.y, v.y);
    q[4 * k + 2] = pack2(v.z, v.z);
    q[4 * k + 3] = pack2(v.w, v.w);
  }
  const float2 x = *reinterpret_cast<const float2*>(B.x);
  float2* slot = reinterpret_cast<float2*>(B.yg + kPitch);
  float2 t;
  if (R1) t = *slot;
  f32x2 h0, h1;
#pragma unroll
  for (int j = 0; j < NL; j++) {
    if (R0) h0 = j == 0 ? mul2(q[0], g0[0]) : fma2(q[j], g0[j], h0);
    if (R1) h1 = j == 0 ? mul2(q[NL], g1[0]) : fma2(q[NL + j], g1[j], h1);
  }
  float ur, ui;
  if (R1) {
    unpack2(h1, ur, ui);
    acc.x = fmaf(ur, x.x, acc.x); acc.x = fmaf(ui, x.y, acc.x);
    acc.y = fmaf(ui, x.x, acc.y); acc.y = fmaf(-ur, x.y, acc.y);
    *slot = make_float2(t.x + acc.x, t.y + acc.y);
  }
  if (R0) {
    unpack2(h0, ur, ui);
    acc = make_float2(fmaf(ui, x.y, ur * x.x), fmaf(-ur, x.y, ui * x.x));
  }
  B.cf += P;
  B.x += xpitch;
  B.yg -= kPitch;
}
__device__ __forceinline__ void add_last(const Band& B, float2 acc) {
  float2* slot = reinterpret_cast<float2*>(B.yg + kPitch);
  const float2 t = *slot;
  *slot = make_float2(t.x + acc.x, t.y + acc.y);
}

template <int NL>
__device__ __forceinline__ void run_item(Band B, int flags, int cnt, int xpitch, const f32x2* g0, const f32x2* g1) {
  float2 acc = make_float2(0.f, 0.f);
  if (flags & kMirPrologue) entry<NL, true, false>(B, xpitch, g0, g1, acc);
#pragma unroll 1
  for (int k = 0; k < cnt; k++) entry<NL, true, true>(B, xpitch, g0, g1, acc);
  if (flags & kMirEpilogue) entry<NL, false, true>(B, xpitch, g0, g1, acc);
  else add_last(B, acc);
}
// A single row m, which one output l has.
__device__ __forceinline__ void run_single(Band B, int cnt, int xpitch, const f32x2* g0) {
  for (int k = 0; k < cnt; k++) {
    float2 acc;
    entry<1, true, false>(B, xpitch, g0, g0, acc);
    add_last(B, acc);
  }
}

__device__ __forceinline__ f32x2 ldg(const float2* p) {
  const float2 q = __ldcs(p);
  return pack2(q.x, q.y);
}
// The g rows of an item.  Of the output l, in ascending order, only the first may have one of the two rows alone.
template <int NL>
__device__ __forceinline__ void load_rows(const unsigned char* it, const unsigned long long* ptr, f32x2* n0, f32x2* n1) {
#pragma unroll
  for (int j = 0; j < NL; j++) {
    const int4 r = *reinterpret_cast<const int4*>(it + 16 + 16 * j);  // {part, offset of row m, rows there are, row pitch}, in complex numbers
    const float2* q = reinterpret_cast<const float2*>(ptr[32 * r.x]) + r.y;
    if (j == 0) {
      n0[0] = n1[0] = 0ull;
      if (r.z & 1) n0[0] = ldg(q);
      if (r.z & 2) n1[0] = ldg(q + r.w);
    } else {
      n0[j] = ldg(q);
      n1[j] = ldg(q + r.w);
    }
  }
}
// Asks the lines of an item's g rows where the warp's columns 0 and 16 lie into the L2, one line per lane.
__device__ __forceinline__ void prefetch_rows(const unsigned char* it, const unsigned long long* ptr) {
  const int lane = threadIdx.x, l = lane >> 2, row = (lane >> 1) & 1;
  if (l < (int)*it) {
    const int4 r = *reinterpret_cast<const int4*>(it + 16 + 16 * l);
    const float2* q = reinterpret_cast<const float2*>(ptr[32 * r.x + 16 * (lane & 1)]) + r.y + (row ? r.w : 0);
    if (r.z & (1 << row)) asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
  }
}

#define GELIB_MIR_SWITCH(nl, BODY) \
  switch (nl) {                    \
    case 1: BODY(1) break;         \
    case 2: BODY(2) break;         \
    case 3: BODY(3) break;         \
    case 4: BODY(4) break;         \
    case 5: BODY(5) break;         \
    case 6: BODY(6) break;         \
    case 7: BODY(7) break;         \
    case 8: BODY(8) break;         \
    default: break;                \
  }

// Two levels: a pair's sums are kept apart and added to those of the pairs before it when the pair ends, as the column kernel sums;
// with up to six l there is room for them.  Error against 64-bit sums, in one level / in two / of the column kernel: maxl 4 x 16
// 1.18e-7 / 0.78e-7 / 0.84e-7, maxl 5 x 16 1.03e-7 / 0.82e-7 / 0.91e-7 (a million columns 2.54 / 2.73 ms).
// NLMAX: most output l of an item.  WARPS: warps that should share an SM; more of them cover the latency of the loads better,
// and registers beyond these numbers bought nothing.
template <int NLMAX, int WARPS>
__global__ void __launch_bounds__(32, WARPS) mir_bwd_kernel(const __grid_constant__ MirBwdArgs A) {
  constexpr bool TWO_LEVELS = NLMAX <= kMirTwoLevels;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x;
  unsigned col = blockIdx.x * 32 + lane;
  const bool ok = col < A.ncols;
  if (!ok) col = A.ncols - 1;
  const unsigned cell = col / A.n, ch = col - cell * A.n, cell0 = blockIdx.x * 32 / A.n;
  // [addresses of the lanes' columns in every g part][ring of item tables][slots of the gradient rows][x rows, one number per cell]
  unsigned long long* ptr = reinterpret_cast<unsigned long long*>(smem);
  unsigned char* ring = smem + 256 * A.nr;
  unsigned char* yg = ring + A.ring_bytes + 8 * lane;
  unsigned char* total = yg + (TWO_LEVELS ? kPitch * A.y_rows : 0);
  unsigned char* xs = ring + A.ring_bytes + kPitch * A.y_rows * (TWO_LEVELS ? 2 : 1);
  const int xpitch = 8 * A.xcells;

  auto dir = [&](int i) { return i < A.nitems ? __ldg(A.dir + i) : make_int2(0, 0); };
  auto table = [&](int2 e) { return ring + 16 * (e.y >> 8); };
  auto fetch = [&](int2 e) {
    const uint32_t dst = sptr(table(e));
    for (int k = lane; k < (e.y & 255); k += 32) cp_async<16>(dst + 16 * k, A.items + e.x + k);
  };
  int2 d0 = dir(0), d1 = dir(1), d2 = dir(2), d3 = dir(3);
  fetch(d0);
  fetch(d1);
  fetch(d2);
  for (int p = 0; p < A.nr; p++)
    ptr[32 * p + lane] = reinterpret_cast<unsigned long long>(A.g[p].base) + (unsigned long long)cell * A.g[p].cell_stride + 8ull * ch;
  const unsigned last = (A.ncols - 1) / A.n;
  for (int i = 0, row = 0; i < A.nx; row += 2 * A.xl[i] + 1, i++)
    for (int e = lane; e < (2 * A.xl[i] + 1) * A.xcells; e += 32) {
      const int m = e / A.xcells, c = e - m * A.xcells;
      cp_async<8>(sptr(xs) + xpitch * (row + m) + 8 * c, reinterpret_cast<const unsigned char*>(A.x[i].base) +
                                                             (unsigned long long)min(cell0 + c, last) * A.x[i].cell_stride +
                                                             (unsigned long long)m * A.x[i].unit);
    }
  cp_wait_all();
  __syncwarp();
  xs += 8 * (cell - cell0);

  f32x2 g0[NLMAX], g1[NLMAX], n0[NLMAX], n1[NLMAX];
#define GELIB_MIR_LOAD(N) if constexpr (N <= NLMAX) load_rows<N>(next, ptr + lane, n0, n1);
#define GELIB_MIR_COPY(N)                               \
  if constexpr (N <= NLMAX) {                           \
    _Pragma("unroll") for (int j = 0; j < N; j++) {     \
      g0[j] = n0[j];                                    \
      g1[j] = n1[j];                                    \
    }                                                   \
  }
#define GELIB_MIR_RUN(N) if constexpr (N <= NLMAX) run_item<N>(B, flags, cnt, xpitch, g0, g1);
  {
    const unsigned char* next = table(d0);
    GELIB_MIR_SWITCH((int)*next, GELIB_MIR_LOAD)
  }
  for (int i = 0; i < A.nitems; i++) {
    const unsigned char* it = table(d0);
    const int4 h = *reinterpret_cast<const int4*>(it);
    const int nl = h.x & 255, cnt = (h.x >> 8) & 255, flags = h.x >> 16;
    if (i + 3 < A.nitems) fetch(d3);
    if (i + 2 < A.nitems) prefetch_rows(table(d2), ptr);
    GELIB_MIR_SWITCH(nl, GELIB_MIR_COPY)
    if (i + 1 < A.nitems) {
      const unsigned char* next = table(d1);
      GELIB_MIR_SWITCH((int)*next, GELIB_MIR_LOAD)
    }
    const int lb = (h.w >> 8) & 255;
    if (flags & kMirFirstOfB)
      for (int r = 0; r <= 2 * lb; r++) *reinterpret_cast<float2*>(yg + kPitch * r) = *reinterpret_cast<float2*>(total + kPitch * r) = make_float2(0.f, 0.f);
    Band B;
    B.cf = reinterpret_cast<const float4*>(it + 16 + 16 * nl);
    B.x = xs + xpitch * h.y;
    B.yg = yg + kPitch * h.z;
    if (flags & kMirSingle) {
      run_single(B, cnt, xpitch, g0);
    } else {
      GELIB_MIR_SWITCH(nl, GELIB_MIR_RUN)
    }
    if (TWO_LEVELS && (flags & kMirLastOfPair))
      for (int r = 0; r <= 2 * lb; r++) {
        float2 *a = reinterpret_cast<float2*>(total + kPitch * r), *b = reinterpret_cast<float2*>(yg + kPitch * r);
        const float2 u = *a, v = *b;
        *a = make_float2(u.x + v.x, u.y + v.y);
        *b = make_float2(0.f, 0.f);
      }
    if ((flags & kMirLastOfB) && ok) {
      const ColPart& p = A.yg[h.w & 255];
      unsigned char* q = reinterpret_cast<unsigned char*>(p.base) + (unsigned long long)cell * p.cell_stride + 8ull * ch;
      for (int r = 0; r <= 2 * lb; r++) {
        const float2 v = *reinterpret_cast<const float2*>(total + kPitch * r);
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(q + (unsigned long long)r * p.unit), "f"(v.x), "f"(v.y) : "memory");
      }
    }
    d0 = d1;
    d1 = d2;
    d2 = d3;
    d3 = dir(i + 4);
    cp_wait_all();
    __syncwarp();
  }
#undef GELIB_MIR_LOAD
#undef GELIB_MIR_COPY
#undef GELIB_MIR_RUN
}

template <int NLMAX, int WARPS>
cudaError_t launch_bwd(const MirBwdArgs& a, size_t smem, cudaStream_t s) {
  auto k = mir_bwd_kernel<NLMAX, WARPS>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<(a.ncols + 31) / 32, 32, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace mir

namespace {

// The items, in order.  Their directory is kept in h_jobs: {first int4, int4 units | place in the ring << 8}; any four neighbours
// of the walk lie apart in the ring.  Words of tables: {bytes of the ring, most y rows}.
void build_bwd(DevicePlan& p, const std::vector<PartSig>& xs, const std::vector<PartSig>& ys, const std::vector<PartSig>& rs, bool diag) {
  build_schedule(xs, ys, rs, diag, false, &p.sched);
  std::map<std::pair<int, int>, std::vector<const Triple*>> pairs;  // by (yi, xi)
  for (const Triple& t : p.sched.triples) pairs[{t.yi, t.xi}].push_back(&t);
  std::vector<int> xrow(1, 0);
  for (const auto& q : xs) xrow.push_back(xrow.back() + 2 * q.l + 1);
  int most_b = 0, last_yi = -1, last_header = -1;
  std::vector<int> sizes;
  for (auto& kv : pairs) {
    const int yi = kv.first.first, xi = kv.first.second, la = xs[xi].l, lb = ys[yi].l;
    auto& ts = kv.second;
    std::sort(ts.begin(), ts.end(), [](const Triple* u, const Triple* v) { return u->l < v->l; });
    const size_t groups = (ts.size() + kMirMaxNl - 1) / kMirMaxNl;
    for (size_t g = 0; g < groups; g++) {
      const std::vector<const Triple*> ls(ts.begin() + ts.size() * g / groups, ts.begin() + ts.size() * (g + 1) / groups);
      const int L = ls.back()->l;
      for (int m = -L; m <= L; m += 2) {
        const bool single = m == L;
        std::vector<const Triple*> at;
        for (const Triple* t : ls)
          if (t->l >= std::abs(m) || (!single && t->l >= std::abs(m + 1))) at.push_back(t);
        const int nl = (int)at.size();
        // entries of row m: lo0 .. hi0, of row m + 1: lo1 .. hi1
        const int lo0 = std::max(-la, m - lb), hi0 = std::min(la, m + lb);
        const int lo1 = std::max(-la, m + 1 - lb), hi1 = std::min(la, m + 1 + lb);
        int flags = single ? kMirSingle : 0;
        if (!single && lo1 > lo0) flags |= kMirPrologue;
        if (!single && hi1 > hi0) flags |= kMirEpilogue;
        if (yi != last_yi) {
          flags |= kMirFirstOfB;
          if (last_header >= 0) p.h_items[last_header].x |= kMirLastOfB << 16;
        }
        last_yi = yi;
        const int cnt = single ? hi0 - lo0 + 1 : hi0 - lo1 + 1, hi = single ? hi0 : hi1;
        last_header = (int)p.h_items.size();
        p.h_items.push_back(make_int4(nl | cnt << 8 | flags << 16, xrow[xi] + lo0 + la, m - lo0 + lb, yi | lb << 8));
        for (const Triple* t : at)
          p.h_items.push_back(make_int4(t->ri, (t->l + m) * rs[t->ri].n + t->offs,
                                        (t->l >= std::abs(m)) | (!single && t->l >= std::abs(m + 1)) << 1, rs[t->ri].n));
        std::vector<float> cf;
        for (int i = lo0; i <= hi; i++) {
          for (int r = 0; r < 2; r++)
            for (const Triple* t : at) {
              const bool in = (r == 0 || !single) && std::abs(m + r) <= t->l && std::abs(m + r - i) <= lb;
              cf.push_back(in ? (float)cg_coefficient(la, lb, t->l, i, m + r - i) : 0.f);
            }
          while (cf.size() % 4) cf.push_back(0.f);
        }
        for (size_t k = 0; k < cf.size(); k += 4) {
          int4 q;
          memcpy(&q, &cf[k], 16);
          p.h_items.push_back(q);
        }
        const int size = (int)p.h_items.size() - last_header;
        if (single && g + 1 == groups) p.h_items[last_header].x |= kMirLastOfPair << 16;
        p.h_jobs.push_back(last_header);
        p.h_jobs.push_back(size);
        sizes.push_back(size);
        most_b = std::max(most_b, 2 * lb + 1);
      }
    }
  }
  if (last_header >= 0) p.h_items[last_header].x |= kMirLastOfB << 16;
  // the smallest ring in which every item can lie apart from the three before it, one after the other
  int ring = 0;
  for (int s : sizes) ring = std::max(ring, s);
  std::vector<int> place(sizes.size());
  for (bool fits = sizes.empty(); !fits; ring++) {
    fits = true;
    int at = 0;
    for (size_t i = 0; i < sizes.size() && fits; i++) {
      if (at + sizes[i] > ring) at = 0;
      for (size_t k = i >= 3 ? i - 3 : 0; k < i; k++)
        if (at < place[k] + sizes[k] && place[k] < at + sizes[i]) fits = false;
      place[i] = at;
      at += sizes[i];
    }
    if (fits) break;
  }
  for (size_t i = 0; i < sizes.size(); i++) p.h_jobs[2 * i + 1] |= place[i] << 8;
  p.tables = {16 * ring, most_b};
}

// The number of columns from which the row-pair kernel takes a signature: nl output l in an item at most, max_la the largest
// min(l1, l2).  0: never.  Measured with 1 million columns, the other kernel / this one, ms:
//   up to five l, where the column kernel has two columns to a lane (even counts) it is the faster one: maxl 3 x 12 .61 / .70, x 20 .62
//     / .68, maxl 4 x 12 1.31 / 1.74, x 20 1.33 / 1.58, x 28 1.34 / 1.51; but with one (odd counts) maxl 3 x 9 1.10 / .77, x 17 1.11 / .70, x
//     15 .79 / .71, x 31 .68 / .67, maxl 4 x 17 2.13 / 1.78, x 23 2.13 / 1.65.  Below, and where cg_narrow1_bwd_kernel pads little, not: maxl 3 x
//     5 1.10 / 1.28, maxl 4 x 9 2.10 / 2.24, x 15 1.62 / 1.84, x 31 1.42 / 1.56.  In the place of cg_narrow1_bwd_kernel at 32 channels the sums
//     are more accurate (maxl 4: error 1.36e-7 / 0.77e-7): maxl 3 .65 / .62, maxl 4 1.36 / 1.31.
//   six l: maxl 5 x 16 3.02 / 2.73, x 32 2.66 / 2.69, x 17 3.80 / 3.66, x 23 3.79 / 3.42; but x 9 3.76 / 4.54, x 12 3.11 / 3.62, x 20 3.08 / 3.28, x
//     28 3.09 / 3.14, x 31 2.86 / 3.25.
//   seven and eight, in the place of cg_narrow1_bwd_kernel only (mir_bwd_kernel): maxl 6 x 16 5.05 / 4.33, x 32 4.87 / 4.28, x 25 6.32 / 5.84, x
//     31 5.24 / 4.96, x 8 5.66 / 5.95, but maxl 7 x 8, 330000 columns 4.78 / 3.83; maxl 6 x 15, with parts of four cells in a warp, 5.75 / 6.66;
//     maxl 6 x 4 8.90 / 10.8.
// The lines in columns: both kernels step by what fills the chip, which decides up to some 400000 columns (maxl 4 x 32: 150000 .21 / .31,
// 200000 .39 / .34, 300000 .40 / .46, 420000 .59 / .60; maxl 5 x 16: 300000 .87 / .95, 420000 1.30 / 1.23); where the gain is larger it
// starts earlier (maxl 3 x 9: 150000 .19 / .20, 200000 .24 / .21; maxl 4 x 17: 200000 .45 / .44; maxl 6 x 16: 112000 .66 / .73, 130000 .80 / .75;
// maxl 7 x 16: 98000 1.17 / 1.10).
unsigned row_pairs_from(int n, int nl, int max_la) {
  const bool odd = n % 2 != 0, narrow = narrow_wins(true, odd ? 1 : 2, n, max_la, 1LL << 40);
  if (n > 32 || nl < 4) return 0;
  if (nl <= 5) {
    if (max_la >= 6) return 0;  // a truncated product: little work per row of g (l up to 6, output up to 4, x 32: 130000 columns .43 / .54)
    if (odd) return n >= 9 && (nl == 4 || (n > 16 && !narrow)) ? 200000 : 0;
    return narrow ? 400000 : 0;
  }
  if (nl == 6) return (32 % n == 0 && n >= 16) || (odd && n > 16 && !narrow) ? 400000 : 0;
  if (!narrow || n < 8 || (n < 16 && 32 % n != 0)) return 0;
  return nl == 7 ? 128000 : 96000;
}

}  // namespace

// Returns -1 when the call does not qualify.
int launch_mir_bwd(const VecCall& c, cudaStream_t s, bool* plan_others) {
  static const char* fn = "SO3vec_addCGproduct_back";
  const int mode = mir_mode();
  if (mode == kColOff || (mode == kColAuto && (col_mode() != kColAuto || !narrow1_enabled()))) return -1;  // other kernels are pinned or off
  if (c.x.empty() || c.y.empty() || c.r.empty() || c.sph || !c.xg.empty() || c.yg.empty()) return -1;
  const int n = c.y[0].n;
  if (c.diag && n > 1) return -1;
  for (const auto& p : c.x) if (p.n != 1 || p.l > 63) return -1;
  for (const auto& p : c.y) if (p.n != n || p.l > 63) return -1;
  if (n < 1 || (long long)n * c.cg.ncells > 0x7fffffffLL) return -1;
  for (const auto& p : c.x)
    for (const auto& q : c.y)
      if (std::min(p.l, q.l) > kMirMaxL) return -1;
  MirBwdArgs a;
  a.nx = (int)c.x.size();
  a.nr = (int)c.r.size();
  int xrows = 0;
  for (int i = 0; i < a.nx; i++) {
    if (!col_fill_part(c.x[i], c.cg, 0, true, &a.x[i])) return -1;
    a.xl[i] = (unsigned char)c.x[i].l;
    xrows += 2 * c.x[i].l + 1;
  }
  for (size_t i = 0; i < c.yg.size(); i++)
    if (!col_fill_part(c.yg[i], c.cg, 0, true, &a.yg[i])) return -1;
  for (int i = 0; i < a.nr; i++) {
    const PartView& p = c.r[i];
    if (p.sm != 2LL * p.n || (2LL * p.l + 2) * p.n > 0x7fffffffLL) return -1;  // the items hold offsets of dense rows
    if (!col_fill_part(p, c.cg, 2LL * c.offs_extra, false, &a.g[i])) return -1;
  }
  a.n = (unsigned)n;
  a.ncols = (unsigned)(c.cg.ncells * n);
  a.xcells = 32 % n == 0 ? 32 / n : (30 + n) / n + 1;
  int nl = 0, max_la = 0;  // most output l of an item, largest min(l1, l2)
  for (const auto& p : c.x)
    for (const auto& q : c.y) {
      int ls = 0;
      for (const auto& r : c.r) ls += r.l >= std::abs(p.l - q.l) && r.l <= p.l + q.l;
      const int groups = (ls + kMirMaxNl - 1) / kMirMaxNl;
      if (groups > 0) nl = std::max(nl, (ls + groups - 1) / groups);
      max_la = std::max(max_la, std::min(p.l, q.l));
    }
  const unsigned least = mode == kColAuto ? row_pairs_from(n, nl, max_la) : 0;
  if (mode == kColAuto && least == 0) return -1;
  std::vector<int> key = {22 /*family*/, c.diag, a.nx, (int)c.y.size(), a.nr, n};
  for (const auto& p : c.x) key.push_back(p.l);
  for (const auto& p : c.y) key.push_back(p.l);
  for (const auto& p : c.r) { key.push_back(p.l); key.push_back(p.n); }
  const auto xs = sig_of(c.x), ys = sig_of(c.y), rs = sig_of(c.r);
  const bool diag = c.diag;
  DevicePlan* plan = get_plan(key, [&](DevicePlan& p) { build_bwd(p, xs, ys, rs, diag); });
  if (!plan) return GELIB_CUDA_ERROR;
  a.nitems = (int)plan->h_jobs.size() / 2;
  if (a.nitems == 0) return GELIB_OK;
  a.ring_bytes = plan->tables[0];
  a.y_rows = plan->tables[1];
  const size_t smem = 256 * (size_t)a.nr + a.ring_bytes + mir::kPitch * (size_t)a.y_rows * (nl <= kMirTwoLevels ? 2 : 1) + 8 * (size_t)a.xcells * xrows;
  if (smem > kColMaxSmem) return -1;
  if (mode == kColAuto) {
    const bool first = plan->first_use.exchange(false);  // another batch of the signature goes to the others
    if (a.ncols < least) return -1;
    *plan_others = first;
  }
  if (c.plan_only) return GELIB_OK;
  a.items = plan->items;
  a.dir = reinterpret_cast<const int2*>(plan->jobs);
  cudaError_t e;
  if (nl <= 5) e = mir::launch_bwd<5, 28>(a, smem, s);
  else if (nl <= 6) e = mir::launch_bwd<6, 20>(a, smem, s);
  else if (nl <= 7) e = mir::launch_bwd<7, 20>(a, smem, s);
  else e = mir::launch_bwd<kMirMaxNl, 16>(a, smem, s);
  if (e != cudaSuccess) return check_cuda(e, fn, "row-pair backward kernel launch");
  count_launch();
  return GELIB_OK;
}

}  // namespace gelib_b200
