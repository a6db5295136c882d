// Forward mirrored-row kernel (see mir.h).
//
// A block owns 32 or 64 consecutive columns (one or two adjacent channels per lane) and stages every x and y row of them in
// shared memory once; its eight warps take the items in turn, those with equal numbers of output l one after the other, and each
// copies the tables of the items it will take (cp.async, two ahead), so no warp ever waits for another.
//
// Measured against the kernels it replaced (diag_fwd_cell_kernel, cg_narrow_fwd_kernel, the column forward), us: diagonal, maxl
// 8 x 128 channels, batch 2048 3056 -> 1779 (71 % of the rate at which its output can be written); one-channel x, maxl 6 x 16,
// 65536 cells 4700 -> 2384 (77 %); diagonal, maxl 4 x 128, batch 1024 155 -> 120, maxl 3 x 12, batch 500 20 -> 11.  Bound by
// issue: 280 k warp instructions per 64 columns at maxl 8, issued in 57 % of the cycles; shared memory is at 77 % of its rate.
// Items in order of their cost alone, which mixes the bodies, took 2340 us (instruction fetch), coefficients stored twice instead
// of paired in registers 1860, unpacked multiply-adds 2020, ten output l per item, which spills, 2720.
#include <algorithm>
#include <cstring>
#include <map>

#include "f32x2.h"
#include "mir.h"

namespace gelib_b200 {
namespace mir {

constexpr int kWarps = 8;

constexpr int kSharedPitch = 64;  // bytes between the staged rows of a one-channel x: one number for each of up to eight cells

template <int CPL>
struct Cols {
  float2 c[CPL];
};
template <int CPL>
__device__ __forceinline__ Cols<CPL> lds_cols(const unsigned char* p) {
  Cols<CPL> v;
  if constexpr (CPL == 2) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v.c[0] = make_float2(q.x, q.y);
    v.c[1] = make_float2(q.z, q.w);
  } else {
    v.c[0] = *reinterpret_cast<const float2*>(p);
  }
  return v;
}
// A row of x: the lane's columns, or (SHARED) the one number of the lane's cell.
template <int CPL, bool SHARED>
__device__ __forceinline__ Cols<CPL> lds_x(const unsigned char* p) {
  if constexpr (SHARED) {
    Cols<CPL> v;
    const float2 q = *reinterpret_cast<const float2*>(p);
#pragma unroll
    for (int e = 0; e < CPL; e++) v.c[e] = q;
    return v;
  } else {
    return lds_cols<CPL>(p);
  }
}
__device__ __forceinline__ f32x2 product(float2 a, float2 b) {
  return pack2(fmaf(-a.y, b.y, a.x * b.x), fmaf(a.y, b.x, a.x * b.y));
}
template <int CPL>
__device__ __forceinline__ void store_row(float2* p, const f32x2 (&v)[CPL], bool add) {
  float o[2 * CPL];
#pragma unroll
  for (int e = 0; e < CPL; e++) unpack2(v[e], o[2 * e], o[2 * e + 1]);
  if constexpr (CPL == 2) {
    if (add) {
      const float4 q = *reinterpret_cast<const float4*>(p);
      o[0] += q.x; o[1] += q.y; o[2] += q.z; o[3] += q.w;
    }
    __stcs(reinterpret_cast<float4*>(p), make_float4(o[0], o[1], o[2], o[3]));
  } else {
    if (add) {
      const float2 q = *p;
      o[0] += q.x; o[1] += q.y;
    }
    __stcs(p, make_float2(o[0], o[1]));
  }
}

// One item.  it: header, records, coefficients; xs, ys: the lane's number in staged row 0.
template <int NL, int CPL, bool SHARED>
__device__ __forceinline__ void run_item(const unsigned char* it, const int4 h, const unsigned char* xs, const unsigned char* ys,
                                         const unsigned long long* ptr, bool ok, bool add) {
  constexpr int YP = 256 * CPL, XP = SHARED ? kSharedPitch : YP, NQ = (NL + 3) / 4;
  const int cnt = (h.x >> 8) & 255;
  const unsigned char *xp = xs + XP * (h.y & 0xffff), *xm = xs + XP * (h.y >> 16);
  const unsigned char *yp = ys + YP * (h.z & 0xffff), *ym = ys + YP * (h.z >> 16);
  const float4* cf = reinterpret_cast<const float4*>(it + 16 + 16 * NL);
  f32x2 sp[NL][CPL], sm[NL][CPL];
#pragma unroll
  for (int j = 0; j < NL; j++)
#pragma unroll
    for (int e = 0; e < CPL; e++) sp[j][e] = sm[j][e] = 0ull;
#pragma unroll 1
  for (int k = 0; k < cnt; k++) {
    const Cols<CPL> a = lds_x<CPL, SHARED>(xp), b = lds_cols<CPL>(yp), c = lds_x<CPL, SHARED>(xm), d = lds_cols<CPL>(ym);
    xp += XP;
    xm -= XP;
    yp -= YP;
    ym += YP;
    f32x2 q[4 * NQ];
#pragma unroll
    for (int j = 0; j < NQ; j++) {
      const float4 v = cf[j];
      q[4 * j] = pack2(v.x, v.x);
      q[4 * j + 1] = pack2(v.y, v.y);
      q[4 * j + 2] = pack2(v.z, v.z);
      q[4 * j + 3] = pack2(v.w, v.w);
    }
    cf += NQ;
#pragma unroll
    for (int e = 0; e < CPL; e++) {
      const f32x2 p = product(a.c[e], b.c[e]), m = product(c.c[e], d.c[e]);
#pragma unroll
      for (int j = 0; j < NL; j++) {
        sp[j][e] = fma2(q[j], p, sp[j][e]);
        sm[j][e] = fma2(q[j], m, sm[j][e]);
      }
    }
  }
  const bool zero_row = h.w != 0;
#pragma unroll
  for (int j = 0; j < NL; j++) {
    const int4 r = *reinterpret_cast<const int4*>(it + 16 + 16 * j);  // {part, complex offset of row m, of row -m, sign}
    const f32x2 s = pack2(__int_as_float(r.w), __int_as_float(r.w));
    float2* p = reinterpret_cast<float2*>(ptr[32 * r.x]);
    if (zero_row) {
#pragma unroll
      for (int e = 0; e < CPL; e++) sp[j][e] = fma2(s, sm[j][e], sp[j][e]);
      if (ok) store_row<CPL>(p + (unsigned)r.y, sp[j], add);
    } else {
#pragma unroll
      for (int e = 0; e < CPL; e++) sm[j][e] = mul2(s, sm[j][e]);
      if (ok) {
        store_row<CPL>(p + (unsigned)r.y, sp[j], add);
        store_row<CPL>(p + (unsigned)r.z, sm[j], add);
      }
    }
  }
}

template <int CPL, bool SHARED>
__global__ void __launch_bounds__(32 * kWarps, CPL == 2 ? 2 : 4) mir_fwd_kernel(const __grid_constant__ MirArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int W = 32 * CPL, YP = 8 * W;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // [addresses of the lanes' columns in every r part][y rows][x rows][three item buffers per warp]
  unsigned long long* ptr = reinterpret_cast<unsigned long long*>(smem);
  const int ys_at = 256 * A.nr, xs_at = ys_at + YP * A.yrows;
  constexpr int xpitch = SHARED ? kSharedPitch : YP;
  const int buf_at = xs_at + xpitch * A.xrows + 3 * A.item_bytes * warp;
  const unsigned col0 = blockIdx.x * W;
  unsigned col = col0 + CPL * lane;
  const bool ok = col < A.ncols;
  if (!ok) col = A.ncols - CPL;
  const unsigned cell = col / A.n, ch = col - cell * A.n;

  // the tables of an item are requested two items ahead
  const int stride = kWarps * gridDim.y;
  int item = blockIdx.y * kWarps + warp;
  auto dir = [&](int i) { return i < A.nitems ? __ldg(A.dir + i) : make_int2(0, 0); };
  auto fetch = [&](int2 d, int buf) {
    const uint32_t dst = sptr(smem) + buf_at + A.item_bytes * buf;
    for (int e = lane; e < d.y; e += 32) cp_async<16>(dst + 16 * e, A.items + d.x + e);
    cp_commit();
  };
  fetch(dir(item), 0);
  fetch(dir(item + stride), 1);
  int2 ahead = dir(item + 2 * stride);

  for (int p = warp; p < A.nr; p += kWarps)
    ptr[32 * p + lane] = reinterpret_cast<unsigned long long>(A.r[p].base) + (unsigned long long)cell * A.r[p].cell_stride + 8ull * ch;
  auto stage = [&](const ColPart& p, int l, int row0, int at, bool one) {
    const unsigned char* src = reinterpret_cast<const unsigned char*>(p.base) + (unsigned long long)cell * p.cell_stride + (one ? 0ull : 8ull * ch);
    for (int m = (warp - row0) & (kWarps - 1); m <= 2 * l; m += kWarps) {
      const uint32_t dst = sptr(smem) + at + YP * (row0 + m) + 8 * CPL * lane;
      if (one) {  // one number for every column of the cell
#pragma unroll
        for (int e = 0; e < CPL; e++) cp_async<8>(dst + 8 * e, src + (unsigned long long)m * p.unit);
      } else {
        cp_async<8 * CPL>(dst, src + (unsigned long long)m * p.unit);
      }
    }
  };
  for (int i = 0, row = 0; i < A.ny; row += 2 * A.yl[i] + 1, i++) stage(A.y[i], A.yl[i], row, ys_at, false);
  const unsigned cell0 = col0 / A.n;
  if constexpr (SHARED) {
    const unsigned last = (A.ncols - 1) / A.n;
    for (int i = 0, row = 0; i < A.nx; row += 2 * A.xl[i] + 1, i++)
      for (int e = threadIdx.x; e < (2 * A.xl[i] + 1) * A.xcells; e += 32 * kWarps) {
        const int m = e / A.xcells, c = e - m * A.xcells;
        const unsigned char* src = reinterpret_cast<const unsigned char*>(A.x[i].base) +
                                   (unsigned long long)min(cell0 + c, last) * A.x[i].cell_stride + (unsigned long long)m * A.x[i].unit;
        cp_async<8>(sptr(smem) + xs_at + xpitch * (row + m) + 8 * c, src);
      }
  } else {
    for (int i = 0, row = 0; i < A.nx; row += 2 * A.xl[i] + 1, i++) stage(A.x[i], A.xl[i], row, xs_at, A.one_channel != 0);
  }
  cp_commit();
  cp_wait<0>();
  __syncthreads();

  const unsigned char* xs = smem + xs_at + (SHARED ? 8 * (cell - cell0) : 8 * CPL * lane);
  const unsigned char* ys = smem + ys_at + 8 * CPL * lane;
  const bool add = A.accumulate != 0;
  for (int buf = 0; item < A.nitems; item += stride) {
    const int spare = buf == 0 ? 2 : buf - 1;
    fetch(ahead, spare);
    ahead = dir(item + 3 * stride);
    const unsigned char* it = smem + buf_at + A.item_bytes * buf;
    const int4 h = *reinterpret_cast<const int4*>(it);
#define GELIB_MIR_CASE(N) case N: run_item<N, CPL, SHARED>(it, h, xs, ys, ptr + lane, ok, add); break;
    switch (h.x & 255) {
      GELIB_MIR_CASE(1) GELIB_MIR_CASE(2) GELIB_MIR_CASE(3) GELIB_MIR_CASE(4)
      GELIB_MIR_CASE(5) GELIB_MIR_CASE(6) GELIB_MIR_CASE(7) GELIB_MIR_CASE(8)
      default: break;
    }
#undef GELIB_MIR_CASE
    cp_wait<1>();
    __syncwarp();
    buf = buf == 2 ? 0 : buf + 1;
  }
}

template <int CPL, bool SHARED>
cudaError_t launch_fwd(const MirArgs& a, int splits, size_t smem, cudaStream_t s) {
  auto k = mir_fwd_kernel<CPL, SHARED>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<dim3((a.ncols + 32 * CPL - 1) / (32 * CPL), splits), 32 * kWarps, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace mir

namespace {

// Items of a forward product; the directory is kept in h_jobs, the size of the largest in tables.
void build_fwd(DevicePlan& p, const std::vector<PartSig>& xs, const std::vector<PartSig>& ys, const std::vector<PartSig>& rs, bool diag) {
  build_schedule(xs, ys, rs, diag, false, &p.sched);
  std::vector<int> xrow(1, 0), yrow(1, 0);
  for (const auto& q : xs) xrow.push_back(xrow.back() + 2 * q.l + 1);
  for (const auto& q : ys) yrow.push_back(yrow.back() + 2 * q.l + 1);
  std::map<std::pair<int, int>, std::vector<const Triple*>> pairs;
  for (const Triple& t : p.sched.triples) pairs[{t.xi, t.yi}].push_back(&t);
  struct Item { std::vector<int4> v; int nl; double cost; };
  std::vector<Item> items;
  for (auto& kv : pairs) {
    auto& ts = kv.second;
    std::sort(ts.begin(), ts.end(), [](const Triple* u, const Triple* v) { return u->l < v->l; });
    const int xi = kv.first.first, yi = kv.first.second, l1 = xs[xi].l, l2 = ys[yi].l;
    for (int m = 0; m <= ts.back()->l; m++) {
      std::vector<const Triple*> with_m;
      for (const Triple* t : ts)
        if (t->l >= m) with_m.push_back(t);
      const size_t groups = (with_m.size() + kMirMaxNl - 1) / kMirMaxNl;
      for (size_t g = 0; g < groups; g++) {
        const std::vector<const Triple*> at(with_m.begin() + with_m.size() * g / groups, with_m.begin() + with_m.size() * (g + 1) / groups);
        const int nl = (int)at.size();
        const int lo = m == 0 ? 0 : std::max(-l1, m - l2), hi = std::min(l1, m + l2), cnt = hi - lo + 1;
        const int x0 = xrow[xi] + l1, y0 = yrow[yi] + l2;  // staged rows of index 0
        Item it;
        it.nl = nl;
        it.cost = cnt * (4 * nl + 24) + 24 * nl + 80;
        it.v.push_back(make_int4(nl | cnt << 8, (x0 + lo) | (x0 - lo) << 16, (y0 + m - lo) | (y0 - (m - lo)) << 16, m == 0));
        std::vector<float> cf;
        for (const Triple* t : at) {
          const float s = (l1 + l2 - t->l) % 2 ? -1.f : 1.f;
          int4 r = make_int4(t->ri, (t->l + m) * rs[t->ri].n + t->offs, (t->l - m) * rs[t->ri].n + t->offs, 0);
          memcpy(&r.w, &s, 4);
          it.v.push_back(r);
        }
        for (int i = lo; i <= hi; i++)
          for (int j = 0; j < (nl + 3) / 4 * 4; j++)
            cf.push_back(j < nl ? (float)cg_coefficient(l1, l2, at[j]->l, i, m - i) * (m == 0 && i == 0 ? 0.5f : 1.f) : 0.f);
        for (size_t k = 0; k < cf.size(); k += 4) {
          int4 q;
          memcpy(&q, &cf[k], 16);
          it.v.push_back(q);
        }
        items.push_back(std::move(it));
      }
    }
  }
  // warps that work on equal numbers of output l share the instructions of one body
  std::stable_sort(items.begin(), items.end(), [](const Item& u, const Item& v) { return u.nl != v.nl ? u.nl > v.nl : u.cost > v.cost; });
  int most = 0;
  for (const Item& it : items) {
    most = std::max(most, 16 * (int)it.v.size());
    p.h_jobs.push_back((int)p.h_items.size());
    p.h_jobs.push_back((int)it.v.size());
    p.h_items.insert(p.h_items.end(), it.v.begin(), it.v.end());
  }
  p.tables = {most};
}

}  // namespace

// Returns -1 when the call does not qualify.
int launch_mir_fwd(const VecCall& c, cudaStream_t s, bool* plan_others) {
  static const char* fn = "SO3vec_addCGproduct";
  const int mode = mir_mode();
  if (mode == kColOff || (mode == kColAuto && col_mode() != kColAuto)) return -1;  // the column kernels are pinned or off
  if (c.x.empty() || c.y.empty() || c.r.empty() || c.sph) return -1;
  MirArgs a;
  const int n = c.y[0].n, nx = c.diag ? n : 1;
  for (const auto& p : c.x) if (p.n != nx) return -1;
  for (const auto& p : c.y) if (p.n != n) return -1;
  if (n < 1 || (long long)n * c.cg.ncells > 0x7fffffffLL) return -1;
  for (const auto& p : c.x)
    for (const auto& q : c.y)
      if (std::min(p.l, q.l) > kMirMaxL) return -1;
  a.nx = (int)c.x.size();
  a.ny = (int)c.y.size();
  a.nr = (int)c.r.size();
  a.xrows = a.yrows = 0;
  for (int i = 0; i < a.nx; i++) {
    if (c.x[i].l > 63 || !col_fill_part(c.x[i], c.cg, 0, true, &a.x[i])) return -1;
    a.xl[i] = (unsigned char)c.x[i].l;
    a.xrows += 2 * c.x[i].l + 1;
  }
  for (int i = 0; i < a.ny; i++) {
    if (c.y[i].l > 63 || !col_fill_part(c.y[i], c.cg, 0, true, &a.y[i])) return -1;
    a.yl[i] = (unsigned char)c.y[i].l;
    a.yrows += 2 * c.y[i].l + 1;
  }
  for (int i = 0; i < a.nr; i++) {
    const PartView& p = c.r[i];
    if (p.sm != 2LL * p.n || (2LL * p.l + 1) * p.n > 0x7fffffffLL) return -1;  // the items hold offsets of dense rows
    if (!col_fill_part(p, c.cg, 2LL * c.offs_extra, false, &a.r[i])) return -1;
  }
  const bool one_channel = nx == 1 && n > 1;
  // two columns per lane: every access is 16 bytes
  bool two = n % 2 == 0 && c.offs_extra % 2 == 0;
  for (const auto* v : {&c.y, &c.r, one_channel ? &c.y : &c.x})
    for (const auto& p : *v)
      if ((uintptr_t)p.base % 16 || p.sb % 4 || p.sg0 % 4 || p.sg1 % 4 || p.sm % 4) two = false;
  const long long columns = c.cg.ncells * n;
  a.n = (unsigned)n;
  a.ncols = (unsigned)columns;
  a.one_channel = one_channel;
  std::vector<int> key = {21 /*family*/, c.diag, a.nx, a.ny, a.nr, n};
  for (const auto& p : c.x) key.push_back(p.l);
  for (const auto& p : c.y) key.push_back(p.l);
  for (const auto& p : c.r) { key.push_back(p.l); key.push_back(p.n); }
  const auto xs = sig_of(c.x), ys = sig_of(c.y), rs = sig_of(c.r);
  const bool diag = c.diag;
  DevicePlan* plan = get_plan(key, [&](DevicePlan& p) { build_fwd(p, xs, ys, rs, diag); });
  if (!plan) return GELIB_CUDA_ERROR;
  a.nitems = (int)plan->h_jobs.size() / 2;
  if (a.nitems == 0) return GELIB_OK;
  a.item_bytes = plan->tables[0];
  // Two columns share the coefficients and the control of an item; blocks of 64 columns must fit twice on an SM, and one
  // channel per lane keeps an x of one channel at one number per cell down to four channels (maxl 6 x 4, 100000 cells 1730 us
  // against 1775).  Two against one, us: maxl 8 x 128, batch 2048 1779 / 2060; one-channel x, maxl 6 x 16, 65536 cells 2384 / 3030.
  int cpl = two && (mode == kColTwo || (mode == kColAuto && !(one_channel && n < 8))) ? 2 : 1;
  bool shared = false;
  size_t smem = 0;
  for (;; cpl = 1) {
    const int W = 32 * cpl;
    a.xcells = W % n == 0 ? W / n : (W + n - 2) / n + 1;
    shared = one_channel && 8 * a.xcells <= mir::kSharedPitch;
    smem = 256 * (size_t)a.nr + 8 * (size_t)W * a.yrows + (size_t)(shared ? mir::kSharedPitch : 8 * W) * a.xrows +
           3 * (size_t)a.item_bytes * mir::kWarps;
    if (cpl == 1 || smem <= kColMaxSmem / 2) break;
  }
  if (smem > kColMaxSmem) return -1;
  // A block that stages its columns for a handful of items pays more than the column and narrow kernels when there are
  // many of them (us, those / this one; 7 items at maxl 1, 23 at maxl 2): maxl 1 x 64, batch 468 14.5 / 10.2, 1562 16.4 / 18.5,
  // 4687 28 / 41; maxl 2 x 8, batch 12500 33 / 30; one-channel x, maxl 1 x 16, 1875 cells 13 / 10, 6250 13 / 19; maxl 2 x 16, 1875
  // 26 / 15, 25000 74 / 91, but, where the narrow kernel pads its lanes, maxl 2 x 7, 57142 140 / 109; maxl 3 x 32, 12500 174 / 164.
  // The narrow kernel, for up to 32 channels of a one-channel x, is ahead earlier when there are least items or y has only
  // l = 0, us at 36000 / 44000 / 62000 columns: maxl 1 x 16 7.7 / 7.6 / 7.8 against 6.2 / 7.6 / 9.8, l = 0 with l <= 2 x 16 6.3 / 6.8 / 7.0 against 5.6 /
  // 7.2 / 9.3, l <= 4 with l = 0 x 16 9.7 / 10.5 / 10.5 against 8.2 / 10.8 / 13.2; but l = 0 with l <= 4 x 16 11.5 / 12.9 / 12.7 against 8.1 / 9.9 / 12.3.
  const bool pow2 = (n & (n - 1)) == 0;
  const bool few_items = a.nitems <= (one_channel && pow2 ? 24 : 8);
  const bool narrow = one_channel && n <= 32 && (a.nitems <= 8 || a.yrows == 1);
  if (mode == kColAuto && few_items) {
    const bool first = plan->first_use.exchange(false);
    if (columns > (narrow ? 40000 : 64000)) return -1;
    *plan_others = first;  // another batch of the signature goes there
  }
  if (c.plan_only) return GELIB_OK;
  a.items = plan->items;
  a.dir = reinterpret_cast<const int2*>(plan->jobs);
  a.accumulate = (c.flags & GELIB_OVERWRITE) ? 0 : 1;
  // Few blocks share the items between them, two blocks to an SM; a second wave that would be short is cut finer (maxl 8 x 128,
  // batch 70 113 -> 94 us, batch 156 235 -> 187, batch 234 284 -> 263; 468, in the fourth wave, 479 either way).
  const int blocks = (int)((columns + 32 * cpl - 1) / (32 * cpl));
  int splits = std::max(1, 296 / blocks);
  if (blocks >= 296 && blocks < 592 && a.nitems >= 256) splits = 1184 / blocks;
  splits = std::min(splits, std::max(1, a.nitems / mir::kWarps));
  cudaError_t e;
  if (cpl == 2) e = shared ? mir::launch_fwd<2, true>(a, splits, smem, s) : mir::launch_fwd<2, false>(a, splits, smem, s);
  else e = shared ? mir::launch_fwd<1, true>(a, splits, smem, s) : mir::launch_fwd<1, false>(a, splits, smem, s);
  if (e != cudaSuccess) return check_cuda(e, fn, "mirrored-row forward kernel launch");
  count_launch();
  return GELIB_OK;
}

}  // namespace gelib_b200
