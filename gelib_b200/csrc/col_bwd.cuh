// Backward column kernel (see col.h): G = sum_l C_l g_l per band entry, xg += G conj(y), yg += G conj(x).
#pragma once
#include <algorithm>

#include "col_device.h"

namespace gelib_b200 {
namespace col {

// s += u conj(v), complex.
__device__ __forceinline__ void add_conj(float2& s, float ur, float ui, float2 v) {
  s.x = fmaf(ur, v.x, s.x); s.x = fmaf(ui, v.y, s.x);
  s.y = fmaf(ui, v.x, s.y); s.y = fmaf(-ur, v.y, s.y);
}
template <int CPL>
__device__ __forceinline__ Row<CPL> to_row(const float2 (&v)[CPL]) {
  Row<CPL> r;
#pragma unroll
  for (int c = 0; c < CPL; c++) r.c[c] = pack2(v[c].x, v[c].y);
  return r;
}

template <int CPL>
__device__ __forceinline__ void add_slot(unsigned char* p, const float2 (&v)[CPL]) {
  const Row<CPL> o = lds_row<CPL>(p);
  float2 s[CPL];
#pragma unroll
  for (int c = 0; c < CPL; c++) {
    unpack2(o.c[c], s[c].x, s[c].y);
    s[c].x += v[c].x;
    s[c].y += v[c].y;
  }
  sts_row<CPL>(p, to_row<CPL>(s));
}

// The row at p (shared memory) of block `rank` of the cluster.
template <int CPL>
__device__ __forceinline__ Row<CPL> lds_row_of(const unsigned char* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  Row<CPL> v;
#pragma unroll
  for (int c = 0; c < CPL; c++) asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(v.c[c]) : "r"(a + 8 * c) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// One step: an output row of a pair against the a block.  Entry i pairs a[i] with the b row at bptr - i rows.
template <int K, int CPL, bool DOA, bool DOB, int NL, int NLMIN = NL - 1>
__device__ __forceinline__ void bwd_step(Walk<CPL>& W, int st, const float2 (&a)[K][CPL], float2 (&ag)[K][CPL], float2 (&bg)[K][CPL],
                                         uint32_t bptr) {
  constexpr int kCoefs = (NL + 3) / 4 * 4;
  cp_wait<kColRing - NL>();
  const int nl = st & 255, lo = (st >> 8) & 255, hi = (st >> 16) & 255;
  f32x2 g[NL][CPL];
#pragma unroll
  for (int j = 0; j < NL; j++) {
    const Row<CPL> r = W.row(j);
#pragma unroll
    for (int c = 0; c < CPL; c++) g[j][c] = j < NLMIN || j < nl ? r.c[c] : 0ull;  // beyond nl: a row of a later step
  }
  W.template refill<NL>(nl);
  const unsigned span = hi - lo;
#pragma unroll
  for (int blk = 0; blk < (K + 3) / 4; blk++) {
    if (hi >= 4 * blk && lo < 4 * blk + 4) {  // the same in every lane of the block
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int i = 4 * blk + e < K ? 4 * blk + e : K - 1;
        if (4 * blk + e >= K) continue;
        f32x2 G[CPL];
#pragma unroll
        for (int j = 0; j < NL; j += 4) {
          const Coefs q = coefs<NL>(W.smem + W.coef + (i * kCoefs + j) * 4);
#pragma unroll
          for (int c = 0; c < CPL; c++) {
            G[c] = j == 0 ? mul2(q.c[0], g[0][c]) : fma2(q.c[0], g[j][c], G[c]);
            G[c] = fma2(q.c[1], g[j + 1][c], G[c]);
            if (j + 2 < NL) {
              G[c] = fma2(q.c[2], g[j + 2][c], G[c]);
              G[c] = fma2(q.c[3], g[j + 3][c], G[c]);
            }
          }
        }
        float gr[CPL], gi[CPL];
#pragma unroll
        for (int c = 0; c < CPL; c++) unpack2(G[c], gr[c], gi[c]);
        if (DOA) {
          if ((unsigned)(i - lo) <= span) {  // outside the band there is no b row, and G may be 0 * inf
            const Row<CPL> w = lds_row<CPL>(W.smem + (bptr - Walk<CPL>::kRow * i));
#pragma unroll
            for (int c = 0; c < CPL; c++) {
              float2 v;
              unpack2(w.c[c], v.x, v.y);
              add_conj(ag[i][c], gr[c], gi[c], v);
            }
          }
        }
        if (DOB) {  // rows outside the band are never added to the slots
#pragma unroll
          for (int c = 0; c < CPL; c++) add_conj(bg[i][c], gr[c], gi[c], a[i][c]);
        }
      }
    }
  }
  W.coef += K * kCoefs * 4;
}

// bval, bacc: byte offsets of the lane's slots of b row 0 (values, gradients).  OWNED: the a rows' gradients are added to
// slots from bacc on instead of to global memory.
template <int K, int CPL, bool DOA, bool DOB, bool OWNED>
__device__ __forceinline__ void bwd_segment(Walk<CPL>& W, const int4 h, int lb, uint32_t bval, uint32_t bacc) {
  constexpr int NLMAX = K < 6 ? K + 1 : kColMaxNl;  // six rows and more may be a part of a larger a part
  constexpr uint32_t kRow = Walk<CPL>::kRow;
  float2 a[K][CPL], ag[K][CPL], bg[K][CPL];
  if (DOB) W.template take<0>(a);
#pragma unroll
  for (int i = 0; i < K; i++)
#pragma unroll
    for (int c = 0; c < CPL; c++) ag[i][c] = bg[i][c] = make_float2(0.f, 0.f);
  const int nsteps = h.x >> 16, nb = 2 * lb + 1;
  int br = h.y + lb;  // row of b that entry 0 meets
  auto leave = [&](int r, const float2 (&v)[CPL]) {
    if ((unsigned)r < (unsigned)nb) add_slot<CPL>(W.smem + bacc + kRow * r, v);
  };
  const uint32_t steps = W.seg + 32;
  int next = *reinterpret_cast<const int*>(W.smem + steps);
  for (int s = 0; s < nsteps; s++, br++) {
    const int st = next;
    next = *reinterpret_cast<const int*>(W.smem + steps + 4 * s + 4);  // past the last one: another word of the chunk
    const uint32_t bptr = bval + kRow * br;
    const int nl = st & 255, nl2 = (nl + 1) >> 1;
    if constexpr (DOA && DOB && K >= 6) {  // the instances of col_nl_padded
      if (nl <= 6) bwd_step<K, CPL, DOA, DOB, 6, 1>(W, st, a, ag, bg, bptr);
      else bwd_step<K, CPL, DOA, DOB, 10, 7>(W, st, a, ag, bg, bptr);
    } else {
      if (nl2 == 1) bwd_step<K, CPL, DOA, DOB, 2>(W, st, a, ag, bg, bptr);
      if constexpr (NLMAX >= 4) if (nl2 == 2) bwd_step<K, CPL, DOA, DOB, 4>(W, st, a, ag, bg, bptr);
      if constexpr (NLMAX >= 6) if (nl2 == 3) bwd_step<K, CPL, DOA, DOB, 6>(W, st, a, ag, bg, bptr);
      if constexpr (NLMAX >= 8) if (nl2 == 4) bwd_step<K, CPL, DOA, DOB, 8>(W, st, a, ag, bg, bptr);
      if constexpr (NLMAX >= 10) if (nl2 == 5) bwd_step<K, CPL, DOA, DOB, 10>(W, st, a, ag, bg, bptr);
    }
    if (DOB) {  // the row that leaves the window, then the window moves by one row
      leave(br - (K - 1), bg[K - 1]);
#pragma unroll
      for (int i = K - 1; i > 0; i--)
#pragma unroll
        for (int c = 0; c < CPL; c++) bg[i][c] = bg[i - 1][c];
#pragma unroll
      for (int c = 0; c < CPL; c++) bg[0][c] = make_float2(0.f, 0.f);
    }
  }
  if (DOB) {
#pragma unroll
    for (int i = 1; i < K; i++) leave(br - i, bg[i]);
  }
  W.seg = steps + 4 * ((nsteps + 3) & ~3);
  if constexpr (OWNED) {
#pragma unroll
    for (int i = 0; i < K; i++) add_slot<CPL>(W.smem + bacc + kRow * i, ag[i]);
  } else if (DOA && W.ok) {
    const ColPart& p = W.A.grad[((h.x >> 8) & kColHalf1 ? kMaxParts : 0) + h.w];
    unsigned char* q = reinterpret_cast<unsigned char*>(p.base) + (unsigned long long)W.cell * p.cell_stride + 8ull * CPL * W.ch +
                       (unsigned long long)h.z * p.unit;
#pragma unroll
    for (int i = 0; i < K; i++) red_row<CPL>(q + (unsigned long long)i * p.unit, to_row<CPL>(ag[i]));
  }
}

// One run of the walk.
template <int KMAX, int CPL, bool DOX, bool DOY, bool OWNED>
__device__ __forceinline__ void walk_bwd(Walk<CPL>& W, uint32_t bufs, uint32_t ring, uint32_t bval, uint32_t bacc) {
  constexpr uint32_t kRow = Walk<CPL>::kRow;
  Row<CPL> zero;
#pragma unroll
  for (int c = 0; c < CPL; c++) zero.c[c] = 0ull;
  W.start(0, bufs, ring);
  int f;
  do {
    const int4 h = *reinterpret_cast<const int4*>(W.smem + W.seg), h1 = *reinterpret_cast<const int4*>(W.smem + W.seg + 16);
    const int kb = h.x & 255, nb = 2 * h1.y + 1;
    f = (h.x >> 8) & 255;
    const bool half1 = (f & kColHalf1) != 0;
    const bool do_a = OWNED || (half1 ? DOY : DOX), do_b = !OWNED && (half1 ? DOX : DOY);
    if (f & kColFirstOfB) {
      if (do_a) W.take_to(bval, nb);
      if (do_b)
        for (int r = 0; r < nb; r++) sts_row<CPL>(W.smem + bacc + kRow * r, zero);
    }
#define GELIB_COL_CASE(N)                                                                          \
  if constexpr (N <= KMAX)                                                                         \
    if (kb == N) {                                                                                 \
      if constexpr (OWNED) bwd_segment<N, CPL, true, false, true>(W, h, h1.y, bval, bacc + kRow * h1.z); \
      else if (DOX == DOY || !half1) bwd_segment<N, CPL, DOX, DOY, false>(W, h, h1.y, bval, bacc); \
      else bwd_segment<N, CPL, DOY, DOX, false>(W, h, h1.y, bval, bacc);                           \
    }
    if (kb <= 5) {
      GELIB_COL_CASE(1)
      GELIB_COL_CASE(3)
      GELIB_COL_CASE(5)
    } else if (kb <= 7) {
      GELIB_COL_CASE(6)
      GELIB_COL_CASE(7)
    } else {
      GELIB_COL_CASE(8)
      GELIB_COL_CASE(9)
      GELIB_COL_CASE(11)
    }
#undef GELIB_COL_CASE
    if (do_b && (f & kColLastOfB) && W.ok) {  // the gradient rows of the b part go to global memory
      const ColPart& p = W.A.grad[(half1 ? 0 : kMaxParts) + h1.x];
      unsigned char* q = reinterpret_cast<unsigned char*>(p.base) + (unsigned long long)W.cell * p.cell_stride + 8ull * CPL * W.ch;
      for (int r = 0; r < nb; r++) red_row<CPL>(q + (unsigned long long)r * p.unit, lds_row<CPL>(W.smem + bacc + kRow * r));
    }
    if ((f & kColLastOfChunk) && !(f & kColLast)) W.next_chunk((f & kColDrain) != 0);
  } while (!(f & kColLast));
  cp_wait<0>();
}

// OWNED: the blocks of a cluster walk everything that is added to the gradient rows of their group, and only these are
// computed.  Each lane sums in slots of its own; at the end the blocks share the rows out and add up each other's sums, in
// the order of their ranks, through distributed shared memory.
template <int KMAX, int CPL, bool DOX, bool DOY, int THREADS, bool OWNED>
__global__ void __launch_bounds__(THREADS, 1) col_bwd_kernel(const __grid_constant__ ColArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr uint32_t kRow = Walk<CPL>::kRow;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // [part table][two chunk buffers][rings][b rows and their gradients (OWNED: sums), per warp]
  const uint32_t bufs = 16 * kColSlots, rings = bufs + 2 * kColChunkBytes, slots = rings + nwarps * Walk<CPL>::kRing;
  const uint32_t bval = slots + warp * kRow * (A.b_rows + (OWNED ? A.sum_rows : A.b_rows)) + 8 * CPL * lane;
  const uint32_t bacc = bval + kRow * A.b_rows;
  Walk<CPL> W(A, smem);
  W.set_lane((blockIdx.x * nwarps + warp) * 32 + lane);
  Row<CPL> zero;
#pragma unroll
  for (int c = 0; c < CPL; c++) zero.c[c] = 0ull;
  bool work = true;
  if constexpr (OWNED) {
    for (int r = 0; r < A.sum_rows; r++) sts_row<CPL>(smem + bacc + kRow * r, zero);
    work = __ldg(A.chunks + 4 * blockIdx.y + 1) > 0;  // a cluster may have more blocks than segments
  }
  if (work) walk_bwd<KMAX, CPL, DOX, DOY, OWNED>(W, bufs, rings + warp * Walk<CPL>::kRing, bval, bacc);
  if constexpr (OWNED) {
    const int rank = blockIdx.y % A.cluster;
    const int4* list = A.blob + __ldg(A.chunks + 4 * blockIdx.y + 3);
    const int rows = __ldg(&list[0].x);
    if (A.cluster > 1) cluster_sync();
    for (int r = rank; r < rows; r += A.cluster) {
      float2 s[CPL];
#pragma unroll
      for (int c = 0; c < CPL; c++) s[c] = make_float2(0.f, 0.f);
      for (int k = 0; k < A.cluster; k++) {
        const Row<CPL> v = lds_row_of<CPL>(smem + bacc + kRow * r, k);
#pragma unroll
        for (int c = 0; c < CPL; c++) {
          float re, im;
          unpack2(v.c[c], re, im);
          s[c].x += re;
          s[c].y += im;
        }
      }
      const int4 d = __ldg(&list[1 + r]);
      const ColPart& p = A.grad[d.x];
      unsigned char* q = reinterpret_cast<unsigned char*>(p.base) + (unsigned long long)W.cell * p.cell_stride + 8ull * CPL * W.ch;
      if (W.ok) red_row<CPL>(q + (unsigned long long)d.y * p.unit, to_row<CPL>(s));
    }
    if (A.cluster > 1) cluster_sync();  // a block's slots stay until every block has read them
  }
}

template <int KMAX, int CPL, bool DOX, bool DOY, int THREADS, bool OWNED = false>
cudaError_t launch_bwd(const ColArgs& a, cudaStream_t s, int block_warps = 0) {
  const size_t per_warp = Walk<CPL>::kRow * (kColRing + (size_t)a.b_rows + (OWNED ? a.sum_rows : a.b_rows));
  const unsigned warps = (a.nlanes + 31) / 32;
  int nw = (int)std::min<size_t>(THREADS / 32, (kColMaxSmem - kColFixedSmem) / per_warp);
  nw = block_warps > 0 ? std::min(nw, block_warps) : col_block_warps(warps, a.nsplits, nw);
  const size_t smem = kColFixedSmem + nw * per_warp;
  auto k = col_bwd_kernel<KMAX, CPL, DOX, DOY, THREADS, OWNED>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((warps + nw - 1) / nw, a.nsplits);
  cfg.blockDim = nw * 32;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = 1;
  cluster.val.clusterDim.y = a.cluster;
  cluster.val.clusterDim.z = 1;
  if (OWNED) {
    cfg.attrs = &cluster;
    cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, k, a);
}

template <bool DOX, bool DOY>
cudaError_t launch_bwd_k(const ColArgs& a, const ColPlan& p, cudaStream_t s) {
  if (p.cpl == 1) return launch_bwd<kColBlockBwd, 1, DOX, DOY, 384>(a, s);
  if (p.max_block <= 5) return launch_bwd<5, 2, DOX, DOY, 512>(a, s);
  return launch_bwd<kColBlockBwd, 2, DOX, DOY, 256>(a, s);
}

}  // namespace col
}  // namespace gelib_b200
