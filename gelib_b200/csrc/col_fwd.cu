// Forward column kernel (see col.h): r_l[m] (+)= sum_{m1} C_l[m1, m-m1] x[m1] y[m-m1], each product x y formed once for
// every output l of the pair.
#include <algorithm>

#include "col_device.h"

namespace gelib_b200 {
namespace col {

template <int K, int CPL, int NL>
__device__ __forceinline__ void fwd_step(Walk<CPL>& W, int st, const float2 (&a)[K][CPL], uint32_t bptr, bool add) {
  const int nl = st & 255, lo = (st >> 8) & 255, hi = (st >> 16) & 255;
  const unsigned span = hi - lo;
  constexpr int kCoefs = (NL + 3) / 4 * 4;
  f32x2 acc[NL][CPL];
#pragma unroll
  for (int j = 0; j < NL; j++)
#pragma unroll
    for (int c = 0; c < CPL; c++) acc[j][c] = 0ull;
#pragma unroll
  for (int blk = 0; blk < (K + 3) / 4; blk++) {
    if (hi >= 4 * blk && lo < 4 * blk + 4) {  // the same in every lane of the block
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int i = 4 * blk + e < K ? 4 * blk + e : K - 1;
        if (4 * blk + e >= K) continue;
        f32x2 p[CPL];
#pragma unroll
        for (int c = 0; c < CPL; c++) p[c] = 0ull;
        if ((unsigned)(i - lo) <= span) {  // outside the band there is no b row
          const Row<CPL> w = lds_row<CPL>(W.smem + (bptr - Walk<CPL>::kRow * i));
#pragma unroll
          for (int c = 0; c < CPL; c++) {
            float2 v;
            unpack2(w.c[c], v.x, v.y);
            p[c] = pack2(fmaf(-a[i][c].y, v.y, a[i][c].x * v.x), fmaf(a[i][c].y, v.x, a[i][c].x * v.y));
          }
        }
#pragma unroll
        for (int j = 0; j < NL; j += 4) {
          const Coefs q = coefs<NL>(W.smem + W.coef + (i * kCoefs + j) * 4);
#pragma unroll
          for (int c = 0; c < CPL; c++) {
            acc[j][c] = fma2(q.c[0], p[c], acc[j][c]);
            acc[j + 1][c] = fma2(q.c[1], p[c], acc[j + 1][c]);
            if (j + 2 < NL) {
              acc[j + 2][c] = fma2(q.c[2], p[c], acc[j + 2][c]);
              acc[j + 3][c] = fma2(q.c[3], p[c], acc[j + 3][c]);
            }
          }
        }
      }
    }
  }
  W.coef += K * kCoefs * 4;
  unsigned long long ad[NL];
#pragma unroll
  for (int j = 0; j < NL; j++)
    if (j < NL - 1 || nl == NL) ad[j] = W.addr(*reinterpret_cast<const uint4*>(W.smem + W.store + 16 * j));
  if (W.ok) {
#pragma unroll
    for (int j = 0; j < NL; j++)
      if (j < NL - 1 || nl == NL) {
        float v[2 * CPL];
#pragma unroll
        for (int c = 0; c < CPL; c++) unpack2(acc[j][c], v[2 * c], v[2 * c + 1]);
        if (add) {
          float o[2 * CPL];
          if constexpr (CPL == 2)
            asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "l"(ad[j]));
          else
            asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(o[0]), "=f"(o[1]) : "l"(ad[j]));
#pragma unroll
          for (int e = 0; e < 2 * CPL; e++) v[e] += o[e];
        }
        if constexpr (CPL == 2)
          asm volatile("st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(ad[j]), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
        else
          asm volatile("st.global.cs.v2.f32 [%0], {%1, %2};" ::"l"(ad[j]), "f"(v[0]), "f"(v[1]));
      }
  }
  W.store += 16 * nl;
}

// bval: byte offset of the lane's slot of b row 0.
template <int K, int CPL>
__device__ __forceinline__ void fwd_segment(Walk<CPL>& W, const int4 h, int lb, uint32_t bval, bool add) {
  constexpr int NLMAX = K + 1 < kColMaxNl ? K + 1 : kColMaxNl;
  constexpr uint32_t kRow = Walk<CPL>::kRow;
  float2 a[K][CPL];
  W.template take<0>(a);
  const int nsteps = h.x >> 16;
  uint32_t bptr = bval + kRow * (h.y + lb);  // the b row that entry 0 meets
  const uint32_t steps = W.seg + 32;
  int next = *reinterpret_cast<const int*>(W.smem + steps);
  for (int s = 0; s < nsteps; s++, bptr += kRow) {
    const int st = next;
    next = *reinterpret_cast<const int*>(W.smem + steps + 4 * s + 4);  // past the last one: another word of the chunk
    const int nl2 = ((st & 255) + 1) >> 1;
    if (nl2 == 1) fwd_step<K, CPL, 2>(W, st, a, bptr, add);
    if constexpr (NLMAX >= 4) if (nl2 == 2) fwd_step<K, CPL, 4>(W, st, a, bptr, add);
    if constexpr (NLMAX >= 6) if (nl2 == 3) fwd_step<K, CPL, 6>(W, st, a, bptr, add);
    if constexpr (NLMAX >= 8) if (nl2 == 4) fwd_step<K, CPL, 8>(W, st, a, bptr, add);
    if constexpr (NLMAX >= 10) if (nl2 == 5) fwd_step<K, CPL, 10>(W, st, a, bptr, add);
  }
  W.seg = steps + 4 * ((nsteps + 3) & ~3);
}

template <int KMAX, int CPL, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) col_fwd_kernel(const __grid_constant__ ColArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // [part table][two chunk buffers][rings][b rows, per warp]
  const uint32_t bufs = 16 * kColSlots, rings = bufs + 2 * kColChunkBytes, slots = rings + nwarps * Walk<CPL>::kRing;
  const uint32_t bval = slots + warp * Walk<CPL>::kRow * A.b_rows + 8 * CPL * lane;
  Walk<CPL> W(A, smem);
  W.set_lane((blockIdx.x * nwarps + warp) * 32 + lane);
  W.start(0, bufs, rings + warp * Walk<CPL>::kRing);
  const bool add = A.accumulate != 0;
  int f;
  do {
    const int4 h = *reinterpret_cast<const int4*>(smem + W.seg);
    const int lb = *reinterpret_cast<const int*>(smem + W.seg + 20), kb = h.x & 255;
    f = (h.x >> 8) & 255;
    if (f & kColFirstOfB) W.take_to(bval, 2 * lb + 1);
#define GELIB_COL_CASE(N) \
  if constexpr (N <= KMAX) \
    if (kb == N) fwd_segment<N, CPL>(W, h, lb, bval, add);
    if (kb <= 5) {
      GELIB_COL_CASE(1)
      GELIB_COL_CASE(3)
      GELIB_COL_CASE(5)
    } else if (kb <= 11) {
      GELIB_COL_CASE(7)
      GELIB_COL_CASE(9)
      GELIB_COL_CASE(11)
    } else {
      GELIB_COL_CASE(13)
      GELIB_COL_CASE(15)
      GELIB_COL_CASE(17)
    }
#undef GELIB_COL_CASE
    if ((f & kColLastOfChunk) && !(f & kColLast)) W.next_chunk((f & kColDrain) != 0);
  } while (!(f & kColLast));
  cp_wait<0>();
}

template <int KMAX, int CPL, int THREADS>
cudaError_t launch_fwd(const ColArgs& a, cudaStream_t s) {
  const size_t per_warp = Walk<CPL>::kRow * (kColRing + (size_t)a.b_rows);
  const unsigned warps = (a.nlanes + 31) / 32;
  int nw = (int)std::min<size_t>(THREADS / 32, (kColMaxSmem - kColFixedSmem) / per_warp);
  nw = col_block_warps(warps, a.nsplits, nw);
  const size_t smem = kColFixedSmem + nw * per_warp;
  auto k = col_fwd_kernel<KMAX, CPL, THREADS>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<dim3((warps + nw - 1) / nw, a.nsplits), nw * 32, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace col

int launch_col_fwd(const VecCall& c, cudaStream_t s, bool* plan_others) {
  static const char* fn = "SO3vec_addCGproduct";
  ColArgs a;
  ColPlan plan;
  if (!col_setup(c, false, &a, &plan)) return -1;
  if (!plan.dev) return GELIB_CUDA_ERROR;
  *plan_others = plan.plan_others;
  if (a.nsplits == 0 || c.plan_only) return GELIB_OK;
  cudaError_t e;
  if (plan.cpl == 1) e = col::launch_fwd<17, 1, 512>(a, s);
  else if (plan.max_block <= 9) e = col::launch_fwd<9, 2, 512>(a, s);
  else e = col::launch_fwd<17, 2, 384>(a, s);
  if (e != cudaSuccess) return check_cuda(e, fn, "column forward kernel launch");
  count_launch();
  return GELIB_OK;
}

}  // namespace gelib_b200
