// Channel mixing of an SO3part by a complex weight matrix, and its two gradients:
//
//   mode 0   r[row][j]  = sum_i x[row][i] W[i][j]              (the product  part * W)
//   mode 1   r[row][i]  = sum_j x[row][j] conj(W[i][j])        (gradient of the part: g * W^H)
//   back_w   Wg[i][j]  += sum_row conj(x[row][i]) g[row][j]    (gradient of the weights: x^H * g)
//
// rows = every (cell, m) of the part; all arrays dense complex64.  In GElib this is torch.matmul per part
// (python/src/gelib/SO3vec.py:174-177, python/src/gelib/SO3weights.py:22-85); with 16 channels the library GEMM runs at
// a tenth of the memory rate, and the mixing of a point cloud's first layer cost as much as a fifth of its product.
//
// Both kernels stage tiles of rows in shared memory (asynchronous copies, one tile in flight while the other is worked on) and
// give a thread a tile of the result: 4 rows x 2 columns of the product, 4 x 4 entries of the weight gradient, so that a 16-byte
// load feeds 11 (16) multiply-adds; products are summed in two halves, and 8, 16 and 32 channels on both sides, and 16 with 32, have a
// body of their own (us without / with: 16 x 16, 3.2 million rows 240 / 197; 1.6 million, 16 x 32 221 / 200, 32 x 16 223 / 175).  Measured
// against one output element (one (i,j) sum) per thread, us, product / adjoint / weight gradient: 16 x 16 channels, 3.2 million rows
// 214 / 238 / 396 -> 197 / 197 / 247; 32 x 32, 400000 96 / 156 / 194 -> 93 / 95 / 104; 8 x 8, 2 million 104 / 104 / 132 -> 57 / 57 / 79; 12 x 20, 500000
// 76 / 70 / 85 -> 49 / 51 / 62; 64 x 64, 100000 197 / 198 / 235 -> 100 / 100 / 98.  At 16 channels the multiply-adds alone take 91 us and the memory 126.
#include <cuda_pipeline.h>

#include <algorithm>

#include "plan.h"

namespace gelib_b200 {

namespace {

constexpr int kMixMaxN = 64;   // channels on either side
constexpr int kThreads = 256;

// How rows of n complex numbers are copied: 16 bytes at a time where they are aligned, `per` copies a row.
struct RowCopy {
  int per, shift;  // shift: of a power of two, else -1
  bool wide;
};

// Copies `rows` rows to shared rows of `pitch` bytes, asynchronously.
__device__ __forceinline__ void tile_copy_async(unsigned char* dst, int pitch, const float2* src, int rows, const RowCopy c) {
  for (int e = threadIdx.x; e < rows * c.per; e += kThreads) {
    const int row = c.shift >= 0 ? e >> c.shift : e / c.per, at = e - row * c.per;
    if (c.wide) __pipeline_memcpy_async(dst + row * pitch + 16 * at, src + 2 * e, 16);
    else __pipeline_memcpy_async(dst + row * pitch + 8 * at, src + e, 8);
  }
}

// s += a b
__device__ __forceinline__ void mac(float2& s, float ar, float ai, float br, float bi) {
  s.x = fmaf(ar, br, s.x); s.x = fmaf(-ai, bi, s.x);
  s.y = fmaf(ar, bi, s.y); s.y = fmaf(ai, br, s.y);
}

// r[row][j] = sum_k x[row][k] M[k][j], M = W (mode 0) or its adjoint (mode 1).  A thread has columns 2 tx, 2 tx + 1 of the rows
// ty, ty + TY, ..; odd lengths are padded with zeros in shared memory.  R: rows per thread.  NK, NJ: the
// channel counts where they are known here.  CHAIN: for up to two products, whose two halves of one product each would cost a
// rounding more than one chain (error 4.10e-8, 3.93e-8).
template <int MODE, int R, int NK, int NJ, bool CHAIN = false>
__global__ void __launch_bounds__(kThreads, 4) mix_kernel(float2* __restrict__ r, const float2* __restrict__ x, const float2* __restrict__ W,
                                                       long long rows, int nk_arg, int nj_arg, int w_cols, int ty_n_arg, RowCopy copy_x, bool wide_r) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int nk = NK > 0 ? NK : nk_arg, nj = NJ > 0 ? NJ : nj_arg;
  const int tx_n = (nj + 1) / 2, nk2 = (nk + 1) / 2, ty_n = NK > 0 ? kThreads / tx_n : ty_n_arg, tile = ty_n * R;
  const int pitch = 16 * nk2 + 16;                        // bytes of a staged row of x
  float4* Ms = reinterpret_cast<float4*>(sm);             // [2 nk2][tx_n]: two columns each
  unsigned char* xs = sm + 32 * nk2 * tx_n;               // two tiles
  const long long stride = (long long)gridDim.x * tile;
  long long row0 = (long long)blockIdx.x * tile;
  if (row0 < rows) tile_copy_async(xs, pitch, x + row0 * nk, (int)min((long long)tile, rows - row0), copy_x);
  __pipeline_commit();
  for (int e = threadIdx.x; e < 4 * nk2 * tx_n; e += kThreads) {  // neighbouring threads read neighbouring weights
    int k, j;
    if (MODE == 0) {
      k = e / (2 * tx_n);
      j = e - k * 2 * tx_n;
    } else {
      j = e / (2 * nk2);
      k = e - j * 2 * nk2;
    }
    float2 w = make_float2(0.f, 0.f);
    if (k < nk && j < nj) {
      w = MODE == 0 ? W[k * w_cols + j] : W[j * w_cols + k];
      if (MODE == 1) w.y = -w.y;
    }
    reinterpret_cast<float2*>(Ms)[k * 2 * tx_n + j] = w;
  }
  if (nk & 1)
    for (int row = threadIdx.x; row < 2 * tile; row += kThreads) *reinterpret_cast<float2*>(xs + row * pitch + 8 * nk) = make_float2(0.f, 0.f);
  const int tx = threadIdx.x % tx_n, ty = threadIdx.x / tx_n;
  const bool works = ty < ty_n;
  for (int buf = 0; row0 < rows; row0 += stride, buf ^= 1) {
    const int nr = (int)min((long long)tile, rows - row0);
    const long long next = row0 + stride;
    if (next < rows) tile_copy_async(xs + (buf ^ 1) * tile * pitch, pitch, x + next * nk, (int)min((long long)tile, rows - next), copy_x);
    __pipeline_commit();
    __pipeline_wait_prior(1);
    __syncthreads();
    if (works) {
      float2 s[R][2], t[R][2];  // sums over even and over odd k
#pragma unroll
      for (int i = 0; i < R; i++) s[i][0] = s[i][1] = t[i][0] = t[i][1] = make_float2(0.f, 0.f);
      const unsigned char* xr = xs + buf * tile * pitch + ty * pitch;
      const float4* m = Ms + tx;
#pragma unroll 2
      for (int k = 0; k < nk2; k++) {  // rows past the end of the part read what the tile held before
        const float4 w0 = m[2 * k * tx_n], w1 = m[(2 * k + 1) * tx_n];
#pragma unroll
        for (int i = 0; i < R; i++) {
          const float4 a = *reinterpret_cast<const float4*>(xr + i * ty_n * pitch + 16 * k);
          mac(s[i][0], a.x, a.y, w0.x, w0.y);
          mac(s[i][1], a.x, a.y, w0.z, w0.w);
          mac(CHAIN ? s[i][0] : t[i][0], a.z, a.w, w1.x, w1.y);
          mac(CHAIN ? s[i][1] : t[i][1], a.z, a.w, w1.z, w1.w);
        }
      }
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int row = ty + i * ty_n;
#pragma unroll
        for (int c = 0; c < 2; c++) {
          s[i][c].x += t[i][c].x;
          s[i][c].y += t[i][c].y;
        }
        if (row < nr) {
          float2* p = r + (row0 + row) * nj + 2 * tx;
          if (wide_r) {
            __stcs(reinterpret_cast<float4*>(p), make_float4(s[i][0].x, s[i][0].y, s[i][1].x, s[i][1].y));
          } else {
            __stcs(p, s[i][0]);
            if (2 * tx + 1 < nj) __stcs(p + 1, s[i][1]);
          }
        }
      }
    }
    __syncthreads();  // the tile may be overwritten by the copy after next
  }
}

// The block's share of sum_row conj(x[row][i]) g[row][j].  Threads: tiles of 4 x 4 entries, times groups of rows;
// the groups' sums meet in shared memory, the blocks' in global memory.
// FOLD, where at most two groups fit (more than 32 x 32 channels) and a thread's rows are many: every eight tiles it adds its sums
// to those of the tiles before.  It takes registers for two blocks on an SM in place of three.  400000 rows, error against 64-bit sums
// and us without / with: 64 x 64 channels 8.4e-7 / 4.2e-7, 347 / 342; 48 x 48 8.5e-7 / 4.9e-7, 275 / 283.
template <bool FOLD>
__global__ void __launch_bounds__(kThreads) mix_back_w_kernel(float* __restrict__ Wg, const float2* __restrict__ x, const float2* __restrict__ g,
                                                              long long rows, int ni, int nj, long long rows_per_block, int tile_rows, int groups, RowCopy copy_x, RowCopy copy_g) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int ti_n = (ni + 3) / 4, tj_n = (nj + 3) / 4, tiles = ti_n * tj_n;
  const int px = 32 * ti_n + 16, pg = 32 * tj_n + 16, tile = tile_rows * (px + pg);
  if ((ni | nj) & 3) {  // padding
    for (int e = threadIdx.x; e < 2 * tile / 16; e += kThreads) reinterpret_cast<float4*>(sm)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
  }
  const long long begin = (long long)blockIdx.x * rows_per_block, end = min(rows, begin + rows_per_block);
  auto copy_tile = [&](int buf, long long row0) {
    const int nr = (int)min((long long)tile_rows, end - row0);
    tile_copy_async(sm + buf * tile, px, x + row0 * ni, nr, copy_x);
    tile_copy_async(sm + buf * tile + tile_rows * px, pg, g + row0 * nj, nr, copy_g);
  };
  if (begin < end) copy_tile(0, begin);
  __pipeline_commit();
  const int at = threadIdx.x % tiles, group = threadIdx.x / tiles, ti = at / tj_n, tj = at - ti * tj_n;
  float2 s[4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) s[a][b] = make_float2(0.f, 0.f);
  float2 before[FOLD ? 4 : 1][4];
  if constexpr (FOLD) {
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) before[a][b] = make_float2(0.f, 0.f);
  }
  int buf = 0, k = 0;
  for (long long row0 = begin; row0 < end; row0 += tile_rows, buf ^= 1, k++) {
    const int nr = (int)min((long long)tile_rows, end - row0);
    if (row0 + tile_rows < end) copy_tile(buf ^ 1, row0 + tile_rows);
    __pipeline_commit();
    __pipeline_wait_prior(1);
    __syncthreads();
    if (group < groups) {
      const unsigned char* xp = sm + buf * tile + 32 * ti;
      const unsigned char* gp = sm + buf * tile + tile_rows * px + 32 * tj;
#pragma unroll 2
      for (int row = group; row < nr; row += groups) {
        const float4 x0 = *reinterpret_cast<const float4*>(xp + row * px), x1 = *reinterpret_cast<const float4*>(xp + row * px + 16);
        const float4 g0 = *reinterpret_cast<const float4*>(gp + row * pg), g1 = *reinterpret_cast<const float4*>(gp + row * pg + 16);
        const float2 xv[4] = {{x0.x, x0.y}, {x0.z, x0.w}, {x1.x, x1.y}, {x1.z, x1.w}};
        const float2 gv[4] = {{g0.x, g0.y}, {g0.z, g0.w}, {g1.x, g1.y}, {g1.z, g1.w}};
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int b = 0; b < 4; b++) mac(s[a][b], xv[a].x, -xv[a].y, gv[b].x, gv[b].y);
      }
      if constexpr (FOLD)
        if ((k & 7) == 7 || row0 + tile_rows >= end) {
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) {
              before[a][b].x += s[a][b].x;
              before[a][b].y += s[a][b].y;
              s[a][b] = make_float2(0.f, 0.f);
            }
        }
    }
    __syncthreads();  // the tiles may be overwritten by the copy after next
  }
  float2* sums = reinterpret_cast<float2*>(sm);  // [group][tile][16]
  if (group < groups) {
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) sums[(group * tiles + at) * 16 + 4 * a + b] = FOLD ? before[FOLD ? a : 0][b] : s[a][b];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ni * nj; e += kThreads) {
    const int i = e / nj, j = e - i * nj, at_e = (i / 4) * tj_n + j / 4, in = 4 * (i % 4) + j % 4;
    float2 t = make_float2(0.f, 0.f);
    for (int q = 0; q < groups; q++) {
      const float2 v = sums[(q * tiles + at_e) * 16 + in];
      t.x += v.x;
      t.y += v.y;
    }
    atomicAdd(Wg + 2 * e, t.x);
    atomicAdd(Wg + 2 * e + 1, t.y);
  }
}

bool aligned(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }
RowCopy row_copy(const void* p, int n) {
  RowCopy c;
  c.wide = n % 2 == 0 && aligned(p);
  c.per = c.wide ? n / 2 : n;
  c.shift = -1;
  for (int k = 0; k < 7; k++)
    if (c.per == 1 << k) c.shift = k;
  return c;
}

}  // namespace

int launch_mix(float* r, const float* x, const float* W, long long rows, int n_in, int n_out, int mode, cudaStream_t s) {
  static const char* fn = "SO3part_mix";
  if (n_in < 1 || n_out < 1 || n_in > kMixMaxN || n_out > kMixMaxN) return fail(GELIB_SKIPPED, fn, "more than 64 channels");
  if (rows <= 0) return GELIB_OK;
  const int nk = mode == 0 ? n_in : n_out, nj = mode == 0 ? n_out : n_in;  // contraction length, output channels
  const int tx_n = (nj + 1) / 2, nk2 = (nk + 1) / 2, pitch = 16 * nk2 + 16;
  const int most = std::min(kThreads / tx_n, 35000 / (4 * pitch));  // groups of rows; a tile of at most 34 KB
  // Few rows: one to a thread, in tiles for two blocks on every SM.  More: four, in tiles for at least two.  us, tiles of full size and
  // four rows a thread always / as here: 5 x 3 channels, 3000 rows 4.9 / 3.2, 30000 4.7 / 3.7, 100000 5.9 / 5.1; 32 x 16, 3000 5.8 / 3.6;
  // 64 x 4, 3000 6.8 / 3.8; 16 x 8, 7000 4.3 / 3.1.  Mean over 37 pairs of counts, against full tiles: 7000 rows, one row a thread 0.83, four 0.88;
  // 14000 rows 0.99 and 0.90.
  const int R = rows <= 10000 ? 1 : 4;
  const int ty_n = (int)std::min<long long>(most, (rows + R * 296 - 1) / (R * 296));
  const int tile = ty_n * R;
  const size_t smem = (size_t)32 * nk2 * tx_n + (size_t)2 * tile * pitch;
  const unsigned blocks = (unsigned)std::min<long long>((rows + tile - 1) / tile, 148LL * 8);
  auto k = mode == 0 ? mix_kernel<0, 4, 0, 0> : mix_kernel<1, 4, 0, 0>;
  if (nk <= 2 && R == 1) k = mode == 0 ? mix_kernel<0, 1, 0, 0, true> : mix_kernel<1, 1, 0, 0, true>;
  else if (nk <= 2) k = mode == 0 ? mix_kernel<0, 4, 0, 0, true> : mix_kernel<1, 4, 0, 0, true>;
  else if (R == 1) k = mode == 0 ? mix_kernel<0, 1, 0, 0> : mix_kernel<1, 1, 0, 0>;
  else if (ty_n == kThreads / tx_n) {  // the bodies of known channel counts take that many groups
#define GELIB_MIX_BODY(a, b) if (nk == a && nj == b) k = mode == 0 ? mix_kernel<0, 4, a, b> : mix_kernel<1, 4, a, b>;
    GELIB_MIX_BODY(8, 8) GELIB_MIX_BODY(16, 16) GELIB_MIX_BODY(32, 32) GELIB_MIX_BODY(16, 32) GELIB_MIX_BODY(32, 16)
#undef GELIB_MIX_BODY
  }
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    k<<<blocks, kThreads, smem, s>>>(reinterpret_cast<float2*>(r), reinterpret_cast<const float2*>(x), reinterpret_cast<const float2*>(W), rows, nk,
                                     nj, n_out, ty_n, row_copy(x, nk), nj % 2 == 0 && aligned(r));
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return check_cuda(e, fn, "mixing kernel launch");
  count_launch();
  return GELIB_OK;
}

int launch_mix_back_w(float* Wg, const float* x, const float* g, long long rows, int n_in, int n_out, cudaStream_t s) {
  static const char* fn = "SO3part_mix_back_w";
  if (n_in < 1 || n_out < 1 || n_in > kMixMaxN || n_out > kMixMaxN) return fail(GELIB_SKIPPED, fn, "more than 64 channels");
  if (rows <= 0) return GELIB_OK;
  const int ti_n = (n_in + 3) / 4, tj_n = (n_out + 3) / 4, tiles = ti_n * tj_n;
  // Tiles of about 32 KB; smaller ones, down to 64 rows, where there would be fewer than a block per SM.
  const long long share = std::max<long long>(64, (rows / 148 + 15) / 16 * 16);
  const int tile_rows = (int)std::min<long long>(std::min(256, 32768 / (32 * (ti_n + tj_n) + 32) / 16 * 16), share);
  const bool fold = kThreads / tiles <= 2;
  const long long want_blocks = std::min<long long>((rows + tile_rows - 1) / tile_rows, 148LL * (fold ? 2 : 3));
  long long rpb = (rows + want_blocks - 1) / want_blocks;
  rpb = (rpb + tile_rows - 1) / tile_rows * tile_rows;
  const unsigned blocks = (unsigned)((rows + rpb - 1) / rpb);
  // As many groups as fit, of at least four rows: their sums are added one after the other.  With the tiles above, us, zeroing of the
  // result included: 5 x 3 channels, 300 rows 7.0 -> 4.8, 3000 6.8 -> 4.7; 16 x 8, 3000 6.3 -> 5.6.
  const int groups = (int)std::min<long long>(kThreads / tiles, std::max<long long>(1, rpb / 4));
  const size_t smem = std::max((size_t)2 * tile_rows * (32 * (ti_n + tj_n) + 32), (size_t)groups * tiles * 128);
  auto k = fold ? mix_back_w_kernel<true> : mix_back_w_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    k<<<blocks, kThreads, smem, s>>>(Wg, reinterpret_cast<const float2*>(x), reinterpret_cast<const float2*>(g), rows, n_in, n_out, rpb,
                                     tile_rows, groups, row_copy(x, n_in), row_copy(g, n_out));
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return check_cuda(e, fn, "weight gradient kernel launch");
  count_launch();
  return GELIB_OK;
}

}  // namespace gelib_b200
