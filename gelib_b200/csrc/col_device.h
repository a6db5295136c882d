// Device side of the column kernels (see col.h).
#pragma once
#include "col.h"
#include "f32x2.h"

namespace gelib_b200 {
namespace col {

template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// CPL complex numbers of a lane.
template <int CPL>
struct Row {
  f32x2 c[CPL];
};
template <int CPL>
__device__ __forceinline__ Row<CPL> lds_row(const unsigned char* p) {
  Row<CPL> v;
  if constexpr (CPL == 2) {
    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(p);
    v.c[0] = q.x;
    v.c[1] = q.y;
  } else {
    v.c[0] = *reinterpret_cast<const f32x2*>(p);
  }
  return v;
}
template <int CPL>
__device__ __forceinline__ void sts_row(unsigned char* p, const Row<CPL>& v) {
  if constexpr (CPL == 2) *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.c[0], v.c[1]);
  else *reinterpret_cast<f32x2*>(p) = v.c[0];
}
template <int CPL>
__device__ __forceinline__ void red_row(unsigned char* p, const Row<CPL>& v) {
  float a, b;
  unpack2(v.c[0], a, b);
  if constexpr (CPL == 2) {
    float c, d;
    unpack2(v.c[1], c, d);
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d));
  } else {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b));
  }
}

// Coefficients of a step's next four output l, each twice for the packed multiply-adds.  They are paired in registers: read as
// pairs they took the rate of shared memory (diagonal product, both gradients, maxl 8 x 128 channels, batch 2048 4919 -> 4697 us,
// maxl 6 x 33, batch 4000 1073 -> 1015; gradient of y, maxl 8 x 128 4493 -> 4299).  For a step of two l nothing would be saved: the
// walk holds its coefficients twice.
struct Coefs {
  f32x2 c[4];
};
template <int NL>
__device__ __forceinline__ Coefs coefs(const unsigned char* p) {
  Coefs q;
  if constexpr (NL == 2) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    q.c[0] = v.x;
    q.c[1] = v.y;
  } else {
    const float4 v = *reinterpret_cast<const float4*>(p);
    q.c[0] = pack2(v.x, v.x);
    q.c[1] = pack2(v.y, v.y);
    q.c[2] = pack2(v.z, v.z);
    q.c[3] = pack2(v.w, v.w);
  }
  return q;
}

// Header of a chunk: {byte offsets of the request list, the store list, the segments, the coefficients}, then
// {address records, 0, 0, 0} and the address records.  A segment: {a rows | flags<<8 | steps<<16, d = m - mlo of the first
// step, first a row, a part}, {b part, lb, first row of the sums (owned walks), 0}, and one int per step (padded to four): nl | first entry of the band<<8 |
// last<<16.
template <int CPL>
struct Walk {
  static constexpr uint32_t kRow = 256 * CPL, kRing = kRow * kColRing;
  const ColArgs& A;
  unsigned char* smem;
  uint32_t ring;    // byte offset of the warp's ring in smem
  uint32_t pb;      // kRow * rows taken + 8 CPL * lane
  uint32_t cell, ch;
  bool ok;
  uint32_t req, store, seg, coef;  // byte offsets in smem: cursors into the chunk
  int chunk, chunk_end;
  uint32_t buf0, part_off;
  int which;

  __device__ __forceinline__ Walk(const ColArgs& a, unsigned char* s) : A(a), smem(s) {}

  __device__ __forceinline__ unsigned long long addr(const uint4 q) const {
    unsigned long long p = ((unsigned long long)q.y << 32) | q.x;
    p += (unsigned long long)cell * q.z;
    return p + (unsigned long long)ch * q.w;
  }
  // A record {slot, v} becomes {address of the row in cell 0, channel 0; cell stride; lane stride}.
  __device__ __forceinline__ uint4 resolve(const int4 r) const {
    const uint4 p = *reinterpret_cast<const uint4*>(smem + part_off + 16 * r.x);
    const unsigned long long b = (((unsigned long long)p.y << 32) | p.x) + (unsigned long long)(unsigned)r.y * p.z;
    const int side = r.x / kMaxParts;
    return make_uint4((unsigned)b, (unsigned)(b >> 32), p.w, side == 0 ? A.ch_stride[0] : side == 1 ? A.ch_stride[1] : A.ch_stride[2]);
  }
  // A row may be one number per cell (lane stride 0), which both columns of a lane get.
  __device__ __forceinline__ void request(unsigned long long src, uint32_t lane_stride, uint32_t pos) const {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem) + ring + (pos & (kRing - 1));
    if constexpr (CPL == 1) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
    } else if (lane_stride == 0) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8), "l"(src) : "memory");
    } else {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
    cp_commit();
  }
  __device__ __forceinline__ Row<CPL> row(int j) const { return lds_row<CPL>(smem + ring + ((pb + kRow * j) & (kRing - 1))); }
  __device__ __forceinline__ uint4 req_rec(int j) const { return *reinterpret_cast<const uint4*>(smem + req + 16 * j); }
  // Requests k <= N rows, four at a time: addresses are formed before the first copy is issued, since copies are barriers
  // to the compiler and the latency of a record would otherwise be paid per row.  Moves the cursors.
  template <int N>
  __device__ __forceinline__ void refill(int k) {
#pragma unroll
    for (int j0 = 0; j0 < N; j0 += 4) {
      unsigned long long ad[4];
      uint32_t ls[4];
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j0 + j < N) {
          const uint4 q = req_rec(min(j0 + j, k - 1));
          ad[j] = addr(q);
          ls[j] = q.w;
        }
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j0 + j < N && j0 + j < k) request(ad[j], ls[j], pb + kRow * (j0 + j));
    }
    req += 16 * k;
    pb += kRow * k;
  }
  // The next N - OFF rows into registers.
  template <int OFF, int N>
  __device__ __forceinline__ void take(float2 (&v)[N][CPL]) {
    constexpr int B = N - OFF < 8 ? N - OFF : 8;
    if constexpr (B > 0) {
      cp_wait<kColRing - B>();
#pragma unroll
      for (int j = 0; j < B; j++) {
        const Row<CPL> r = row(j);
#pragma unroll
        for (int c = 0; c < CPL; c++) unpack2(r.c[c], v[OFF + j][c].x, v[OFF + j][c].y);
      }
      refill<B>(B);
      take<OFF + B>(v);
    }
  }
  // The next n rows into the lane's slots from dst on.
  __device__ __forceinline__ void take_to(uint32_t dst, int n) {
    for (int r = 0; r < n; r += 4) {
      const int k = min(4, n - r);
      cp_wait<kColRing - 4>();
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j < k) sts_row<CPL>(smem + dst + kRow * (r + j), row(j));
      refill<4>(k);
    }
  }

  __device__ __forceinline__ void fetch(int c) {  // copies chunk c into the buffer that is not in use
    const int* t = A.chunks + 4 * A.nsplits + 2 * c;
    const int off = __ldg(t), size = __ldg(t + 1);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem) + buf0 + (which ^ 1) * kColChunkBytes;
    for (int e = threadIdx.x; e < size; e += blockDim.x)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(A.blob + off + e) : "memory");
    cp_commit();
  }
  // Makes chunk `chunk` (already copied) the current one and starts the copy of the next.  A thread resolves the address
  // records that it copied itself, so one barrier is enough.
  __device__ __forceinline__ void enter() {
    which ^= 1;
    const uint32_t b = buf0 + which * kColChunkBytes;
    // the records' count lies in a word that another thread may have copied: it is read from global memory
    const int* t = A.chunks + 4 * A.nsplits + 2 * chunk;
    const int nrec = __ldg(&A.blob[__ldg(t) + 1].x);
    for (int e = threadIdx.x; e < nrec + 2; e += blockDim.x)
      if (e >= 2) {
        uint4* q = reinterpret_cast<uint4*>(smem + b + 16 * e);
        *q = resolve(*reinterpret_cast<const int4*>(q));
      }
    __syncthreads();
    const int4 h = *reinterpret_cast<const int4*>(smem + b);
    req = b + h.x;
    store = b + h.y;
    seg = b + h.z;
    coef = b + h.w;
    if (chunk + 1 < chunk_end) fetch(chunk + 1);
  }
  __device__ __forceinline__ void next_chunk(bool drain) {
    if (drain) cp_wait<0>();
    chunk++;
    enter();
  }

  // part table, first chunk, ring prologue
  __device__ __forceinline__ void start(uint32_t part_offset, uint32_t buffers, uint32_t ring_offset) {
    part_off = part_offset;
    buf0 = buffers;
    ring = ring_offset;
    which = 1;
    for (int e = threadIdx.x; e < kColSlots; e += blockDim.x) {
      const ColPart& p = A.part[e];
      const unsigned long long b = reinterpret_cast<unsigned long long>(p.base);
      *reinterpret_cast<uint4*>(smem + part_off + 16 * e) = make_uint4((unsigned)b, (unsigned)(b >> 32), p.unit, p.cell_stride);
    }
    const int* sp = A.chunks + 4 * blockIdx.y;
    chunk = __ldg(sp);
    chunk_end = chunk + __ldg(sp + 1);
    const int pro = __ldg(sp + 2);
    fetch(chunk);
    cp_wait<0>();
    __syncthreads();  // the part table
    enter();
    const uint32_t lane = threadIdx.x & 31;
    pb = 8 * CPL * lane;
    for (int j = 0; j < kColRing; j++) {
      const uint4 q = resolve(__ldg(A.blob + pro + j));
      request(addr(q), q.w, pb + kRow * j);
    }
  }

  __device__ __forceinline__ void set_lane(unsigned i) {
    ok = i < A.nlanes;
    if (!ok) i = A.nlanes - 1;
    cell = i / A.n;
    ch = i - cell * A.n;
  }
};

}  // namespace col
}  // namespace gelib_b200
