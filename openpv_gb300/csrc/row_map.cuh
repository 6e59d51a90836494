// row_map.cuh -- walking a layer's neurons in restricted order with their extended indices.
//
// A restricted row (one y of one batch element) is nx * nf contiguous values both in the restricted
// and in the extended layout, so a unit of VEC consecutive values needs one division by the units of a
// row and one by the rows of an image -- multiplications by a precomputed reciprocal -- instead of the
// four 64-bit divisions per neuron that locating it through (f, x, y, b) takes.
#pragma once

#include "pvgpu_internal.cuh"

namespace pvgpu {

// n / d for n < 2^31 by multiplication: with s = ceil(log2 d) and m = ceil(2^(31 + s) / d), the
// quotient is (n * m) >> (31 + s): n * (m d - 2^(31 + s)) < 2^31 * d <= 2^(31 + s).
struct FastDiv {
   uint32_t d;
   uint64_t m;
   int shift;
   static FastDiv make(uint32_t d) {
      int s = 0;
      while ((1ull << s) < d) s++;
      return FastDiv{d, ((1ull << (31 + s)) + d - 1) / d, 31 + s};
   }
   // m < 2^32: d > 2^(s - 1) gives 2^(31 + s) / d < 2^32
   __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const { return (uint32_t)((n * m) >> shift); }
};

struct RowMap {
   int64_t units;        // VEC values each
   int64_t extNum;       // extended values per batch element
   int64_t extRow, extOrg;
   FastDiv perRow, rows;
   int64_t rowLen;
   int ny;
};

struct RowAt {
   int64_t res, ext;
   int b;
};

// 4 where whole rows come in aligned groups of four values, else 1.  `all`: every pointer's bits or-ed.
inline int row_vec(const Loc &l, uintptr_t all) {
   const int64_t n = (int64_t)l.nx * l.nf;
   return n % 4 == 0 && (int64_t)l.lt * l.nf % 4 == 0 && (int64_t)l.nxExt() * l.nf % 4 == 0 && all % 16 == 0 ? 4 : 1;
}

inline RowMap row_map(const Loc &l, int vec) {
   RowMap m;
   m.rowLen = (int64_t)l.nx * l.nf;
   m.units = l.numRes() * l.nb / vec;
   m.extNum = l.numExt();
   m.extRow = (int64_t)l.nxExt() * l.nf;
   m.extOrg = (int64_t)l.up * m.extRow + (int64_t)l.lt * l.nf;
   m.ny = l.ny;
   if (m.units <= 0x7fffffffLL) {
      m.perRow = FastDiv::make((uint32_t)(m.rowLen / vec));
      m.rows = FastDiv::make((uint32_t)l.ny);
   }
   return m;
}

// WIDE: 2^31 units or more
template <int VEC, bool WIDE>
__device__ __forceinline__ RowAt row_at(const RowMap &m, int64_t u) {
   RowAt a;
   int64_t row, j, b;
   if (WIDE) {
      row = u * VEC / m.rowLen;
      b = row / m.ny;
      j = u * VEC - row * m.rowLen;
   } else {
      const uint32_t r = m.perRow.div((uint32_t)u);
      row = r;
      b = m.rows.div(r);
      j = (int64_t)((uint32_t)u - r * m.perRow.d) * VEC;
   }
   a.res = u * VEC;
   a.ext = b * m.extNum + (row - b * m.ny) * m.extRow + m.extOrg + j;
   a.b = (int)b;
   return a;
}

template <int VEC>
struct Vec {
   float v[VEC];
   __device__ __forceinline__ void load(const float *p) {
      if constexpr (VEC == 4) {
         const float4 t = *reinterpret_cast<const float4 *>(p);
         v[0] = t.x;
         v[1] = t.y;
         v[2] = t.z;
         v[3] = t.w;
      } else {
#pragma unroll
         for (int i = 0; i < VEC; i++) v[i] = p[i];
      }
   }
   __device__ __forceinline__ void store(float *p) const {
      if constexpr (VEC == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
      else {
#pragma unroll
         for (int i = 0; i < VEC; i++) p[i] = v[i];
      }
   }
};

}  // namespace pvgpu
