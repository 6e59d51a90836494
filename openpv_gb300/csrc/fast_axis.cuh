// fast_axis.cuh -- one axis of a connection's geometry without divisions.
#pragma once

#include "pvgpu_internal.cuh"

namespace pvgpu {

// Axis::start as shifts: every legal ratio of layer sizes is a power of two (axis_legal), so
// start(i) = (((i - c) << tl) >> sr) + o, the arithmetic shift being the floor of the many-to-one
// case.  first_ge is its inverse in closed form (a binary search over start() cost each thread
// about 2,000 cycles before the first entry was read).
struct FastAxis {
   int c, tl, sr, o, n;
   __host__ __device__ __forceinline__ int start(int i) const { return (((i - c) << tl) >> sr) + o; }
   // first i in [0, n] with start(i) >= v
   __host__ __device__ __forceinline__ int first_ge(int v) const {
      const int i = c + ((((v - o) << sr) + (1 << tl) - 1) >> tl);
      return i < 0 ? 0 : (i > n ? n : i);
   }
};

inline FastAxis fast_axis(const Axis &a, int nExt) {
   auto log2i = [](int n) {
      int s = 0;
      while ((1 << s) < n) s++;
      return s;
   };
   if (a.nPre == a.nPost) return FastAxis{a.preBorder + (a.patch - 1) / 2, 0, 0, 0, nExt};
   if (a.nPre < a.nPost) {
      const int t = a.nPost / a.nPre;
      return FastAxis{a.preBorder, log2i(t), 0, -((a.patch - t) / 2), nExt};
   }
   const int s = a.nPre / a.nPost;
   return FastAxis{a.preBorder + (s / 2) * (a.patch - 1), 0, log2i(s), 0, nExt};
}

}  // namespace pvgpu
