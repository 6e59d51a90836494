// layer_update.cu -- a6..a9: GSyn accumulation, LCA membrane update and the ANN threshold.
//
// Element-wise and HBM-bound.  Every product and sum is rounded separately (__fmul_rn /
// __fadd_rn / __fdiv_rn), in the order the reference's C++ evaluates it, so the results
// equal the reference CPU path bit for bit (nvcc would otherwise contract a*b+c into an
// FMA).  The per-batch decay factor e = (float)exp(-dt/tau) is computed once per batch
// element per block in double, as HyPerLCAInternalStateBuffer.kpp:50 does per neuron.
//
// One kernel walks the layer for every update (rows_kernel): units of four values of a row where
// the rows allow it, two units per thread with all their loads issued before the first result is
// stored, and two multiplications per unit to locate it (row_map.cuh).  32 x 16x16x512: an LCA update
// and a threshold 13 us together, against 35 + 33 us with one value per load and four 64-bit
// divisions for each.
#include "row_map.cuh"

#include <cfloat>

namespace {

using pvgpu::Loc;

constexpr int kThreads = 256;
constexpr int kItems = 4;  // neurons per thread of the blocks that blocks_fit_batch's limit refers to
constexpr int kUnits = 2;  // units per thread and round

struct Thresh {
   float VThresh, AMin, AMax, AShift, VWidth;
};

// HyPerActivityBuffer::updateBufferCPU then ANNActivityBuffer::applyVThresh / applyAMax
// (components/ANNActivityBuffer.cpp:490-558), on one neuron.
__device__ __forceinline__ float ann_threshold(float v, const Thresh &t) {
   float a = v;
   if (t.VThresh > -FLT_MAX) {
      float vtw = __fadd_rn(t.VThresh, t.VWidth);
      if (v < t.VThresh) {
         a = t.AMin;
      } else if (v < vtw) {
         float c = __fadd_rn(__fadd_rn(vtw, -t.AShift), -t.AMin);
         a = __fadd_rn(t.AMin, __fdiv_rn(__fmul_rn(c, __fadd_rn(v, -t.VThresh)), t.VWidth));
      } else {
         a = __fadd_rn(a, -t.AShift);
      }
   }
   if (t.AMax < FLT_MAX && a > t.AMax) a = t.AMax;
   return a;
}

// HyPerLCAInternalStateBuffer.kpp:52-61
__device__ __forceinline__ float lca_step(float v, float g, float a, float e, float si) {
   return __fadd_rn(__fmul_rn(e, v), __fmul_rn(__fadd_rn(1.0f, -e), __fadd_rn(g, __fmul_rn(si, a))));
}

using pvgpu::row_at;
using pvgpu::row_map;
using pvgpu::row_vec;
using pvgpu::RowAt;
using pvgpu::RowMap;
using pvgpu::Vec;

// Batch elements that a block's kUnits * kThreads * 4 neurons can touch: a layer has at least
// kThreads * kItems / (kMaxB - 1) neurons (blocks_fit_batch).
constexpr int kMaxB = 8;
constexpr int kBlockB = 2 * kMaxB;

// One pass over a layer: F loads a unit's operands, then computes and stores.  With F::kDecay a block
// owns consecutive units, so that it needs the decay factors of few batch elements.
template <int VEC, bool WIDE, typename F>
__global__ void __launch_bounds__(kThreads) rows_kernel(RowMap m, F f) {
   __shared__ float eS[kBlockB];
   const int64_t first = (int64_t)blockIdx.x * kThreads * kUnits;
   typename F::template Regs<VEC> r[kUnits];
   RowAt at[kUnits];
#pragma unroll
   for (int i = 0; i < kUnits; i++) {
      const int64_t u = first + i * kThreads + threadIdx.x;
      if (u < m.units) {
         at[i] = row_at<VEC, WIDE>(m, u);
         f.template load<VEC>(r[i], at[i]);
      }
   }
   int b0 = 0;
   if constexpr (F::kDecay) {
      b0 = row_at<VEC, WIDE>(m, first).b;
      if (threadIdx.x < kBlockB && b0 + (int)threadIdx.x < f.nb)
         eS[threadIdx.x] = (float)exp(-f.dtAdapt[b0 + threadIdx.x] / (double)f.tau);
      __syncthreads();
   }
#pragma unroll
   for (int i = 0; i < kUnits; i++)
      if (first + i * kThreads + threadIdx.x < m.units)
         f.template finish<VEC>(r[i], at[i], F::kDecay ? eS[at[i].b - b0] : 0.0f);
}

template <typename F>
pvgpu_status run_rows(const Loc &l, const F &f, uintptr_t all, cudaStream_t s, const char *where) {
   int vec = row_vec(l, all);
   if (l.numRes() * l.nb / vec > 0x7fffffffLL) vec = 1;
   const RowMap m = row_map(l, vec);
   const int64_t blocks = (m.units + kThreads * kUnits - 1) / (kThreads * kUnits);
   if (blocks > 0x7fffffff) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   if (vec == 4) rows_kernel<4, false><<<(unsigned)blocks, kThreads, 0, s>>>(m, f);
   else if (m.units <= 0x7fffffffLL) rows_kernel<1, false><<<(unsigned)blocks, kThreads, 0, s>>>(m, f);
   else rows_kernel<1, true><<<(unsigned)blocks, kThreads, 0, s>>>(m, f);
   PVGPU_CHECK_LAUNCH(where);
   return PVGPU_OK;
}

uintptr_t bits(const void *p) { return reinterpret_cast<uintptr_t>(p); }

template <int VEC>
__global__ void __launch_bounds__(kThreads) accumulate_kernel(int64_t units, int64_t n, int nch, float c0, float c1,
                                                              float c2, float c3, const float *__restrict__ gsyn,
                                                              float *__restrict__ g) {
   const float cs[4] = {c0, c1, c2, c3};
   for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += (int64_t)gridDim.x * blockDim.x) {
      Vec<VEC> x[4], out;
#pragma unroll
      for (int ch = 0; ch < 4; ch++)
         if (ch < nch) x[ch].load(gsyn + (size_t)ch * n + u * VEC);
#pragma unroll
      for (int i = 0; i < VEC; i++) {
         float value = 0.0f;
#pragma unroll
         for (int ch = 0; ch < 4; ch++)
            if (ch < nch) value = __fadd_rn(value, __fmul_rn(cs[ch], x[ch].v[i]));
         out.v[i] = value;
      }
      out.store(g + u * VEC);
   }
}

struct LcaUpdate {
   static constexpr bool kDecay = true;
   int nb;
   float si, tau;
   const double *__restrict__ dtAdapt;
   const float *__restrict__ g;
   const float *__restrict__ aExt;
   float *__restrict__ v;
   template <int VEC>
   struct Regs {
      Vec<VEC> v, g, a;
   };
   template <int VEC>
   __device__ __forceinline__ void load(Regs<VEC> &r, const RowAt &at) const {
      r.a.load(aExt + at.ext);
      r.g.load(g + at.res);
      r.v.load(v + at.res);
   }
   template <int VEC>
   __device__ __forceinline__ void finish(Regs<VEC> &r, const RowAt &at, float e) const {
#pragma unroll
      for (int i = 0; i < VEC; i++) r.v.v[i] = lca_step(r.v.v[i], r.g.v[i], r.a.v[i], e, si);
      r.v.store(v + at.res);
   }
};

// MomentumLCAInternalStateBuffer.kpp:51-66, rounded as the reference's C++ evaluates it:
// drive = (1 - e)(G + si A); V = (e V + drive) + rate * prevDrive; prevDrive = drive.
struct MomentumUpdate {
   static constexpr bool kDecay = true;
   int nb;
   float si, rate, tau;
   const double *__restrict__ dtAdapt;
   const float *__restrict__ g;
   const float *__restrict__ aExt;
   float *__restrict__ prevDrive;
   float *__restrict__ v;
   template <int VEC>
   struct Regs {
      Vec<VEC> v, g, a, d;
   };
   template <int VEC>
   __device__ __forceinline__ void load(Regs<VEC> &r, const RowAt &at) const {
      r.a.load(aExt + at.ext);
      r.g.load(g + at.res);
      r.v.load(v + at.res);
      r.d.load(prevDrive + at.res);
   }
   template <int VEC>
   __device__ __forceinline__ void finish(Regs<VEC> &r, const RowAt &at, float e) const {
#pragma unroll
      for (int i = 0; i < VEC; i++) {
         const float drive = __fmul_rn(__fadd_rn(1.0f, -e), __fadd_rn(r.g.v[i], __fmul_rn(si, r.a.v[i])));
         r.v.v[i] = __fadd_rn(__fadd_rn(__fmul_rn(e, r.v.v[i]), drive), __fmul_rn(rate, r.d.v[i]));
         r.d.v[i] = drive;
      }
      r.v.store(v + at.res);
      r.d.store(prevDrive + at.res);
   }
};

// ISTAInternalStateBuffer.kpp:46-60: V += ((float)dt / tau)(G - VThresh sign(A)).
struct IstaUpdate {
   static constexpr bool kDecay = false;
   float VThresh, tau;
   const double *__restrict__ dtAdapt;
   const float *__restrict__ g;
   const float *__restrict__ aExt;
   float *__restrict__ v;
   template <int VEC>
   struct Regs {
      Vec<VEC> v, g, a;
      float q;
   };
   template <int VEC>
   __device__ __forceinline__ void load(Regs<VEC> &r, const RowAt &at) const {
      r.a.load(aExt + at.ext);
      r.g.load(g + at.res);
      r.v.load(v + at.res);
      r.q = __fdiv_rn((float)dtAdapt[at.b], tau);
   }
   template <int VEC>
   __device__ __forceinline__ void finish(Regs<VEC> &r, const RowAt &at, float) const {
#pragma unroll
      for (int i = 0; i < VEC; i++) {
         const float a = r.a.v[i];
         float sign = 0.0f;
         if (a != 0.0f) sign = __fdiv_rn(a, fabsf(a));
         r.v.v[i] = __fadd_rn(r.v.v[i], __fmul_rn(r.q, __fadd_rn(r.g.v[i], -__fmul_rn(VThresh, sign))));
      }
      r.v.store(v + at.res);
   }
};

struct AnnThreshold {
   static constexpr bool kDecay = false;
   Thresh t;
   const float *__restrict__ v;
   float *__restrict__ aExt;
   template <int VEC>
   struct Regs {
      Vec<VEC> v;
   };
   template <int VEC>
   __device__ __forceinline__ void load(Regs<VEC> &r, const RowAt &at) const {
      r.v.load(v + at.res);
   }
   template <int VEC>
   __device__ __forceinline__ void finish(Regs<VEC> &r, const RowAt &at, float) const {
#pragma unroll
      for (int i = 0; i < VEC; i++) r.v.v[i] = ann_threshold(r.v.v[i], t);
      r.v.store(aExt + at.ext);
   }
};

// The piecewise-linear transfer function given by vertices (ANNActivityBuffer::setVertices /
// applyVerticesANNActivityBufferOnGPU, components/ANNActivityBuffer.kpp:16-77): below the first
// vertex and from the last one on, the outer slopes; between vertices v and v + 1 the slope
// slopes[v + 1]; a potential equal to a vertex takes the vertex's activity, the last of equal
// vertices winning (jumps are continuous from the right).  Products and sums are rounded
// separately, as the CPU form of the same function.
struct AnnVertices {
   static constexpr bool kDecay = false;
   int nv;
   const float *__restrict__ vV;
   const float *__restrict__ vA;
   const float *__restrict__ slopes;
   const float *__restrict__ v;
   float *__restrict__ aExt;
   template <int VEC>
   struct Regs {
      Vec<VEC> v;
   };
   template <int VEC>
   __device__ __forceinline__ void load(Regs<VEC> &r, const RowAt &at) const {
      r.v.load(v + at.res);
   }
   __device__ __forceinline__ float transfer(float x) const {
      const int last = nv - 1;
      if (x < vV[0]) return __fadd_rn(vA[0], __fmul_rn(slopes[0], __fsub_rn(x, vV[0])));
      if (x >= vV[last]) return __fadd_rn(vA[last], __fmul_rn(slopes[nv], __fsub_rn(x, vV[last])));
      float a = 0.0f;
      for (int j = 0; j < last && x >= vV[j]; j++) {
         if (x == vV[j]) a = vA[j];
         else if (x < vV[j + 1]) a = __fadd_rn(vA[j], __fmul_rn(slopes[j + 1], __fsub_rn(x, vV[j])));
      }
      return a;
   }
   template <int VEC>
   __device__ __forceinline__ void finish(Regs<VEC> &r, const RowAt &at, float) const {
#pragma unroll
      for (int i = 0; i < VEC; i++) r.v.v[i] = transfer(r.v.v[i]);
      r.v.store(aExt + at.ext);
   }
};

// GSynAccumulator -> HyPerLCAInternalStateBuffer -> ANNActivityBuffer in one pass.
struct LcaLayer {
   static constexpr bool kDecay = true;
   int nb, nch;
   float cs[4];
   float si, tau;
   Thresh t;
   int64_t total;
   const float *__restrict__ gsyn;
   const double *__restrict__ dtAdapt;
   float *__restrict__ v;
   float *__restrict__ aExt;
   template <int VEC>
   struct Regs {
      Vec<VEC> v, a, g[4];
   };
   template <int VEC>
   __device__ __forceinline__ void load(Regs<VEC> &r, const RowAt &at) const {
#pragma unroll
      for (int ch = 0; ch < 4; ch++)
         if (ch < nch) r.g[ch].load(gsyn + (size_t)ch * total + at.res);
      r.v.load(v + at.res);
      r.a.load(aExt + at.ext);
   }
   template <int VEC>
   __device__ __forceinline__ void finish(Regs<VEC> &r, const RowAt &at, float e) const {
#pragma unroll
      for (int i = 0; i < VEC; i++) {
         float gv = 0.0f;
#pragma unroll
         for (int ch = 0; ch < 4; ch++)
            if (ch < nch) gv = __fadd_rn(gv, __fmul_rn(cs[ch], r.g[ch].v[i]));
         r.v.v[i] = lca_step(r.v.v[i], gv, r.a.v[i], e, si);
         r.a.v[i] = ann_threshold(r.v.v[i], t);
      }
      r.v.store(v + at.res);
      r.a.store(aExt + at.ext);
   }
};

bool blocks_fit_batch(const Loc &loc) {
   // a block spans kThreads*kItems neurons: it must not touch more than kMaxB batch elements
   int64_t span = (int64_t)kThreads * kItems;
   return loc.numRes() * (kMaxB - 1) >= span;
}

}  // namespace

extern "C" pvgpu_status pvgpu_gsyn_accumulate(int64_t n, int numChannels, const float *coeffs, const float *gsyn,
                                              float *g, void *stream) {
   if (n <= 0 || numChannels < 0 || numChannels > 4 || (numChannels > 0 && (!coeffs || !gsyn)) || !g)
      return PVGPU_ERR_BAD_ARG;
   float c[4] = {0, 0, 0, 0};
   for (int i = 0; i < numChannels; i++) c[i] = coeffs[i];
   // channels lie n values apart, so n decides whether all of them start on 16 bytes
   const int vec = n % 4 == 0 && (bits(gsyn) | bits(g)) % 16 == 0 ? 4 : 1;
   const int64_t units = n / vec;
   int64_t blocks = (units + kThreads - 1) / kThreads;
   if (blocks > 152 * 64) blocks = 152 * 64;
   auto kernel = vec == 4 ? accumulate_kernel<4> : accumulate_kernel<1>;
   kernel<<<(unsigned)blocks, kThreads, 0, pvgpu::as_stream(stream)>>>(units, n, numChannels, c[0], c[1], c[2], c[3],
                                                                      gsyn, g);
   PVGPU_CHECK_LAUNCH("gsyn_accumulate");
   return PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_lca_update(const pvgpu_loc *loc, int selfInteract, const double *dtAdapt, float tau,
                                         const float *g, const float *aExt, float *v, void *stream) {
   if (!loc || !pvgpu::loc_valid(*loc) || !dtAdapt || !g || !aExt || !v) return PVGPU_ERR_BAD_ARG;
   Loc l = pvgpu::to_loc(*loc);
   if (!blocks_fit_batch(l)) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   const LcaUpdate f = {l.nb, selfInteract ? 1.0f : 0.0f, tau, dtAdapt, g, aExt, v};
   return run_rows(l, f, bits(g) | bits(aExt) | bits(v), pvgpu::as_stream(stream), "lca_update");
}

extern "C" pvgpu_status pvgpu_momentum_lca_update(const pvgpu_loc *loc, int selfInteract, float momentumRate,
                                                  const double *dtAdapt, float tau, const float *g, const float *aExt,
                                                  float *prevDrive, float *v, void *stream) {
   if (!loc || !pvgpu::loc_valid(*loc) || !dtAdapt || !g || !aExt || !prevDrive || !v) return PVGPU_ERR_BAD_ARG;
   Loc l = pvgpu::to_loc(*loc);
   if (!blocks_fit_batch(l)) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   const MomentumUpdate f = {l.nb, selfInteract ? 1.0f : 0.0f, momentumRate, tau, dtAdapt, g, aExt, prevDrive, v};
   return run_rows(l, f, bits(g) | bits(aExt) | bits(prevDrive) | bits(v), pvgpu::as_stream(stream),
                   "momentum_lca_update");
}

extern "C" pvgpu_status pvgpu_ista_update(const pvgpu_loc *loc, float VThresh, const double *dtAdapt, float tau,
                                          const float *g, const float *aExt, float *v, void *stream) {
   if (!loc || !pvgpu::loc_valid(*loc) || !dtAdapt || !g || !aExt || !v) return PVGPU_ERR_BAD_ARG;
   Loc l = pvgpu::to_loc(*loc);
   const IstaUpdate f = {VThresh, tau, dtAdapt, g, aExt, v};
   return run_rows(l, f, bits(g) | bits(aExt) | bits(v), pvgpu::as_stream(stream), "ista_update");
}

extern "C" pvgpu_status pvgpu_ann_activity(const pvgpu_loc *loc, const float *v, float VThresh, float AMin, float AMax,
                                           float AShift, float VWidth, float *aExt, void *stream) {
   if (!loc || !pvgpu::loc_valid(*loc) || !v || !aExt) return PVGPU_ERR_BAD_ARG;
   if (VWidth < 0) {  // ANNActivityBuffer::setVertices reinterprets a negative width
      VThresh += VWidth;
      VWidth = -VWidth;
   }
   Loc l = pvgpu::to_loc(*loc);
   const AnnThreshold f = {Thresh{VThresh, AMin, AMax, AShift, VWidth}, v, aExt};
   return run_rows(l, f, bits(v) | bits(aExt), pvgpu::as_stream(stream), "ann_activity");
}

extern "C" pvgpu_status pvgpu_ann_vertices(const pvgpu_loc *loc, int numVertices, const float *verticesV,
                                           const float *verticesA, const float *slopes, const float *v, float *aExt,
                                           void *stream) {
   if (!loc || !pvgpu::loc_valid(*loc) || numVertices < 1 || !verticesV || !verticesA || !slopes || !v || !aExt)
      return PVGPU_ERR_BAD_ARG;
   Loc l = pvgpu::to_loc(*loc);
   const AnnVertices f = {numVertices, verticesV, verticesA, slopes, v, aExt};
   return run_rows(l, f, bits(v) | bits(aExt), pvgpu::as_stream(stream), "ann_vertices");
}

extern "C" pvgpu_status pvgpu_lca_layer_update(const pvgpu_lca_layer_desc *d, const float *gsyn,
                                               const double *dtAdapt, float *v, float *aExt, void *stream) {
   if (!d || !pvgpu::loc_valid(d->loc) || !dtAdapt || !v || !aExt) return PVGPU_ERR_BAD_ARG;
   if (d->numChannels < 0 || d->numChannels > 4 || (d->numChannels > 0 && !gsyn)) return PVGPU_ERR_BAD_ARG;
   Loc l = pvgpu::to_loc(d->loc);
   if (!blocks_fit_batch(l)) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   float vt = d->VThresh, vw = d->VWidth;
   if (vw < 0) {
      vt += vw;
      vw = -vw;
   }
   const LcaLayer f = {l.nb,
                       d->numChannels,
                       {d->coeffs[0], d->coeffs[1], d->coeffs[2], d->coeffs[3]},
                       d->selfInteract ? 1.0f : 0.0f,
                       d->tau,
                       Thresh{vt, d->AMin, d->AMax, d->AShift, vw},
                       l.numRes() * l.nb,
                       gsyn,
                       dtAdapt,
                       v,
                       aExt};
   // channels lie total values apart; total is a multiple of four where whole rows are
   return run_rows(l, f, bits(gsyn) | bits(v) | bits(aExt), pvgpu::as_stream(stream), "lca_layer_update");
}
