// deliver_pre_fast.cu -- a4 in FAST mode (FP32 fused multiply-add, tiled order): presynaptic
// delivery without atomics for every geometry, by two kernels.
//
//   deliver_pre_cols_kernel     wide post layers: the lanes of a warp are post features, a warp owns
//                               one post column and keeps a sliding window of rows in registers;
//   deliver_pre_scatter_kernel  narrow post layers: the lanes of a warp are the weights of one
//                               entry's patch, accumulated into the warp's own copy of an output tile
//                               in shared memory; the copies are summed in warp order.
//
// Both are deterministic: every output's additions happen in an order that the inputs and the
// launch shape fix.
#include "deliver_pre.cuh"
#include "fast_axis.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace {

namespace cg = cooperative_groups;

using pvgpu::fast_axis;
using pvgpu::FastAxis;
using pvgpu::num_sms;
using pvgpu::PreGeom;

struct FastGeom {
   FastAxis ax, ay;
   int nxExt, nf, rowElems;       // presynaptic row: nxExt * nf values
   int64_t preNumExt, postNumRes;
   int preLt, preUp;
   int postNx, postNy;
   int nxp, nyp, nfp, nkx, nky, patchSize;
   float dtf;
};

FastGeom fast_geom(const PreGeom &g) {
   FastGeom q;
   q.ax = fast_axis(g.ax, g.pre.nxExt());
   q.ay = fast_axis(g.ay, g.pre.nyExt());
   q.nxExt = g.pre.nxExt();
   q.nf = g.pre.nf;
   q.rowElems = q.nxExt * q.nf;
   q.preNumExt = g.pre.numExt();
   q.postNumRes = g.post.numRes();
   q.preLt = g.pre.lt;
   q.preUp = g.pre.up;
   q.postNx = g.post.nx;
   q.postNy = g.post.ny;
   q.nxp = g.nxp;
   q.nyp = g.nyp;
   q.nfp = g.nfp;
   q.nkx = g.nkx;
   q.nky = g.nky;
   q.patchSize = g.patchSize;
   q.dtf = g.dtf;
   return q;
}

// Weights::calcDataIndexFromPatchIndex (components/Weights.cpp:208-232); nkx, nky powers of two
__device__ __forceinline__ int kernel_index(const FastGeom &g, int xe, int ye, int f) {
   const int x = (xe - g.preLt) & (g.nkx - 1), y = (ye - g.preUp) & (g.nky - 1);
   return (y * g.nkx + x) * g.nf + f;
}

// lower_bound of `keys` extended indices in the ascending list e[0, n), eight lanes to a key: each
// round cuts the range to an eighth, so a list of 40,000 entries takes five dependent loads instead
// of sixteen; and each group of lanes searches for four keys at once, so that those loads overlap (one
// key at a time cost a CTA that visits 36 rows 15 round trips to L2).  put(t, position) is called by one
// lane for each key t.
template <typename Key, typename Put>
__device__ __forceinline__ void search_keys(const pvgpu_entry *e, int n, int keys, Key key, Put put) {
   constexpr int KP = 4;
   const int lane = threadIdx.x & 31, l = lane & 7, groups = blockDim.x >> 3;
   const unsigned gmask = 0xffu << (lane & 24);
   for (int t0 = 0; t0 < keys; t0 += groups * KP) {
      int64_t k[KP];
      int lo[KP], hi[KP];
#pragma unroll
      for (int i = 0; i < KP; i++) {
         const int t = t0 + i * groups + (threadIdx.x >> 3);
         k[i] = t < keys ? key(t) : 0;
         lo[i] = 0;
         hi[i] = t < keys ? n : 0;
      }
      for (;;) {
         bool open = false;
         uint32_t at[KP];
#pragma unroll
         for (int i = 0; i < KP; i++) {
            const int q = (hi[i] - lo[i] + 7) >> 3, p = lo[i] + q * (l + 1) - 1;
            open = open || lo[i] < hi[i];
            at[i] = lo[i] < hi[i] && p < hi[i] ? e[p].index : 0xffffffffu;
         }
         if (!__any_sync(0xffffffffu, open)) break;
#pragma unroll
         for (int i = 0; i < KP; i++) {
            const int q = (hi[i] - lo[i] + 7) >> 3, p = lo[i] + q * (l + 1) - 1;
            const bool less = lo[i] < hi[i] && p < hi[i] && (int64_t)at[i] < k[i];
            const int cnt = __popc(__ballot_sync(0xffffffffu, less) & gmask);
            if (lo[i] < hi[i]) {
               hi[i] = min(hi[i], lo[i] + q * (cnt + 1) - 1);
               lo[i] += q * cnt;
            }
         }
      }
#pragma unroll
      for (int i = 0; i < KP; i++) {
         const int t = t0 + i * groups + (threadIdx.x >> 3);
         if (t < keys && l == 0) put(t, lo[i]);
      }
   }
}

// -------------------------------------------------------------------------------------------
// Wide post layers.
//
// A CTA owns 8 post columns (one per warp) x RS post rows x 32 * FPL features (FPL consecutive ones
// per lane).  It walks the presynaptic extended rows that reach its rows in ascending order -- the
// SparseList order -- and each warp keeps one register accumulator per patch row in a sliding
// window: while presynaptic row ye is processed, acc[ky] holds post row start(ye) + ky, so patch row
// ky of an entry always adds into acc[ky] (a static index).  Rows that no later presynaptic row
// reaches are added into GSyn once (no atomics) and the window shifts (register moves, so that the
// row loop need not be unrolled: an unrolled loop outgrew the instruction cache at 11 patch rows).
// Each entry is read and decoded once per warp and feeds nyp x FPL multiply-adds per lane.
//
// What bounds it: the weight stream.  Every (entry, weight) product is distinct, so each FMA takes
// its own 4 bytes from L2: 8.2 GB at 17.4 TB/s, 71 % of L2's rate, on the delivery microbenchmark at
// 1 % activity (0.469 ms; 0.522 ms with a test per patch row, which ran 2.7 times the instructions
// and left the issue slots the limit).  A patch is therefore
// added whole, also where some of its rows lie outside [P0, P1) (they are dropped when the window
// moves past them): tests per patch row cost more than the (nyp - 1) / RS extra products.
// -------------------------------------------------------------------------------------------
constexpr int kCols = 8;
constexpr int kRowsMax = 256;  // presynaptic rows a CTA may visit

template <int FPL>
struct VecF;
template <>
struct VecF<1> {
   __device__ static void ld(const float *p, float *v) { v[0] = __ldg(p); }
   __device__ static void rmw(float *p, const float *v) { p[0] += v[0]; }
};
template <>
struct VecF<2> {
   __device__ static void ld(const float *p, float *v) {
      const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
      v[0] = t.x;
      v[1] = t.y;
   }
   __device__ static void rmw(float *p, const float *v) {
      float2 t = *reinterpret_cast<float2 *>(p);
      t.x += v[0];
      t.y += v[1];
      *reinterpret_cast<float2 *>(p) = t;
   }
};
template <>
struct VecF<4> {
   __device__ static void ld(const float *p, float *v) {
      const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
      v[0] = t.x;
      v[1] = t.y;
      v[2] = t.z;
      v[3] = t.w;
   }
   __device__ static void rmw(float *p, const float *v) {
      float4 t = *reinterpret_cast<float4 *>(p);
      t.x += v[0];
      t.y += v[1];
      t.z += v[2];
      t.w += v[3];
      *reinterpret_cast<float4 *>(p) = t;
   }
};

// acc[q] += a * w[q] for the lane's FPL features: pairs of features by the packed FP32 FMA (one
// instruction, each element rounded once, as fmaf), a single feature by fmaf
template <int FPL>
__device__ __forceinline__ void fma_row(float *acc, float a, const float *w) {
   if constexpr (FPL % 2 == 0) {
      const float2 a2 = make_float2(a, a);
#pragma unroll
      for (int q = 0; q < FPL; q += 2) {
         const float2 r = __ffma2_rn(a2, make_float2(w[q], w[q + 1]), make_float2(acc[q], acc[q + 1]));
         acc[q] = r.x;
         acc[q + 1] = r.y;
      }
   } else {
#pragma unroll
      for (int q = 0; q < FPL; q++) acc[q] = fmaf(a, w[q], acc[q]);
   }
}

// More than 16 accumulators per lane (NYP x FPL) do not fit the 64 registers of four CTAs per SM
// next to the entry pipeline; those instantiations take two CTAs per SM (128 registers) instead.
template <int FPL, int NYP, bool SPARSE>
__global__ void __launch_bounds__(kCols * 32, (FPL * NYP > 16) ? 2 : 4)
      deliver_pre_cols_kernel(FastGeom g, int RS, const pvgpu_entry *__restrict__ entries,
                              const int64_t *__restrict__ numActive, const float *__restrict__ aExt,
                              const float *__restrict__ W, float *__restrict__ gsyn) {
   __shared__ int rowLo[kRowsMax], rowHi[kRowsMax];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int nColT = (g.postNx + kCols - 1) / kCols;
   const int X0 = (blockIdx.x % nColT) * kCols, X = X0 + warp;
   const int fo0 = (blockIdx.x / nColT) * 32 * FPL + lane * FPL;
   const int P0 = blockIdx.y * RS, P1 = min(P0 + RS, g.postNy);
   const int b = blockIdx.z;
   // presynaptic rows reaching post rows [P0, P1) and the columns reaching [X0, X0 + 8)
   const int yeLo = g.ay.first_ge(P0 - g.nyp + 1), yeEnd = g.ay.first_ge(P1);
   const int xlo = g.ax.first_ge(X0 - g.nxp + 1), xEnd = g.ax.first_ge(min(X0 + kCols, g.postNx));
   const int nRows = yeEnd - yeLo;
   if (nRows <= 0 || xlo >= xEnd) return;  // CTA-uniform
   const pvgpu_entry *eb = SPARSE ? entries + (size_t)b * g.preNumExt : nullptr;
   if (SPARSE) {
      const int nAct = (int)min(max(numActive[b], (int64_t)0), g.preNumExt);
      search_keys(
            eb, nAct, 2 * nRows,
            [&](int t) { return (int64_t)(yeLo + (t >> 1)) * g.rowElems + ((t & 1) ? xEnd : xlo) * g.nf; },
            [&](int t, int v) { ((t & 1) ? rowHi : rowLo)[t >> 1] = v; });
      __syncthreads();
   }
   if (X >= g.postNx) return;  // no barrier below

   const float *ab = SPARSE ? nullptr : aExt + (size_t)b * g.preNumExt;
   const bool on = fo0 < g.nfp;  // a slab's last lanes have no feature
   const float *Wl = W + (on ? fo0 : 0);
   const int rowStrideW = g.nxp * g.nfp;
   float *gcol = gsyn + (size_t)b * g.postNumRes + (size_t)X * g.nfp + fo0;
   const size_t gRow = (size_t)g.postNx * g.nfp;

   float acc[NYP][FPL];
#pragma unroll
   for (int s = 0; s < NYP; s++)
#pragma unroll
      for (int q = 0; q < FPL; q++) acc[s][q] = 0.0f;
   int py = g.ay.start(yeLo);  // the post row of acc[0]
   auto shift = [&]() {
      if (py >= P0 && py < P1 && on) VecF<FPL>::rmw(gcol + (size_t)py * gRow, acc[0]);
#pragma unroll
      for (int j = 0; j + 1 < NYP; j++)
#pragma unroll
         for (int q = 0; q < FPL; q++) acc[j][q] = acc[j + 1][q];
#pragma unroll
      for (int q = 0; q < FPL; q++) acc[NYP - 1][q] = 0.0f;
      py++;
   };

   for (int ye = yeLo; ye < yeEnd; ye++) {
      const int start = g.ay.start(ye);
      while (py < start) shift();
      const int lo = SPARSE ? rowLo[ye - yeLo] : xlo * g.nf, hi = SPARSE ? rowHi[ye - yeLo] : xEnd * g.nf;
      const uint32_t kRow = (uint32_t)ye * (uint32_t)g.rowElems;
      for (int base = lo; base < hi; base += 32) {
         int kr = 0;
         float a = 0.0f;
         if (base + lane < hi) {
            if (SPARSE) {
               const pvgpu_entry en = eb[base + lane];
               kr = (int)(en.index - kRow);
               a = en.value;
            } else {
               kr = base + lane;
               a = ab[kRow + (uint32_t)kr];
            }
         }
         const int xe = (int)((uint32_t)kr / (uint32_t)g.nf), f = kr - xe * g.nf;
         const int kx = X - g.ax.start(xe);
         unsigned m = __ballot_sync(0xffffffffu, a != 0.0f && kx >= 0 && kx < g.nxp);
         const int woffMine = kernel_index(g, xe, ye, f) * g.patchSize + kx * g.nfp;
         a *= g.dtf;
         // two entries per round: their weight loads are all in flight before the FMAs
         while (m & (m - 1)) {
            const int j1 = __ffs(m) - 1;
            m &= m - 1;
            const int j2 = __ffs(m) - 1;
            m &= m - 1;
            const float a1 = __shfl_sync(0xffffffffu, a, j1), a2 = __shfl_sync(0xffffffffu, a, j2);
            const float *wp1 = Wl + __shfl_sync(0xffffffffu, woffMine, j1);
            const float *wp2 = Wl + __shfl_sync(0xffffffffu, woffMine, j2);
            float w1[NYP][FPL], w2[NYP][FPL];
#pragma unroll
            for (int ky = 0; ky < NYP; ky++) {
               VecF<FPL>::ld(wp1 + ky * rowStrideW, w1[ky]);
               VecF<FPL>::ld(wp2 + ky * rowStrideW, w2[ky]);
            }
#pragma unroll
            for (int ky = 0; ky < NYP; ky++) {
               fma_row<FPL>(acc[ky], a1, w1[ky]);
               fma_row<FPL>(acc[ky], a2, w2[ky]);
            }
         }
         if (m) {
            const int j1 = __ffs(m) - 1;
            const float a1 = __shfl_sync(0xffffffffu, a, j1);
            const float *wp1 = Wl + __shfl_sync(0xffffffffu, woffMine, j1);
            float w1[NYP][FPL];
#pragma unroll
            for (int ky = 0; ky < NYP; ky++) VecF<FPL>::ld(wp1 + ky * rowStrideW, w1[ky]);
#pragma unroll
            for (int ky = 0; ky < NYP; ky++) fma_row<FPL>(acc[ky], a1, w1[ky]);
         }
      }
   }
   // the rows still in the window
#pragma unroll
   for (int j = 0; j < NYP; j++)
      if (py + j >= P0 && py + j < P1 && on) VecF<FPL>::rmw(gcol + (size_t)(py + j) * gRow, acc[j]);
}

template <int FPL, int NYP>
pvgpu_status launch_cols(const FastGeom &g, dim3 grid, int RS, cudaStream_t s, const pvgpu_entry *entries,
                         const int64_t *numActive, const float *aExt, const float *W, float *gsyn) {
   if (entries)
      deliver_pre_cols_kernel<FPL, NYP, true><<<grid, kCols * 32, 0, s>>>(g, RS, entries, numActive, nullptr, W, gsyn);
   else
      deliver_pre_cols_kernel<FPL, NYP, false><<<grid, kCols * 32, 0, s>>>(g, RS, nullptr, nullptr, aExt, W, gsyn);
   PVGPU_CHECK_LAUNCH("deliver_pre cols");
   return PVGPU_OK;
}

template <int FPL>
pvgpu_status launch_cols_nyp(const FastGeom &g, dim3 grid, int RS, cudaStream_t s, const pvgpu_entry *entries,
                             const int64_t *numActive, const float *aExt, const float *W, float *gsyn) {
#define PVGPU_NYP(N) \
   if (g.nyp == N) return launch_cols<FPL, N>(g, grid, RS, s, entries, numActive, aExt, W, gsyn);
   PVGPU_NYP(1)
   PVGPU_NYP(2)
   PVGPU_NYP(3)
   PVGPU_NYP(4)
   PVGPU_NYP(5)
   PVGPU_NYP(6)
   PVGPU_NYP(7)
   PVGPU_NYP(8)
   PVGPU_NYP(9)
   // taller patches keep NYP x FPL accumulators per lane: one or two features per lane only
   if constexpr (FPL <= 2) {
      PVGPU_NYP(10)
      PVGPU_NYP(11)
      PVGPU_NYP(12)
      PVGPU_NYP(13)
      PVGPU_NYP(14)
      PVGPU_NYP(15)
      PVGPU_NYP(16)
   }
#undef PVGPU_NYP
   return PVGPU_ERR_UNSUPPORTED_SHAPE;
}

// One launch of the column kernel: features per lane, slabs of 32 * fpl features, rows and CTAs per SM of a
// CTA, and its estimated cycles.
struct ColPlan {
   int fpl, slabs, RS, occ;
   double cost;
};

// Activity that the estimates of both kernels assume (the result does not depend on it).
double assumed_density(bool sparse) { return sparse ? 0.05 : 0.3; }

// g.nyp: the patch rows of the pass.  false for a shape that the kernel does not take.
bool cols_plan(const PreGeom &pg, const FastGeom &g, const float *W, const float *gsyn, bool sparse, ColPlan *p) {
   // features per lane: the fewest slabs of 32 * FPL features whose vector loads are aligned (a
   // weight row starts at a multiple of nfp floats)
   const uintptr_t al = reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(gsyn);
   const int maxFpl = g.nyp > 9 ? 2 : 4;
   int fpl = 1;
   while (fpl < maxFpl && 32 * fpl < g.nfp && g.nfp % (2 * fpl) == 0 && al % (8 * fpl) == 0) fpl *= 2;
   p->fpl = fpl;
   p->slabs = (g.nfp + 32 * fpl - 1) / (32 * fpl);
   const int64_t gx = (int64_t)((g.postNx + kCols - 1) / kCols) * p->slabs;
   // rows per CTA: a CTA also visits the nyp - 1 presynaptic rows around its own, so the cost is the
   // CTAs per SM times RS + nyp - 1, and more where an SM has too few CTAs (8 warps each) to hide
   // their loads; no more than the row table holds, which 64 rows of a layer four times as fine exceed.
   // 16 x 128x128x256 -> 64, 7x7, 1 % active: 545 / 504 / 469 / 606 us at 16 / 32 / 64 / 128 rows.
   p->occ = fpl * g.nyp > 16 ? 2 : 4;
   const int rowsPer = pg.pre.ny > pg.post.ny ? pg.pre.ny / pg.post.ny : 1;
   double best = 1e300;
   p->RS = 0;
   for (int r = 4; r <= 64 && (r + g.nyp) * rowsPer <= kRowsMax; r *= 2) {
      const double perSm = std::max(1.0, (double)gx * ((g.postNy + r - 1) / r) * pg.pre.nb / num_sms());
      const double cost = perSm * (r + g.nyp - 1) * (1.0 + 1.5 / std::min(perSm, (double)p->occ));
      if (cost < best) {
         best = cost;
         p->RS = r;
      }
   }
   if (p->RS == 0) return false;
   const int gy = (g.postNy + p->RS - 1) / p->RS;
   if (gx > 0x7fffffff || gy > 65535) return false;
   // entries of a presynaptic row that one column takes, and 32-entry chunks that its warp reads for them
   const double perCol = (double)pg.pre.nx / pg.post.nx * g.nf * assumed_density(sparse);
   const double took = g.nxp * perCol, read = (kCols + g.nxp - 1) * perCol, chunks = read / 32 + 1 - std::exp(-read);
   const double perEntry = 1 + g.nyp * (1 + std::max(1.0, fpl / 2.0));
   const double rows = (double)(std::min(p->RS, g.postNy) + g.nyp - 1) * pg.pre.ny / pg.post.ny;
   const double ctas = (double)gx * gy * pg.pre.nb;
   const double instr = rows * (33 + 22 * chunks + took * perEntry) + 64;
   const double serial = rows * (900 + 870 * chunks + took / 2 * (280 + 2 * perEntry));
   p->cost = std::max(ctas * std::min(g.postNx, kCols) * instr / (num_sms() * 0.62),
                      serial * std::max(1.0, ctas / ((double)num_sms() * p->occ)));
   return true;
}

// Patches taller than the window of 16 rows go in passes of equal heights, each a delivery of its own.
constexpr int kWindow = 16;

FastGeom cols_part(const FastGeom &g, int pass, int *ky0) {
   const int passes = (g.nyp + kWindow - 1) / kWindow;
   FastGeom q = g;
   *ky0 = (int)((int64_t)g.nyp * pass / passes);
   q.nyp = (int)((int64_t)g.nyp * (pass + 1) / passes) - *ky0;
   q.ay.o += *ky0;
   return q;
}

// The estimate of all passes; false where the kernel does not take one of them.
bool cols_cost(const PreGeom &pg, const FastGeom &g, const float *W, const float *gsyn, bool sparse, double *cost) {
   *cost = 0;
   for (int i = 0; i < (g.nyp + kWindow - 1) / kWindow; i++) {
      int ky0;
      ColPlan p;
      const FastGeom q = cols_part(g, i, &ky0);
      if (!cols_plan(pg, q, W, gsyn, sparse, &p)) return false;
      *cost += p.cost;
   }
   return true;
}

// One pass, or several that cols_cost has accepted: nothing is launched for a shape that the kernel does not take.
pvgpu_status run_cols(const PreGeom &pg, const FastGeom &g, const pvgpu_entry *entries, const int64_t *numActive,
                      const float *aExt, const float *W, float *gsyn, cudaStream_t s) {
   for (int i = 0; i < (g.nyp + kWindow - 1) / kWindow; i++) {
      int ky0;
      ColPlan p;
      const FastGeom q = cols_part(g, i, &ky0);
      if (!cols_plan(pg, q, W, gsyn, entries != nullptr, &p)) return PVGPU_ERR_UNSUPPORTED_SHAPE;
      const dim3 grid((unsigned)((g.postNx + kCols - 1) / kCols * p.slabs), (g.postNy + p.RS - 1) / p.RS, pg.pre.nb);
      const float *Wp = W + (size_t)ky0 * g.nxp * g.nfp;
      const pvgpu_status r = p.fpl == 1   ? launch_cols_nyp<1>(q, grid, p.RS, s, entries, numActive, aExt, Wp, gsyn)
                             : p.fpl == 2 ? launch_cols_nyp<2>(q, grid, p.RS, s, entries, numActive, aExt, Wp, gsyn)
                                          : launch_cols_nyp<4>(q, grid, p.RS, s, entries, numActive, aExt, Wp, gsyn);
      if (r != PVGPU_OK) return r;
   }
   return PVGPU_OK;
}

// -------------------------------------------------------------------------------------------
// Narrow post layers.
//
// A cluster of cz CTAs owns an output tile of TY x TX positions x FT features.  The entries that reach it
// (their ranges in each presynaptic row found first) are numbered through and dealt to the warps of the
// cluster in chunks of 32: the lanes decode one entry each, then the warp takes the chunk's entries one
// after the other with its lanes spread over the weights of the patch, VEC neighbouring ones each -- one
// entry's patch is contiguous in memory, so the loads are coalesced and its addresses are the entry's
// plus a constant per lane.  Products go into the warp's own copy of the tile in shared memory, which has
// a margin of the patch size on every side so that no lane tests whether its output lies inside.  The
// copies are summed in warp order, then over the cluster in rank order, into GSyn.
//
// The tile kernel this replaces gave each warp one output row and tested every entry of its range
// against every output: on the delivery of a V1 layer to an image (one to three features, 8x8
// patches) seven of eight lanes had nothing to add, and one image kept 8 CTAs busy.  Measured:
// one 16x16x64 V1 layer to 32x32x1 160 -> 9 us; 8 x 256x256x32 spikes (2 %) to 128x128x8, 3x3 at
// stride 2, 425 -> 60 us; 32 x 16x16x512 (5 %) to 32x32x3 754 -> 49 us.  What bounds it is the
// read-add-write on shared memory (one entry's adds must land before the next one's), hence vectors of
// up to four weights per lane, and tiles as large as the warps' copies allow -- a tile wastes what patches
// hang over its edge -- with the entries of one tile divided over a cluster.
// -------------------------------------------------------------------------------------------
// A plan takes at most this much shared memory.  The limit that a launch is checked against belongs to the
// kernel, and another thread may be launching it with a smaller plan, so it is always set to the bound.
constexpr size_t kScatSmem = 200 * 1024;

struct ScatPlan {
   int TX, TY, FT, NW, cz, vec;
   int nTX, nTY, nFT;
   int PW, tileFloats;   // floats per row of the padded tile; one copy (a multiple of 4)
   int padX;             // columns left of the tile: the margin, rounded so that patches start on vectors
   int rowsMax;
   size_t smem;
   double cost;
};

template <int VEC>
struct VecW {
   __device__ static __forceinline__ void ldg(const float *p, float *v) {
      if constexpr (VEC == 4) {
         const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
         v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
      } else if constexpr (VEC == 2) {
         const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
         v[0] = t.x, v[1] = t.y;
      } else v[0] = __ldg(p);
   }
   __device__ static __forceinline__ void ld(const float *p, float *v) {
      if constexpr (VEC == 4) {
         const float4 t = *reinterpret_cast<const float4 *>(p);
         v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
      } else if constexpr (VEC == 2) {
         const float2 t = *reinterpret_cast<const float2 *>(p);
         v[0] = t.x, v[1] = t.y;
      } else v[0] = *p;
   }
   __device__ static __forceinline__ void st(float *p, const float *v) {
      if constexpr (VEC == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
      else if constexpr (VEC == 2) *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
      else *p = v[0];
   }
};

// EPT vectors of the patch per lane at a time, U entries' weights in flight
template <int EPT, int U, int VEC, bool SPARSE>
__global__ void __launch_bounds__(256) deliver_pre_scatter_kernel(FastGeom g, ScatPlan pl,
                                                                  const pvgpu_entry *__restrict__ entries,
                                                                  const int64_t *__restrict__ numActive,
                                                                  const float *__restrict__ aExt,
                                                                  const float *__restrict__ W,
                                                                  float *__restrict__ gsyn) {
   extern __shared__ __align__(16) float sm[];
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NW = pl.NW;
   int4 *stage = reinterpret_cast<int4 *>(sm) + warp * 32;             // decoded entries of a chunk
   int *rowBeg = reinterpret_cast<int *>(sm) + NW * 128;               // [rowsMax]
   int *rowPre = rowBeg + pl.rowsMax;                                  // [rowsMax + 1], then padding
   float *acc0 = sm + NW * 128 + ((2 * pl.rowsMax + 1 + 3) & ~3);      // [NW][tileFloats]
   float *acc = acc0 + (size_t)warp * pl.tileFloats;

   const int rank = pl.cz > 1 ? blockIdx.x % pl.cz : 0;
   int t = blockIdx.x / pl.cz;
   const int X0 = (t % pl.nTX) * pl.TX;
   t /= pl.nTX;
   const int Y0 = (t % pl.nTY) * pl.TY, F0 = (t / pl.nTY) * pl.FT;
   const int b = blockIdx.y;
   const int tx = min(pl.TX, g.postNx - X0), ty = min(pl.TY, g.postNy - Y0), ft = min(pl.FT, g.nfp - F0);
   const int yeLo = g.ay.first_ge(Y0 - g.nyp + 1), nRows = g.ay.first_ge(Y0 + ty) - yeLo;
   const int xlo = g.ax.first_ge(X0 - g.nxp + 1), nX = g.ax.first_ge(X0 + tx) - xlo;
   if (nRows <= 0 || nX <= 0) return;  // cluster-uniform: nothing reaches the tile

   for (int i = lane; i < pl.tileFloats / 4; i += 32) reinterpret_cast<float4 *>(acc)[i] = make_float4(0, 0, 0, 0);
   const pvgpu_entry *eb = SPARSE ? entries + (size_t)b * g.preNumExt : nullptr;
   const float *ab = SPARSE ? nullptr : aExt + (size_t)b * g.preNumExt;
   if (SPARSE) {
      const int nAct = (int)min(max(numActive[b], (int64_t)0), g.preNumExt);
      search_keys(
            eb, nAct, 2 * nRows,
            [&](int k) { return (int64_t)(yeLo + (k >> 1)) * g.rowElems + (xlo + ((k & 1) ? nX : 0)) * g.nf; },
            [&](int k, int v) { ((k & 1) ? rowPre + 1 : rowBeg)[k >> 1] = v; });
      __syncthreads();
      if (warp == 0) {  // the rows' counts, summed
         int run = 0;
         for (int r0 = 0; r0 < nRows; r0 += 32) {
            const int r = r0 + lane;
            int c = r < nRows ? rowPre[1 + r] - rowBeg[r] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
               const int o = __shfl_up_sync(0xffffffffu, c, d);
               if (lane >= d) c += o;
            }
            if (r < nRows) rowPre[1 + r] = run + c;
            run += __shfl_sync(0xffffffffu, c, 31);
         }
         if (lane == 0) rowPre[0] = 0;
      }
   }
   __syncthreads();
   const int perRow = nX * g.nf;  // dense form
   const int total = SPARSE ? rowPre[nRows] : nRows * perRow;

   // this lane's patch vectors: offset in the entry's patch and in the tile
   const int L = g.nxp * ft, elems = g.nyp * L;
   int wo[EPT], so[EPT];
   bool in[EPT];
   auto offsets = [&](int e0) {
#pragma unroll
      for (int i = 0; i < EPT; i++) {
         const int e = e0 + (lane + 32 * i) * VEC;
         in[i] = e < elems;
         const int ky = e / L, r = e - ky * L, kx = r / ft, fl = r - kx * ft;
         wo[i] = in[i] ? (ky * g.nxp + kx) * g.nfp + fl : 0;
         so[i] = ky * pl.PW + kx * pl.FT + fl;
      }
   };
   offsets(0);

   for (int c0 = (rank * NW + warp) * 32; c0 < total; c0 += pl.cz * NW * 32) {
      const int i = c0 + lane;
      int4 d = make_int4(0, 0, 0, 0);
      float a = 0.0f;
      if (i < total) {
         int r, kr;
         if (SPARSE) {
            int lo = 0, hi = nRows;  // the row: largest r with rowPre[r] <= i
            while (hi - lo > 1) {
               const int mid = (lo + hi) >> 1;
               if (rowPre[mid] <= i) lo = mid;
               else hi = mid;
            }
            r = lo;
            const pvgpu_entry en = eb[rowBeg[r] + (i - rowPre[r])];
            kr = (int)(en.index - (uint32_t)(yeLo + r) * (uint32_t)g.rowElems);
            a = en.value;
         } else {
            r = i / perRow;
            kr = xlo * g.nf + (i - r * perRow);
            a = ab[(size_t)(yeLo + r) * g.rowElems + kr];
         }
         const int ye = yeLo + r, xe = (int)((uint32_t)kr / (uint32_t)g.nf), f = kr - xe * g.nf;
         d.x = kernel_index(g, xe, ye, f) * g.patchSize + F0;
         d.y = (g.ay.start(ye) - Y0 + g.nyp - 1) * pl.PW + (g.ax.start(xe) - X0 + pl.padX) * pl.FT;
         d.z = __float_as_int(a * g.dtf);
      }
      const unsigned m = __ballot_sync(0xffffffffu, a != 0.0f);
      const int cnt = __popc(m);
      if (a != 0.0f) stage[__popc(m & ((1u << lane) - 1))] = d;
      __syncwarp();
      for (int e0 = 0; e0 < elems; e0 += 32 * EPT * VEC) {
         if (elems > 32 * EPT * VEC) offsets(e0);
         int j = 0;
         auto take = [&](auto un) {
            constexpr int UN = decltype(un)::value;
            int4 q[UN];
            float w[UN][EPT][VEC];
#pragma unroll
            for (int u = 0; u < UN; u++) q[u] = stage[j + u];
#pragma unroll
            for (int u = 0; u < UN; u++)
#pragma unroll
               for (int i2 = 0; i2 < EPT; i2++)
                  if (in[i2]) VecW<VEC>::ldg(W + q[u].x + wo[i2], w[u][i2]);
#pragma unroll
            for (int u = 0; u < UN; u++) {
               const float av = __int_as_float(q[u].z);
               float *p = acc + q[u].y;
               float v[EPT][VEC];
#pragma unroll
               for (int i2 = 0; i2 < EPT; i2++)
                  if (in[i2]) VecW<VEC>::ld(p + so[i2], v[i2]);
#pragma unroll
               for (int i2 = 0; i2 < EPT; i2++)
                  if (in[i2]) {
#pragma unroll
                     for (int x = 0; x < VEC; x++) v[i2][x] = fmaf(av, w[u][i2][x], v[i2][x]);
                     VecW<VEC>::st(p + so[i2], v[i2]);
                  }
               __syncwarp();  // the next entry's lanes may add to these outputs
            }
            j += UN;
         };
         while (j + U <= cnt) take(std::integral_constant<int, U>());
         while (j < cnt) take(std::integral_constant<int, 1>());
      }
      __syncwarp();
   }
   __syncthreads();
   const int outs = ty * tx * ft;
   float *gb = gsyn + (size_t)b * g.postNumRes + F0;
   // f(output's offset in the tile, its GSyn value) for this thread's outputs of [lo, hi)
   auto outputs = [&](int lo, int hi, auto f) {
      for (int o = lo + tid; o < hi; o += NW * 32) {
         const int fl = o % ft, x = (o / ft) % tx, y = o / (ft * tx);
         f((y + g.nyp - 1) * pl.PW + (x + pl.padX) * pl.FT + fl,
           gb + ((size_t)(Y0 + y) * g.postNx + X0 + x) * g.nfp + fl);
      }
   };
   if (pl.cz == 1) {
      outputs(0, outs, [&](int at, float *gp) {
         float s = acc0[at];
         for (int w = 1; w < NW; w++) s += acc0[at + (size_t)w * pl.tileFloats];
         *gp += s;
      });
      return;
   }
   outputs(0, outs, [&](int at, float *) {
      float s = acc0[at];
      for (int w = 1; w < NW; w++) s += acc0[at + (size_t)w * pl.tileFloats];
      acc0[at] = s;
   });
   cg::cluster_group cl = cg::this_cluster();
   cl.sync();
   const int share = (outs + pl.cz - 1) / pl.cz;
   outputs(min(rank * share, outs), min((rank + 1) * share, outs), [&](int at, float *gp) {
      float s = cl.map_shared_rank(acc0, 0)[at];
      for (int c = 1; c < pl.cz; c++) s += cl.map_shared_rank(acc0, c)[at];
      *gp += s;
   });
   cl.sync();  // no CTA leaves while another reads its tile
}

// Tile shape by an estimate of the launch's time (cycles): the instructions of all CTAs over the
// chip's issue slots, or the serial time of one CTA's warps times the waves of CTAs, whichever is
// longer.  Activity is taken as 5 % (30 % for a dense layer; the result does not depend on it).
bool scatter_plan(const PreGeom &pg, const FastGeom &g, const float *W, bool sparse, ScatPlan *best) {
   const int sms = num_sms();
   best->cost = 1e300;
   const int sx = std::max(1, pg.pre.nx / pg.post.nx), tx = std::max(1, pg.post.nx / pg.pre.nx);
   const int sy = std::max(1, pg.pre.ny / pg.post.ny), ty = std::max(1, pg.post.ny / pg.pre.ny);
   // patches start at columns congruent to this modulo tx (one-to-many; else at any column)
   const int phase = ((-((g.nxp - tx) / 2)) % tx + tx) % tx;
   for (int T = 64; T >= 4; T >>= 1) {
      if (T > 4 && T >= 2 * std::max(g.postNx, g.postNy)) continue;  // the same tile as the next
      for (int nft = 1; nft <= 32; nft *= 2) {
         ScatPlan p;
         p.FT = (g.nfp + nft - 1) / nft;
         p.nFT = (g.nfp + p.FT - 1) / p.FT;
         if (nft > 1 && p.FT < 2) continue;
         p.TX = std::min(T, g.postNx);
         p.TY = std::min(T, g.postNy);
         p.nTX = (g.postNx + p.TX - 1) / p.TX;
         p.nTY = (g.postNy + p.TY - 1) / p.TY;
         // vectors: patch rows, patches and their starts in whole vectors (tiles start at multiples of tx)
         p.vec = 1;
         for (int v = 4; v >= 2 && p.vec == 1; v /= 2) {
            const bool rows = p.nFT == 1 ? g.nxp * g.nfp % v == 0 : p.FT % v == 0 && g.nfp % v == 0;
            const bool starts = (p.FT % v == 0 || (tx * p.FT % v == 0 && p.TX % tx == 0));
            if (rows && starts && g.patchSize % v == 0 && reinterpret_cast<uintptr_t>(W) % (4 * v) == 0) p.vec = v;
         }
         p.padX = g.nxp - 1;
         if (p.vec > 1 && p.FT % p.vec != 0) p.padX += (2 * tx - (p.padX + phase) % tx) % tx;
         p.PW = ((p.TX + p.padX + g.nxp - 1) * p.FT + 3) & ~3;
         // a patch's rows, of L values, in neighbouring banks: the pitch is L or -L modulo the 32 banks
         if (const int L = (g.nxp * p.FT + 3) & 31 & ~3)
            while (p.PW % 32 != L && p.PW % 32 != 32 - L) p.PW += 4;
         const int64_t tf = (int64_t)p.PW * (p.TY + 2 * (g.nyp - 1));
         if (tf > 14000) continue;
         p.tileFloats = (int)tf;
         const int covY = (p.TY + g.nyp - 1) * sy / ty + 2, covX = (p.TX + g.nxp - 1) * sx / tx + 2;
         p.rowsMax = covY + sy;
         for (p.NW = 8; p.NW >= 4; p.NW >>= 1) {
            p.smem = 4 * ((size_t)p.NW * 128 + ((2 * p.rowsMax + 4) & ~3) + (size_t)p.NW * p.tileFloats);
            if (p.smem <= kScatSmem) break;
         }
         if (p.NW < 4) continue;
         const int64_t tiles = (int64_t)p.nTX * p.nTY * p.nFT;
         const int occ = (int)std::min<size_t>(2048 / (p.NW * 32), (227 * 1024) / (p.smem + 1024));
         const int vectors = (g.nyp * g.nxp * p.FT / p.vec + 31) / 32;
         // a vector of one entry: load, read, multiply-adds, write; serially a read-add-write's latency
         const double perEntry = 18 + vectors * (4.0 + p.vec), latency = 45 + vectors * (4.0 + 2.0 * p.vec);
         const double E = (double)covX * covY * g.nf * assumed_density(sparse) + 1.0;
         const double outs = (double)p.TX * p.TY * p.FT / 32;
         for (p.cz = 1; p.cz <= 8; p.cz *= 2) {
            if (tiles * p.cz > 0x7fffffff || (p.cz > 1 && E / p.cz < 64)) break;
            const double instr = E / p.cz * perEntry + p.NW * (p.tileFloats / 128.0 + 500) + outs * (p.NW * 2 + 8 + (p.cz > 1 ? 20 : 0));
            const double n = (double)tiles * p.cz * pg.pre.nb;
            const double serial = 3000 + E / p.cz / p.NW * latency + p.tileFloats / 64.0 + outs * 4 + (p.cz > 1 ? 4000 : 0);
            const double waves = std::max(1.0, n / ((double)sms * occ));
            p.cost = std::max(n * instr / (sms * 2.5), serial * waves);
            if (p.cost < best->cost) *best = p;
         }
      }
   }
   return best->cost < 1e300;
}

template <int EPT, int U, int VEC>
pvgpu_status launch_scatter(const FastGeom &g, const ScatPlan &pl, int nb, cudaStream_t s, const pvgpu_entry *entries,
                            const int64_t *numActive, const float *aExt, const float *W, float *gsyn) {
   auto go = [&](auto kernel) -> pvgpu_status {
      if (pl.smem > 48 * 1024)
         PVGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScatSmem),
                    "deliver_pre scatter attribute");
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = pl.cz;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t c = {};
      c.gridDim = dim3((unsigned)(pl.nTX * pl.nTY * pl.nFT * pl.cz), nb);
      c.blockDim = dim3(pl.NW * 32);
      c.dynamicSmemBytes = pl.smem;
      c.stream = s;
      c.attrs = attr;
      c.numAttrs = pl.cz > 1 ? 1 : 0;
      PVGPU_CUDA(cudaLaunchKernelEx(&c, kernel, g, pl, entries, numActive, aExt, W, gsyn), "deliver_pre scatter");
      return PVGPU_OK;
   };
   return entries ? go(deliver_pre_scatter_kernel<EPT, U, VEC, true>) : go(deliver_pre_scatter_kernel<EPT, U, VEC, false>);
}

template <int VEC>
pvgpu_status scatter_vec(const FastGeom &g, const ScatPlan &pl, int nb, cudaStream_t s, const pvgpu_entry *entries,
                         const int64_t *numActive, const float *aExt, const float *W, float *gsyn) {
   // vectors per lane for the whole patch, up to four (larger patches go round in blocks); entries in
   // flight so that their weights take at most 32 registers
   const int ept = (g.nyp * g.nxp * pl.FT / VEC + 31) / 32;
   if (ept <= 1) return launch_scatter<1, 4, VEC>(g, pl, nb, s, entries, numActive, aExt, W, gsyn);
   if (ept <= 2) return launch_scatter<2, 4, VEC>(g, pl, nb, s, entries, numActive, aExt, W, gsyn);
   if (ept <= 3) return launch_scatter<3, VEC == 4 ? 2 : 4, VEC>(g, pl, nb, s, entries, numActive, aExt, W, gsyn);
   return launch_scatter<4, VEC == 4 ? 2 : 4, VEC>(g, pl, nb, s, entries, numActive, aExt, W, gsyn);
}

// The chosen plan's cycles on the scale of ColPlan::cost: as in scatter_plan, but with the decoding of a large
// patch's blocks and the latencies as 1,000 measured geometries have them.
double scatter_cost(const PreGeom &pg, const FastGeom &g, bool sparse, const ScatPlan &p) {
   const int sx = std::max(1, pg.pre.nx / pg.post.nx), sy = std::max(1, pg.pre.ny / pg.post.ny);
   const int tx = std::max(1, pg.post.nx / pg.pre.nx), ty = std::max(1, pg.post.ny / pg.pre.ny);
   const int vectors = (g.nyp * g.nxp * p.FT / p.vec + 31) / 32, ept = std::min(vectors, 4);
   const double cov = ((double)(p.TX + g.nxp - 1) * sx / tx) * ((double)(p.TY + g.nyp - 1) * sy / ty);
   const double E = cov * g.nf * assumed_density(sparse) + 1.0, warps = (double)p.cz * p.NW;
   const double chunks = std::max(E / 32, std::min(E, warps));
   const double perChunk = 2 + (vectors > ept ? (vectors + ept - 1) / ept * ept * 200.0 : 0.0);
   const double outs = (double)p.TX * p.TY * p.FT / 32;
   const double instr = E / p.cz * (28 + vectors * (13.3 + p.vec)) + chunks / p.cz * perChunk +
                        p.NW * (p.tileFloats / 128.0 + 900) + outs * (p.NW * 2 + 8 + (p.cz > 1 ? 20 : 0));
   const double serial = 4800 + std::max(1.0, E / warps) * (210 + vectors * (23.0 + 2 * p.vec)) +
                         std::max(1.0, chunks / warps) * perChunk * 6.9 + p.tileFloats / 64.0 + outs * 4 + (p.cz > 1 ? 4000 : 0);
   const double n = (double)p.nTX * p.nTY * p.nFT * p.cz * pg.pre.nb, sms = num_sms();
   const int occ = (int)std::min<size_t>(2048 / (p.NW * 32), (227 * 1024) / (p.smem + 1024));
   return std::max(n * instr / (sms * 1.46), serial * std::max(1.0, n / (sms * occ)));
}

pvgpu_status run_scatter(const PreGeom &pg, const FastGeom &g, const ScatPlan &pl, const pvgpu_entry *entries,
                         const int64_t *numActive, const float *aExt, const float *W, float *gsyn, cudaStream_t s) {
   const int nb = pg.pre.nb;
   return pl.vec == 4   ? scatter_vec<4>(g, pl, nb, s, entries, numActive, aExt, W, gsyn)
          : pl.vec == 2 ? scatter_vec<2>(g, pl, nb, s, entries, numActive, aExt, W, gsyn)
                        : scatter_vec<1>(g, pl, nb, s, entries, numActive, aExt, W, gsyn);
}

}  // namespace

// Which kernel: with 24 post features or more and a patch that fits the window, a column's lanes are at least
// three quarters full and its accumulators stay in registers.  Else the scatter kernel, whose lanes are the
// weights of a patch -- unless no plan for it exists, or the patch is so large that a tile is mostly margin (25 x
// 23 weights of 21 features on tiles of 16 x 16 x 3: every entry is added to 41 of them); then columns, where the
// scatter kernel would take 20 us and more and their estimate is 1.5 times lower.  (Both lines keep close calls
// with the scatter kernel: over 2,000 geometries with patches of up to 33 x 33 the pick is within 3 to 8 % of the
// faster of the two on average.)  12 x 122x40x40 -> 138, 23x21 patches, 0.6 % active: scatter 75 ms, the tile
// kernel 1.9, columns 0.46; 9 x 57x73x17 -> 21, 25x23: 2.4, 0.76, 0.26 ms; 2 x 11x5x206 -> 53, 9x19: 51, 623,
// 102 us.
pvgpu_status pvgpu::deliver_pre_fast(const PreGeom &pg, const pvgpu_entry *entries, const int64_t *numActive,
                                     const float *aExt, const float *W, float *gsyn, cudaStream_t s) {
   // 32-bit offsets inside an image's activity and inside the weights
   const int64_t weights = (int64_t)pg.nkx * pg.nky * pg.nkf * pg.patchSize;
   if (pg.pre.numExt() > 0x7fffffffLL || weights > 0x7fffffffLL) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   const FastGeom g = fast_geom(pg);
   const bool sparse = entries != nullptr;
   if (g.nfp >= 24 && g.nyp <= kWindow) {
      const pvgpu_status r = run_cols(pg, g, entries, numActive, aExt, W, gsyn, s);
      if (r != PVGPU_ERR_UNSUPPORTED_SHAPE) return r;
   }
   ScatPlan pl;
   const bool takesScatter = scatter_plan(pg, g, W, sparse, &pl);
   const double scatter = takesScatter ? scatter_cost(pg, g, sparse, pl) : 1e300;
   double cols;
   if (scatter > 40000 && cols_cost(pg, g, W, gsyn, sparse, &cols) && 1.5 * cols < scatter)
      return run_cols(pg, g, entries, numActive, aExt, W, gsyn, s);
   if (takesScatter) return run_scatter(pg, g, pl, entries, numActive, aExt, W, gsyn, s);
   return PVGPU_ERR_UNSUPPORTED_SHAPE;
}
