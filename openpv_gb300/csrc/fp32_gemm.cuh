// fp32_gemm.cuh -- the FP32 GEMM on the FMA pipes behind the postsynaptic delivery and the plain form of
// the LCA solver: operands gathered row by row, any epilogue.
#pragma once

#include "pvgpu_internal.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace pvgpu {
namespace fp32_gemm {

namespace cg = cooperative_groups;

// C[m][n] = sum_k A[m][k] B[n][k], one launch for all phases of a problem (blockIdx.z).  A CTA
// computes BM x BN with TM x TN per thread; the K loop runs over kStages buffers of BK, filled by
// asynchronous copies of VW floats (4, 2 or 1: what the alignment of the receptive fields' rows
// allows -- an image of three features starts anywhere).  Both operands lie [row][k] in shared
// memory, rows 80 bytes apart, so that copies go along k and a thread's fragments are conflict-free
// 16-byte loads of four k.  Even and odd k accumulate in the two halves of a packed FMA
// (__ffma2_rn): its operands are the fragments as they were loaded, without the moves that pairing
// two outputs would need, and each half is a chain of K/2 additions.  With cz > 1 the K loop is
// divided over a cluster of cz CTAs and the partial tiles are summed through distributed shared
// memory in rank order.
//
// What bounds it: shared-memory and FMA cycles about equally for large layers, 44 TFLOP/s of the
// 66 that a register-only loop of the same FMAs reaches (M = 32,768, N = 64, K = 12,544; 13 to 19 with 64 x 64
// tiles of 4 x 4 per thread and one register-staged buffer); for one image the length of the K loop, which the
// division over a cluster cuts.
constexpr int BK = 16, LDK = BK + 4, kStages = 4;

template <int VW>
__device__ __forceinline__ void copy_async(float *dst, const float *src, bool valid) {
   const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
   const int n = valid ? 4 * VW : 0;
   if constexpr (VW == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
   else if constexpr (VW == 2) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
   else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int BM, int BN, int TM, int TN>
struct Tile {
   static constexpr int kThreads = (BM / TM) * (BN / TN);
   static constexpr size_t kSmem = sizeof(float) * kStages * LDK * (BM + BN) + 2 * sizeof(int64_t) * BM;
   static_assert((size_t)BM * BN <= (size_t)kStages * LDK * (BM + BN), "the partial tile reuses the buffers");
   static_assert(kThreads % 32 == 0, "whole warps");
};

// Problem: M, N, K; A's row m is K / stride runs of `stride` values, `sy` apart, from row()'s base; B's
// row n of a phase is K values at b(phase) + n K; old() reads what store() needs beside the sum.
template <int BM, int BN, int TM, int TN, int VW, typename Problem>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_kernel(const Problem p, int cz) {
   constexpr int T = Tile<BM, BN, TM, TN>::kThreads;
   constexpr int RM = BM / TM, RN = BN / TN;  // a thread's rows are RM apart, its columns RN apart
   constexpr int CH = BK / VW;                // copies per row and step
   constexpr int RS = T / CH;                 // rows that one copy of all threads covers
   static_assert(T % CH == 0 && BM % RS == 0, "whole rounds of copies");
   extern __shared__ __align__(16) float sm[];
   float *As = sm, *Bs = sm + kStages * BM * LDK;
   int64_t *rowBase = reinterpret_cast<int64_t *>(sm + kStages * (BM + BN) * LDK), *outBase = rowBase + BM;

   const int phase = blockIdx.z;
   const int rank = cz > 1 ? blockIdx.x % cz : 0;
   const int64_t m0 = (int64_t)(blockIdx.x / cz) * BM;
   const int n0 = blockIdx.y * BN;
   const int tid = threadIdx.x;

   {  // each row's first operand value and its output
      const auto at = p.begin(phase, m0);
      for (int i = tid; i < BM; i += T) {
         int64_t base = -1, out = -1;
         if (m0 + i < p.M) p.row(at, phase, m0, i, &base, &out);
         rowBase[i] = base;
         outBase[i] = out;
      }
   }
   __syncthreads();

   // this CTA's K range: whole steps
   const int steps = (p.K + BK - 1) / BK;
   const int per = (steps + cz - 1) / cz;
   const int s0 = min(rank * per, steps), nk = min(s0 + per, steps) - s0;

   // a thread copies the same VW columns of each step: its place (ky, r) in the field moves on by BK
   const int lc = (tid % CH) * VW, lr = tid / CH;
   int k = s0 * BK + lc;
   int r = k % p.stride;
   const float *ak = p.a + (int64_t)(k / p.stride) * p.sy;
   const float *wk = p.b(phase) + ((size_t)(n0 + lr) * p.K + k);
   auto fill = [&](int buf) {
      float *a = As + (buf * BM + lr) * LDK + lc, *b = Bs + (buf * BN + lr) * LDK + lc;
      const bool kOn = k < p.K;
      const float *src = ak + r;
#pragma unroll 8
      for (int j = 0; j < BM / RS; j++) {
         const int64_t base = rowBase[lr + j * RS];
         const bool on = kOn && base >= 0;
         copy_async<VW>(a + j * RS * LDK, on ? src + base : p.a, on);
      }
#pragma unroll
      for (int j = 0; j < (BN + RS - 1) / RS; j++) {
         const bool on = kOn && n0 + lr + j * RS < p.N;
         if (BN % RS == 0 || lr + j * RS < BN)
            copy_async<VW>(b + j * RS * LDK, on ? wk + (size_t)j * RS * p.K : p.a, on);
      }
      k += BK;
      wk += BK;
      r += BK;
      while (r >= p.stride) {
         r -= p.stride;
         ak += p.sy;
      }
   };

   const int tx = tid % RN, ty = tid / RN;
   float2 acc[TM][TN];
#pragma unroll
   for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) acc[i][j] = make_float2(0.0f, 0.0f);

#pragma unroll
   for (int s = 0; s < kStages - 1; s++) {
      if (s < nk) fill(s);
      asm volatile("cp.async.commit_group;" ::: "memory");
   }
   for (int t = 0; t < nk; t++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncthreads();
      if (t + kStages - 1 < nk) fill((t + kStages - 1) % kStages);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float *a = As + ((t % kStages) * BM + ty) * LDK, *b = Bs + ((t % kStages) * BN + tx) * LDK;
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
         float4 bv[TN];
#pragma unroll
         for (int j = 0; j < TN; j++) bv[j] = *reinterpret_cast<const float4 *>(b + j * RN * LDK + kk);
#pragma unroll
         for (int i = 0; i < TM; i++) {
            const float4 av = *reinterpret_cast<const float4 *>(a + i * RM * LDK + kk);
#pragma unroll
            for (int j = 0; j < TN; j++) {
               acc[i][j] = __ffma2_rn(make_float2(av.x, av.y), make_float2(bv[j].x, bv[j].y), acc[i][j]);
               acc[i][j] = __ffma2_rn(make_float2(av.z, av.w), make_float2(bv[j].z, bv[j].w), acc[i][j]);
            }
         }
      }
   }

   if (cz == 1) {
      // half of the rows at a time: all their reads, then all their stores
#pragma unroll
      for (int h = 0; h < TM; h += TM / 2) {
         typename Problem::Old old[TM / 2][TN];
#pragma unroll
         for (int i = 0; i < TM / 2; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) {
               const int64_t out = outBase[ty + (h + i) * RM];
               const int n = n0 + tx + j * RN;
               if (out >= 0 && n < p.N) old[i][j] = p.old(out, n);
            }
#pragma unroll
         for (int i = 0; i < TM / 2; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) {
               const int64_t out = outBase[ty + (h + i) * RM];
               const int n = n0 + tx + j * RN;
               if (out >= 0 && n < p.N) p.store(out, n, acc[h + i][j].x + acc[h + i][j].y, old[i][j]);
            }
      }
      return;
   }
   // the cluster's partial tiles, each CTA summing its share of the rows
   asm volatile("cp.async.wait_group 0;" ::: "memory");
   __syncthreads();
#pragma unroll
   for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) sm[(ty + i * RM) * BN + tx + j * RN] = acc[i][j].x + acc[i][j].y;
   cg::cluster_group cl = cg::this_cluster();
   cl.sync();
   for (int e = rank * (BM / cz) * BN + tid; e < (rank + 1) * (BM / cz) * BN; e += T) {
      const int64_t out = outBase[e / BN];
      const int n = n0 + e % BN;
      if (out >= 0 && n < p.N) {
         float v = cl.map_shared_rank(sm, 0)[e];
         for (int c = 1; c < cz; c++) v += cl.map_shared_rank(sm, c)[e];
         p.store(out, n, v, p.old(out, n));
      }
   }
   cl.sync();  // no CTA leaves while another reads its tile
}

struct Pick {
   int tile, cz;
   double cost;
};

// Estimated cycles of a launch: per k and warp the FMA pipe's cycles, the instructions issued or the
// shared-memory cycles of a scheduler's share (fragment loads at 2.6 cycles, the copies' stores),
// whichever is most; times the steps of a CTA's K range and the warps that share a scheduler on the
// busiest SM, more where few of them are resident; the start and end of each wave of CTAs; and the
// exchange of a cluster.  The factors reproduce, within about a fifth, a sweep of all tiles and
// divisions over eight shapes (M 256 to 78,000, N 6 to 512, K 64 to 12,544), and pick the fastest or
// one within 7 % of it on seven of them (M = 78,000, N = 6: 218 us picked, 173 us at cz = 4).
template <int BM, int BN, int TM, int TN>
void consider(int tile, int64_t M, int N, int K, int phases, int vw, int sms, Pick *best) {
   using Shape = Tile<BM, BN, TM, TN>;
   constexpr int T = Shape::kThreads;
   const double tiles = (double)((M + BM - 1) / BM) * ((N + BN - 1) / BN) * phases;
   const double copies = (double)(BM + BN) / T / vw;
   const double fma = TM * TN, issue = fma / 2 + 0.3 * (TM + TN) + 14 * copies, lds = 2.6 * (TM + TN) + 4 * copies * (vw + 2);
   const double perK = std::max(fma, std::max(issue, lds)) * 1.15;
   const double occ = (int)std::min(2048.0 / T, std::min(220.0 * 1024 / Shape::kSmem, 65536.0 / T / (2 * TM * TN + 76)));
   for (int cz = 1; cz <= 8; cz *= 2) {
      if (cz > 1 && K / cz < 4 * BK) break;
      const double perSm = (double)(int64_t)((tiles * cz + sms - 1) / sms);
      const double share = perSm * T / 128, resident = std::min(share, occ * T / 128);
      const double cost = std::max(1.0, perSm / occ) * 2500 + perSm * ((cz > 1 ? 6500 : 0) + BM * BN / 128) +
                          (double)K / cz * perK * share * (1 + 0.8 / resident);
      if (cost < best->cost) *best = Pick{tile, cz, cost};
   }
}

template <int BM, int BN, int TM, int TN, int VW, typename Problem>
pvgpu_status launch(const Problem &p, int phases, int cz, cudaStream_t s, const char *where) {
   using Shape = Tile<BM, BN, TM, TN>;
   const int64_t gx = (p.M + BM - 1) / BM * cz;
   const int gy = (p.N + BN - 1) / BN;
   if (gx > 0x7fffffff || gy > 65535) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   auto kernel = gemm_kernel<BM, BN, TM, TN, VW, Problem>;
   if (Shape::kSmem > 48 * 1024)
      PVGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape::kSmem), where);
   cudaLaunchAttribute attr[1];
   attr[0].id = cudaLaunchAttributeClusterDimension;
   attr[0].val.clusterDim.x = cz;
   attr[0].val.clusterDim.y = 1;
   attr[0].val.clusterDim.z = 1;
   cudaLaunchConfig_t c = {};
   c.gridDim = dim3((unsigned)gx, gy, phases);
   c.blockDim = dim3(Shape::kThreads);
   c.dynamicSmemBytes = Shape::kSmem;
   c.stream = s;
   c.attrs = attr;
   c.numAttrs = cz > 1 ? 1 : 0;
   PVGPU_CUDA(cudaLaunchKernelEx(&c, kernel, p, cz), where);
   return PVGPU_OK;
}

// Runs the problem with the tile and the division of K of least estimated time.  VW: floats per copy
// (every run of A, every row of B and both pointers start on a multiple of it).
template <int VW, typename Problem>
pvgpu_status run(const Problem &p, int phases, cudaStream_t s, const char *where) {
   const int sms = num_sms();
   Pick q = {0, 1, 1e300};
   consider<64, 64, 8, 4>(0, p.M, p.N, p.K, phases, VW, sms, &q);
   consider<128, 32, 8, 4>(1, p.M, p.N, p.K, phases, VW, sms, &q);
   consider<64, 32, 8, 4>(2, p.M, p.N, p.K, phases, VW, sms, &q);
   consider<32, 32, 4, 4>(3, p.M, p.N, p.K, phases, VW, sms, &q);
   consider<128, 16, 8, 4>(4, p.M, p.N, p.K, phases, VW, sms, &q);
   consider<128, 4, 4, 4>(5, p.M, p.N, p.K, phases, VW, sms, &q);
   switch (q.tile) {
      case 0: return launch<64, 64, 8, 4, VW>(p, phases, q.cz, s, where);
      case 1: return launch<128, 32, 8, 4, VW>(p, phases, q.cz, s, where);
      case 2: return launch<64, 32, 8, 4, VW>(p, phases, q.cz, s, where);
      case 3: return launch<32, 32, 4, 4, VW>(p, phases, q.cz, s, where);
      case 4: return launch<128, 16, 8, 4, VW>(p, phases, q.cz, s, where);
      default: return launch<128, 4, 4, 4, VW>(p, phases, q.cz, s, where);
   }
}

}  // namespace fp32_gemm
}  // namespace pvgpu
