// deliver_post.cu -- a5: postsynaptic-perspective delivery (dense gather) in FP32.
//
// The reference computes, for every restricted target neuron, the dot product of its
// receptive field (nypPost rows of nxpPost*nf contiguous source values, starting at the
// unshrunken patch start) with the post-perspective weights
// (PostsynapticPerspectiveConvolveDelivery.cpp:56-151); its GPU path hands this to
// cudnnConvolutionForward after permuting NHWC->NCHW (CudaRecvPost.cpp:357-389).
//
// FAST mode is an implicit GEMM read straight from the NHWC extended activity: M = target
// positions, N = target features, K = nypPost * nxpPost * src.nf.  Positions are grouped by
// kernel phase (x mod nkx, y mod nky) so that one CTA tile shares one weight matrix.
// REFERENCE_ORDER mode runs one thread per target neuron with the reference's loop order and
// separately rounded products and sums.
#include "pvgpu_internal.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace {

using pvgpu::Axis;
using pvgpu::Loc;
namespace cg = cooperative_groups;
using pvgpu::num_sms;

struct PostGeom {
   Loc src, tgt;
   Axis ax, ay;       // tgt -> src geometry (pre = target layer, post = source layer)
   int nxpP, nypP;    // post-perspective patch
   int nkx, nky;      // kernel phases of the target layer
   int nkf;           // = tgt.nf
   int K, numPerStride, sy;
   float dtf;
};

// unshrunken source start (extended index) for a restricted target position (x, y)
__device__ __forceinline__ int64_t src_start(const PostGeom &g, int x, int y) {
   int sx = g.ax.start(x + g.tgt.lt) + g.src.lt;
   int sy = g.ay.start(y + g.tgt.dn) + g.src.dn;
   return ((int64_t)sy * g.src.nxExt() + sx) * g.src.nf;
}

__device__ __forceinline__ int post_kernel(const PostGeom &g, int x, int y, int f) {
   return ((y % g.nky) * g.nkx + (x % g.nkx)) * g.nkf + f;
}

// FAST mode: C[m][n] = sum_k A[m][k] B[n][k], one launch for all kernel phases (blockIdx.z).  A CTA
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
// 66 that a register-only loop of the same FMAs reaches (M = 32,768, N = 64, K = 12,544); for one
// image the length of the K loop, which the division over a cluster cuts.  8 x 8 per thread gained
// 8 % at K = 12,544 and lost 18 % at K = 192 (too few warps); operands laid out [k][row] with
// unpacked FMAs reached 0.8 of this.  Before: 64 x 64 tiles, 4 x 4 per thread, one register-staged
// buffer, 13 to 19 TFLOP/s.
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
struct PostTile {
   static constexpr int kThreads = (BM / TM) * (BN / TN);
   static constexpr size_t kSmem = sizeof(float) * kStages * LDK * (BM + BN) + 2 * sizeof(int64_t) * BM;
   static_assert((size_t)BM * BN <= (size_t)kStages * LDK * (BM + BN), "the partial tile reuses the buffers");
   static_assert(kThreads % 32 == 0, "whole warps");
};

template <int BM, int BN, int TM, int TN, int VW>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
      post_gemm_kernel(PostGeom g, int cz, const float *__restrict__ aExt, const float *__restrict__ W,
                       float *__restrict__ gsyn) {
   constexpr int T = PostTile<BM, BN, TM, TN>::kThreads;
   constexpr int RM = BM / TM, RN = BN / TN;  // a thread's rows are RM apart, its columns RN apart
   constexpr int CH = BK / VW;                // copies per row and step
   constexpr int RS = T / CH;                 // rows that one copy of all threads covers
   static_assert(T % CH == 0 && BM % RS == 0, "whole rounds of copies");
   extern __shared__ __align__(16) float sm[];
   float *As = sm, *Bs = sm + kStages * BM * LDK;
   int64_t *rowBase = reinterpret_cast<int64_t *>(sm + kStages * (BM + BN) * LDK), *outBase = rowBase + BM;

   const int phase = blockIdx.z;
   const int phx = phase % g.nkx, phy = phase / g.nkx;
   const int nxPh = g.tgt.nx / g.nkx, perImg = nxPh * (g.tgt.ny / g.nky);
   const int64_t M = (int64_t)perImg * g.tgt.nb;
   const int rank = cz > 1 ? blockIdx.x % cz : 0;
   const int64_t m0 = (int64_t)(blockIdx.x / cz) * BM;
   const int n0 = blockIdx.y * BN;
   const int tid = threadIdx.x;

   {  // each row's receptive field and output
      const int b0 = (int)(m0 / perImg), r0 = (int)(m0 - (int64_t)b0 * perImg);
      for (int i = tid; i < BM; i += T) {
         int64_t base = -1, out = -1;
         if (m0 + i < M) {
            const uint32_t q = (uint32_t)r0 + i, db = q / (uint32_t)perImg, p = q - db * perImg;
            const uint32_t yp = p / (uint32_t)nxPh;
            const int x = phx + g.nkx * (int)(p - yp * nxPh), y = phy + g.nky * (int)yp;
            base = (int64_t)(b0 + db) * g.src.numExt() + src_start(g, x, y);
            out = (int64_t)(b0 + db) * g.tgt.numRes() + ((int64_t)y * g.tgt.nx + x) * g.tgt.nf;
         }
         rowBase[i] = base;
         outBase[i] = out;
      }
   }
   __syncthreads();

   // this CTA's K range: whole steps
   const int steps = (g.K + BK - 1) / BK;
   const int per = (steps + cz - 1) / cz;
   const int s0 = min(rank * per, steps), nk = min(s0 + per, steps) - s0;

   // a thread copies the same VW columns of each step: its place (ky, r) in the field moves on by BK
   const int lc = (tid % CH) * VW, lr = tid / CH;
   int k = s0 * BK + lc;
   int r = k % g.numPerStride;
   const float *ak = aExt + (int64_t)(k / g.numPerStride) * g.sy;
   const float *wk = W + ((size_t)post_kernel(g, phx, phy, n0 + lr) * g.K + k);
   auto fill = [&](int buf) {
      float *a = As + (buf * BM + lr) * LDK + lc, *b = Bs + (buf * BN + lr) * LDK + lc;
      const bool kOn = k < g.K;
      const float *src = ak + r;
#pragma unroll 8
      for (int j = 0; j < BM / RS; j++) {
         const int64_t base = rowBase[lr + j * RS];
         const bool on = kOn && base >= 0;
         copy_async<VW>(a + j * RS * LDK, on ? src + base : aExt, on);
      }
#pragma unroll
      for (int j = 0; j < (BN + RS - 1) / RS; j++) {
         const bool on = kOn && n0 + lr + j * RS < g.nkf;
         if (BN % RS == 0 || lr + j * RS < BN)
            copy_async<VW>(b + j * RS * LDK, on ? wk + (size_t)j * RS * g.K : W, on);
      }
      k += BK;
      wk += BK;
      r += BK;
      while (r >= g.numPerStride) {
         r -= g.numPerStride;
         ak += g.sy;
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
#pragma unroll
      for (int i = 0; i < TM; i++) {
         const int64_t out = outBase[ty + i * RM];
         if (out < 0) continue;
#pragma unroll
         for (int j = 0; j < TN; j++) {
            const int n = n0 + tx + j * RN;
            if (n < g.nkf) gsyn[out + n] = fmaf(g.dtf, acc[i][j].x + acc[i][j].y, gsyn[out + n]);
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
      if (out >= 0 && n < g.nkf) {
         float v = cl.map_shared_rank(sm, 0)[e];
         for (int c = 1; c < cz; c++) v += cl.map_shared_rank(sm, c)[e];
         gsyn[out + n] = fmaf(g.dtf, v, gsyn[out + n]);
      }
   }
   cl.sync();  // no CTA leaves while another reads its tile
}

struct PostPick {
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
void consider(int tile, int64_t M, int N, int K, int phases, int vw, int sms, PostPick *best) {
   using Tile = PostTile<BM, BN, TM, TN>;
   constexpr int T = Tile::kThreads;
   const double tiles = (double)((M + BM - 1) / BM) * ((N + BN - 1) / BN) * phases;
   const double copies = (double)(BM + BN) / T / vw;
   const double fma = TM * TN, issue = fma / 2 + 0.3 * (TM + TN) + 14 * copies, lds = 2.6 * (TM + TN) + 4 * copies * (vw + 2);
   const double perK = std::max(fma, std::max(issue, lds)) * 1.15;
   const double occ = (int)std::min(2048.0 / T, std::min(220.0 * 1024 / Tile::kSmem, 65536.0 / T / (2 * TM * TN + 76)));
   for (int cz = 1; cz <= 8; cz *= 2) {
      if (cz > 1 && K / cz < 4 * BK) break;
      const double perSm = (double)(int64_t)((tiles * cz + sms - 1) / sms);
      const double share = perSm * T / 128, resident = std::min(share, occ * T / 128);
      const double cost = std::max(1.0, perSm / occ) * 2500 + perSm * ((cz > 1 ? 6500 : 0) + BM * BN / 128) +
                          (double)K / cz * perK * share * (1 + 0.8 / resident);
      if (cost < best->cost) *best = PostPick{tile, cz, cost};
   }
}

template <int BM, int BN, int TM, int TN, int VW>
pvgpu_status launch_post(const PostGeom &g, int64_t M, int cz, const float *aExt, const float *W, float *gsyn,
                         cudaStream_t s) {
   using Tile = PostTile<BM, BN, TM, TN>;
   const int64_t gx = (M + BM - 1) / BM * cz;
   const int gy = (g.nkf + BN - 1) / BN;
   if (gx > 0x7fffffff || gy > 65535) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   auto kernel = post_gemm_kernel<BM, BN, TM, TN, VW>;
   if (Tile::kSmem > 48 * 1024)
      PVGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile::kSmem),
                 "deliver_post attribute");
   cudaLaunchAttribute attr[1];
   attr[0].id = cudaLaunchAttributeClusterDimension;
   attr[0].val.clusterDim.x = cz;
   attr[0].val.clusterDim.y = 1;
   attr[0].val.clusterDim.z = 1;
   cudaLaunchConfig_t c = {};
   c.gridDim = dim3((unsigned)gx, gy, g.nkx * g.nky);
   c.blockDim = dim3(Tile::kThreads);
   c.dynamicSmemBytes = Tile::kSmem;
   c.stream = s;
   c.attrs = attr;
   c.numAttrs = cz > 1 ? 1 : 0;
   PVGPU_CUDA(cudaLaunchKernelEx(&c, kernel, g, cz, aExt, W, gsyn), "deliver_post");
   return PVGPU_OK;
}

template <int VW>
pvgpu_status run_post(const PostGeom &g, int64_t M, const float *aExt, const float *W, float *gsyn, cudaStream_t s) {
   const int phases = g.nkx * g.nky, sms = num_sms();
   PostPick p = {0, 1, 1e300};
   consider<64, 64, 8, 4>(0, M, g.nkf, g.K, phases, VW, sms, &p);
   consider<128, 32, 8, 4>(1, M, g.nkf, g.K, phases, VW, sms, &p);
   consider<64, 32, 8, 4>(2, M, g.nkf, g.K, phases, VW, sms, &p);
   consider<32, 32, 4, 4>(3, M, g.nkf, g.K, phases, VW, sms, &p);
   consider<128, 16, 8, 4>(4, M, g.nkf, g.K, phases, VW, sms, &p);
   consider<128, 4, 4, 4>(5, M, g.nkf, g.K, phases, VW, sms, &p);
   switch (p.tile) {
      case 0: return launch_post<64, 64, 8, 4, VW>(g, M, p.cz, aExt, W, gsyn, s);
      case 1: return launch_post<128, 32, 8, 4, VW>(g, M, p.cz, aExt, W, gsyn, s);
      case 2: return launch_post<64, 32, 8, 4, VW>(g, M, p.cz, aExt, W, gsyn, s);
      case 3: return launch_post<32, 32, 4, 4, VW>(g, M, p.cz, aExt, W, gsyn, s);
      case 4: return launch_post<128, 16, 8, 4, VW>(g, M, p.cz, aExt, W, gsyn, s);
      default: return launch_post<128, 4, 4, 4, VW>(g, M, p.cz, aExt, W, gsyn, s);
   }
}

// REFERENCE_ORDER: one thread per restricted target neuron, loops as in the reference.
__global__ void post_exact_kernel(PostGeom g, const float *__restrict__ aExt, const float *__restrict__ W,
                                  float *__restrict__ gsyn) {
   int64_t idxAll = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   int64_t nRes = g.tgt.numRes();
   if (idxAll >= nRes * g.tgt.nb) return;
   int b = (int)(idxAll / nRes);
   int64_t idx = idxAll % nRes;
   int f = (int)(idx % g.tgt.nf);
   int x = (int)((idx / g.tgt.nf) % g.tgt.nx);
   int y = (int)(idx / ((int64_t)g.tgt.nf * g.tgt.nx));
   const float *a0 = aExt + (size_t)b * g.src.numExt() + src_start(g, x, y);
   const float *w0 = W + (size_t)post_kernel(g, x, y, f) * g.K;
   float gs = gsyn[idxAll];
   for (int ky = 0; ky < g.nypP; ky++) {
      const float *a = a0 + (int64_t)ky * g.sy;
      const float *w = w0 + ky * g.numPerStride;
      float dv = 0.0f;
      for (int k = 0; k < g.numPerStride; k++) dv = __fadd_rn(dv, __fmul_rn(a[k], w[k]));
      gs = __fadd_rn(gs, __fmul_rn(g.dtf, dv));
   }
   gsyn[idxAll] = gs;
}

}  // namespace

extern "C" pvgpu_status pvgpu_deliver_post(const pvgpu_conn_desc *conn, const float *aExt, const float *postWeights,
                                           float *gsyn, int mode, void *stream) {
   if (!conn || !aExt || !postWeights || !gsyn) return PVGPU_ERR_BAD_ARG;
   const pvgpu_loc &pre = conn->pre, &post = conn->post;
   if (!pvgpu::loc_valid(pre) || !pvgpu::loc_valid(post) || pre.nbatch != post.nbatch) return PVGPU_ERR_BAD_ARG;
   if (!pvgpu::axis_legal(pre.nx, post.nx, conn->nxp) || !pvgpu::axis_legal(pre.ny, post.ny, conn->nyp))
      return PVGPU_ERR_ILLEGAL_GEOMETRY;
   PostGeom g;
   g.src = pvgpu::to_loc(pre);
   g.tgt = pvgpu::to_loc(post);
   g.nxpP = pvgpu::post_patch_size(conn->nxp, pre.nx, post.nx);
   g.nypP = pvgpu::post_patch_size(conn->nyp, pre.ny, post.ny);
   // The post-perspective read needs the whole unshrunken receptive field inside the halo.
   int mx = pvgpu::required_margin(post.nx, pre.nx, g.nxpP), my = pvgpu::required_margin(post.ny, pre.ny, g.nypP);
   if (pre.halo.lt < mx || pre.halo.rt < mx || pre.halo.dn < my || pre.halo.up < my) return PVGPU_ERR_BAD_ARG;
   // PatchGeometry::setPatchGeometry offsets x by the post halo's dn (components/PatchGeometry.cpp:194-206);
   // equal margins on both axes keep that identical to lt.
   if (pre.halo.lt != pre.halo.dn || pre.halo.lt != pre.halo.rt || pre.halo.dn != pre.halo.up)
      return PVGPU_ERR_UNSUPPORTED_SHAPE;
   g.ax = Axis{post.nx, pre.nx, g.nxpP, post.halo.lt};
   g.ay = Axis{post.ny, pre.ny, g.nypP, post.halo.dn};
   g.nkx = post.nx > pre.nx ? post.nx / pre.nx : 1;
   g.nky = post.ny > pre.ny ? post.ny / pre.ny : 1;
   g.nkf = post.nf;
   g.numPerStride = g.nxpP * pre.nf;
   g.K = g.nypP * g.numPerStride;
   g.sy = g.src.nxExt() * pre.nf;
   g.dtf = conn->dt_factor;
   cudaStream_t s = pvgpu::as_stream(stream);
   if (mode == PVGPU_DELIVER_REFERENCE_ORDER) {
      int64_t n = g.tgt.numRes() * g.tgt.nb;
      post_exact_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, aExt, postWeights, gsyn);
      PVGPU_CHECK_LAUNCH("deliver_post exact");
      return PVGPU_OK;
   }
   const int64_t M = (int64_t)(post.nx / g.nkx) * (post.ny / g.nky) * post.nbatch;
   if (g.nkx * g.nky > 65535) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   // floats per copy: every receptive field's row, every weight row and both buffers start on a
   // multiple of it.  Fields start at multiples of pre.nf * stride (consecutive positions) from the
   // first one's offset.
   const int strideX = pre.nx > post.nx ? pre.nx / post.nx : 1, strideY = pre.ny > post.ny ? pre.ny / post.ny : 1;
   auto aligned = [&](int n) {
      if (reinterpret_cast<uintptr_t>(aExt) % (4 * n) || reinterpret_cast<uintptr_t>(postWeights) % (4 * n)) return false;
      if (g.numPerStride % n || g.src.numExt() % n || (int64_t)strideY * g.sy % n || g.sy % n) return false;
      if ((int64_t)strideX * pre.nf % n) return false;
      for (int ph = 0; ph < g.nkx; ph++)  // the first field of each phase; rows are multiples of sy apart
         if ((int64_t)(g.ax.start(ph + g.tgt.lt) + g.src.lt) * pre.nf % n) return false;
      return true;
   };
   if (aligned(4)) return run_post<4>(g, M, aExt, postWeights, gsyn, s);
   if (aligned(2)) return run_post<2>(g, M, aExt, postWeights, gsyn, s);
   return run_post<1>(g, M, aExt, postWeights, gsyn, s);
}
