// weights.cu -- a3 / a12: weight transpose for post-perspective delivery and the Hebbian
// weight update (the weight gradient of delivery).
#include "fast_axis.cuh"

#include <climits>
#include <type_traits>

namespace {

using pvgpu::Axis;
using pvgpu::FastAxis;
using pvgpu::Loc;

struct TGeom {
   int nxp, nyp, nfp;           // pre patch (nfp = post.nf)
   int nkx, nky, nkf;           // pre kernels
   int xStride, yStride, xTStride, yTStride;
   int nxpPost, nypPost;
   int nkxPost, nkyPost, nkfPost;
};

// PatchGeometry::setTransposeItemIndices (components/PatchGeometry.cpp:264-332) and
// TransposeWeights::transposeShared (utils/TransposeWeights.cpp:56-115), one thread per pre weight.
__global__ void transpose_kernel(TGeom g, const float *__restrict__ wPre, float *__restrict__ wPost) {
   const int patchSize = g.nxp * g.nyp * g.nfp;
   const int64_t total = (int64_t)g.nkx * g.nky * g.nkf * patchSize;
   int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= total) return;
   int kp = (int)(t / patchSize), item = (int)(t % patchSize);
   int kxPre = (kp / g.nkf) % g.nkx, kyPre = kp / (g.nkf * g.nkx), kfPre = kp % g.nkf;
   int ixPre = (item / g.nfp) % g.nxp, iyPre = item / (g.nfp * g.nxp), ifPre = item % g.nfp;
   int extX = (g.nxp - 1) * g.xStride / 2;
   int ksX = (kxPre - extX) % g.xStride;
   if (ksX < 0) ksX += g.xStride;
   int ixPost = (g.xStride * (g.nxp - 1 - ixPre) + ksX) / g.xTStride;
   int extY = (g.nyp - 1) * g.yStride / 2;
   int ksY = (kyPre - extY) % g.yStride;
   if (ksY < 0) ksY += g.yStride;
   int iyPost = (g.yStride * (g.nyp - 1 - iyPre) + ksY) / g.yTStride;
   int itemPost = (iyPost * g.nxpPost + ixPost) * g.nkf + kfPre;
   int pxPost = 0, pyPost = 0;
   if (g.nkxPost > 1) {
      pxPost = (-(g.nxp - g.nkxPost) / 2 + ixPre) % g.nkxPost;
      if (pxPost < 0) pxPost += g.nkxPost;
   }
   if (g.nkyPost > 1) {
      pyPost = (-(g.nyp - g.nkyPost) / 2 + iyPre) % g.nkyPost;
      if (pyPost < 0) pyPost += g.nkyPost;
   }
   int patchPost = (pyPost * g.nkxPost + pxPost) * g.nkfPost + ifPre;
   int patchSizePost = g.nxpPost * g.nypPost * g.nkf;
   wPost[(size_t)patchPost * patchSizePost + itemPost] = wPre[t];
}

struct HGeom {
   FastAxis ax, ay;
   int64_t nPreExt, nPostExt;
   int nb, preNf, preNxExt, postNx, postNy, postNf, postNxExt, postDn;
   int nxp, nyp, patchSize;
   int nkx, nky;
   float dWMax;
};

// HebbianUpdater::update_dW / updateInd_dW (weightupdaters/HebbianUpdater.cpp:476-629): each weight
// (kernel, ky, kx, fp) sums dWMax*pre*post over the batch, then the kernel's unit cells in (y, x)
// order -- the order the reference accumulates into that weight -- wherever the weight lies inside
// the (shrunken) patch and pre is not zero.
//
// That order makes every weight one serial chain, so the work is laid out for the chain's latency:
// a CTA takes FC consecutive presynaptic features of one kernel phase; its warps first read a segment
// of the activity (lanes = FC features x 32/FC positions of a row, so that a sector is read once)
// and list the nonzeros of each feature in order in shared memory, decoded; then each warp walks one
// feature's list with its lanes on 32 * EPT weights of the patch.  Zeros cost a lane's share of a load
// instead of a step of every chain.  The next segment's loads are issued before the lists are walked.
//
// 32 images of 16x16x512 at 5 % against 32x32x3 errors, 8x8 patches: 92 us (57 M instructions, issue slots
// 62 % busy: the scan, and the walk, where nearly every group of entries has a patch that hangs over the
// image's edge and is tested weight by weight); one thread per weight walking every position itself took 4.3 ms.
// W = the most warps a CTA has.  Patches whose weights take more than 16 warps at one weight a lane get up
// to 32 warps of one or two weights a lane, with half the loads per warp and segment (the lists of a
// segment stay at 128 KB): twice the chains in flight.  The call above: 118 us with 16 warps of two
// weights, 92 with 24 of one; half the loads per segment without the warps 134; two features a CTA
// instead of four 146 (each sector read by four CTAs).

// WIDE: post activities of 2^31 values and more (64-bit offsets, computed in the walk).
// OVER: a patch wider or taller than the post layer lies mostly outside it, so the entries that put some weight
// of the warp inside are picked out first, 32 at a time.  4x1x107 -> 171 features, 7x13 patches, dense: 110 us
// with every weight of every entry tested (39 with one thread per weight walking the positions), now 32.
template <int EPT, int FC, int W, bool WIDE, bool OVER>
__global__ void __launch_bounds__(W * 32) hebbian_kernel(HGeom g, int slabsPerCta,
                                                                  const float *__restrict__ preExt,
                                                                  const float *__restrict__ postExt,
                                                                  float *__restrict__ dw) {
   constexpr int PL = 32 / FC;    // positions per load
   constexpr int kSL = 256 / W;   // loads per warp and segment
   extern __shared__ __align__(16) int4 recs[];  // [FC][cap]
   __shared__ int counts[2][W][8];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
   const int cap = NW * kSL * PL;
   const int groups = (g.preNf + FC - 1) / FC;
   const int phase = blockIdx.x / groups, F0 = (blockIdx.x % groups) * FC;
   const int kxc = phase % g.nkx, kyc = phase / g.nkx;

   // the phase's rows and columns whose patch reaches the post layer
   auto range = [](const FastAxis &ax, int c, int step, int patch, int nPost, int &first) {
      first = c;
      while (first < ax.n && ax.start(first) + patch <= 0) first += step;
      int end = ax.first_ge(nPost);  // one past the last
      return end > first ? (end - first + step - 1) / step : 0;
   };
   int ye0, xe0;
   const int nyC = range(g.ay, kyc, g.nky, g.nyp, g.postNy, ye0);
   const int nxC = range(g.ax, kxc, g.nkx, g.nxp, g.postNx, xe0);
   const int G = (nxC + PL - 1) / PL;                 // loads per row
   const int64_t loads = (int64_t)g.nb * nyC * G;

   // scanning: this lane's feature and position within a load
   const int sf = lane % FC, sp = lane / FC;
   const unsigned fmask = (FC == 1 ? 0xffffffffu : FC == 2 ? 0x55555555u : FC == 4 ? 0x11111111u : 0x01010101u) << sf;
   const bool fOn = F0 + sf < g.preNf;

   // walking: this warp's feature and this lane's weights
   const int wf = warp % FC, slab = blockIdx.y * slabsPerCta + warp / FC;
   using Offset = typename std::conditional<WIDE, int64_t, int>::type;
   Offset eo[EPT];
   int kx[EPT], ky[EPT];
   float acc[EPT];
#pragma unroll
   for (int i = 0; i < EPT; i++) {
      int e = slab * 32 * EPT + lane + 32 * i;
      if (e >= g.patchSize) e = 0;
      const int fp = e % g.postNf;
      kx[i] = (e / g.postNf) % g.nxp;
      ky[i] = e / (g.postNf * g.nxp);
      eo[i] = ((Offset)ky[i] * g.postNxExt + kx[i]) * g.postNf + fp;
      acc[i] = 0.0f;
   }
   const bool walks = warp / FC < slabsPerCta && slab * 32 * EPT < g.patchSize && F0 + wf < g.preNf;

   // the position of a load: image, row and load within the row
   struct At {
      int b, y, c;
   };
   auto at = [&](int64_t q) {
      const int row = (int)(q / G);
      At p;
      p.c = (int)(q - (int64_t)row * G);
      p.b = row / nyC;
      p.y = row - p.b * nyC;
      return p;
   };
   auto next = [&](At &p) {
      if (++p.c == G) {
         p.c = 0;
         if (++p.y == nyC) {
            p.y = 0;
            p.b++;
         }
      }
   };
   float val[kSL];
   At mine = {0, 0, 0};  // of this warp's first load in the segment
   auto fetch = [&](int64_t q0) {
#pragma unroll
      for (int s = 0; s < kSL; s++) val[s] = 0.0f;
      if (q0 >= loads) return;
      mine = at(q0);
      At p = mine;
#pragma unroll
      for (int s = 0; s < kSL; s++) {
         const int xi = p.c * PL + sp;
         if (q0 + s < loads && xi < nxC && fOn)
            val[s] = __ldg(preExt + (size_t)p.b * g.nPreExt +
                           ((size_t)(ye0 + p.y * g.nky) * g.preNxExt + xe0 + xi * g.nkx) * g.preNf + F0 + sf);
         next(p);
      }
   };
   const int64_t perSeg = (int64_t)NW * kSL;
   const int segs = (int)((loads + perSeg - 1) / perSeg);
   fetch((int64_t)warp * kSL);
   for (int seg = 0; seg < segs; seg++) {
      // this warp's count of each feature
      unsigned ball[kSL];
      int cnt = 0;
#pragma unroll
      for (int s = 0; s < kSL; s++) {
         ball[s] = __ballot_sync(0xffffffffu, val[s] != 0.0f) & fmask;
         cnt += __popc(ball[s]);
      }
      int *cn = &counts[seg & 1][0][0];
      if (lane < FC) cn[warp * 8 + lane] = cnt;
      __syncthreads();  // counts written; the lists of the segment before walked
      int base = 0, n = 0;
#pragma unroll
      for (int f = 0; f < FC; f++) {
         const int c = lane < NW ? cn[lane * 8 + f] : 0;
         const int before = __reduce_add_sync(0xffffffffu, lane < warp ? c : 0), all = __reduce_add_sync(0xffffffffu, c);
         if (f == sf) base = before;
         if (f == wf) n = all;
      }
      At p = mine;
#pragma unroll
      for (int s = 0; s < kSL; s++) {
         if (val[s] != 0.0f) {
            const int sy = g.ay.start(ye0 + p.y * g.nky), sx = g.ax.start(xe0 + (p.c * PL + sp) * g.nkx);
            // the x offset uses the post halo's dn, as PatchGeometry::setPatchGeometry's aPostOffset
            // does (components/PatchGeometry.cpp:194-206); margins are equal on both axes in practice
            int4 q;
            q.x = WIDE ? p.b : (int)(p.b * g.nPostExt) + ((sy + g.postDn) * g.postNxExt + sx + g.postDn) * g.postNf;
            q.y = sx;
            q.z = sy;
            if (!WIDE && sx >= 0 && sy >= 0 && sx + g.nxp <= g.postNx && sy + g.nyp <= g.postNy) q.y = q.z = INT_MIN;  // whole
            q.w = __float_as_int(__fmul_rn(g.dWMax, val[s]));
            recs[sf * cap + base + __popc(ball[s] & ((1u << lane) - 1))] = q;
         }
         base += __popc(ball[s]);
         next(p);
      }
      __syncthreads();
      fetch((int64_t)(seg + 1) * perSeg + (int64_t)warp * kSL);
      if (walks) {
         const int4 *list = recs + wf * cap;
         auto offset = [&](const int4 &q) -> Offset {
            if constexpr (WIDE)
               return (int64_t)q.x * g.nPostExt + ((int64_t)(q.z + g.postDn) * g.postNxExt + q.y + g.postDn) * g.postNf;
            else return q.x;
         };
         auto take = [&](auto un, int k) {
            constexpr int U = decltype(un)::value;
            int4 q[U];
            float v[U][EPT];
            bool whole = true;
#pragma unroll
            for (int u = 0; u < U; u++) {
               q[u] = list[k + u];
               whole = whole && q[u].z == INT_MIN;
            }
            if (whole) {
#pragma unroll
               for (int u = 0; u < U; u++)
#pragma unroll
                  for (int i = 0; i < EPT; i++) v[u][i] = __ldg(postExt + (offset(q[u]) + eo[i]));
#pragma unroll
               for (int u = 0; u < U; u++)
#pragma unroll
                  for (int i = 0; i < EPT; i++)
                     acc[i] = __fadd_rn(acc[i], __fmul_rn(__int_as_float(q[u].w), v[u][i]));
            } else {
               bool ok[U][EPT];
#pragma unroll
               for (int u = 0; u < U; u++)
#pragma unroll
                  for (int i = 0; i < EPT; i++) {
                     ok[u][i] = q[u].z == INT_MIN ||
                                ((unsigned)(q[u].y + kx[i]) < (unsigned)g.postNx && (unsigned)(q[u].z + ky[i]) < (unsigned)g.postNy);
                     v[u][i] = ok[u][i] ? __ldg(postExt + (offset(q[u]) + eo[i])) : 0.0f;
                  }
#pragma unroll
               for (int u = 0; u < U; u++)
#pragma unroll
                  for (int i = 0; i < EPT; i++)
                     if (ok[u][i]) acc[i] = __fadd_rn(acc[i], __fmul_rn(__int_as_float(q[u].w), v[u][i]));
            }
         };
         if constexpr (OVER) {
            const int e0 = slab * 32 * EPT, e1 = min(e0 + 32 * EPT, g.patchSize) - 1, perRow = g.postNf * g.nxp;
            const int kyLo = e0 / perRow, kyHi = e1 / perRow;  // the patch rows and columns of the warp's weights
            const int kxLo = kyLo == kyHi ? e0 / g.postNf - kyLo * g.nxp : 0;
            const int kxHi = kyLo == kyHi ? e1 / g.postNf - kyLo * g.nxp : g.nxp - 1;
            for (int k0 = 0; k0 < n; k0 += 32) {
               bool reaches = false;
               if (k0 + lane < n) {
                  const int4 q = list[k0 + lane];
                  reaches = q.z + kyHi >= 0 && q.z + kyLo < g.postNy && q.y + kxHi >= 0 && q.y + kxLo < g.postNx;
               }
               unsigned m = __ballot_sync(0xffffffffu, reaches);
               while (m) {
                  constexpr int U = EPT >= 8 ? 2 : 4;
                  int4 q[U];
                  float v[U][EPT];
                  bool ok[U][EPT];
#pragma unroll
                  for (int u = 0; u < U; u++) {
                     const bool on = m != 0;
                     q[u] = list[on ? k0 + __ffs(m) - 1 : k0];
                     m &= m - 1;
#pragma unroll
                     for (int i = 0; i < EPT; i++) {
                        ok[u][i] = on && (unsigned)(q[u].y + kx[i]) < (unsigned)g.postNx && (unsigned)(q[u].z + ky[i]) < (unsigned)g.postNy;
                        v[u][i] = ok[u][i] ? __ldg(postExt + (offset(q[u]) + eo[i])) : 0.0f;
                     }
                  }
#pragma unroll
                  for (int u = 0; u < U; u++)
#pragma unroll
                     for (int i = 0; i < EPT; i++)
                        if (ok[u][i]) acc[i] = __fadd_rn(acc[i], __fmul_rn(__int_as_float(q[u].w), v[u][i]));
               }
            }
         } else {
            constexpr int U = EPT >= 8 ? 2 : EPT >= 2 ? 4 : 8;
            int k = 0;
            for (; k + U <= n; k += U) take(std::integral_constant<int, U>(), k);
            for (; k < n; k++) take(std::integral_constant<int, 1>(), k);
         }
      }
   }
   if (walks) {
      float *d = dw + ((size_t)phase * g.preNf + F0 + wf) * g.patchSize;
#pragma unroll
      for (int i = 0; i < EPT; i++) {
         const int e = slab * 32 * EPT + lane + 32 * i;
         if (e < g.patchSize) d[e] = acc[i];
      }
   }
}

// The lists of a CTA of W warps, the most that any launch takes.  The limit that a launch is checked against
// belongs to the kernel, and another thread may be launching it with a smaller layer, so it is always set to this.
constexpr size_t kListBytes = sizeof(int4) * 256 * 32;

template <int EPT, int FC, int W, bool WIDE = false, bool OVER = false>
pvgpu_status launch_hebbian(const HGeom &g, const float *preExt, const float *postExt, float *dw, cudaStream_t s) {
   const int slabs = (g.patchSize + 32 * EPT - 1) / (32 * EPT);
   const int perCta = slabs < W / FC ? slabs : W / FC;
   const int64_t gx = (int64_t)g.nkx * g.nky * ((g.preNf + FC - 1) / FC);
   const int warps = perCta * FC < 8 ? 8 : perCta * FC;  // warps beyond the lists only scan
   const int gy = (slabs + perCta - 1) / perCta;
   if (gx > 0x7fffffff || gy > 65535) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   const size_t smem = kListBytes / W * warps;
   PVGPU_CUDA(cudaFuncSetAttribute(hebbian_kernel<EPT, FC, W, WIDE, OVER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kListBytes),
              "hebbian_dw attribute");
   hebbian_kernel<EPT, FC, W, WIDE, OVER><<<dim3((unsigned)gx, gy), warps * 32, smem, s>>>(g, perCta, preExt, postExt, dw);
   PVGPU_CHECK_LAUNCH("hebbian_dw");
   return PVGPU_OK;
}

template <int FC, bool OVER>
pvgpu_status launch_hebbian_ept(const HGeom &g, const float *preExt, const float *postExt, float *dw, cudaStream_t s) {
   // The fewest weights per lane, for short chains of loads behind each list entry and more warps to
   // hide them, whose warps one pass over the activity serves: in one CTA, or in several where the SMs
   // that would take them have nothing else (57 x 15x70x1 -> 32 features, 9x9 patches, 20 %: one CTA of
   // eight weights a lane 5.8 ms, three of one 1.3).
   const int slabs = (g.patchSize + 31) / 32;
   const int64_t gx = (int64_t)g.nkx * g.nky * ((g.preNf + FC - 1) / FC);
   auto fits = [&](int ept) {
      const int per = 32 / FC * ept;
      return slabs <= per || gx * ((slabs + per - 1) / per) <= pvgpu::num_sms();
   };
   if (slabs <= 16 / FC) return launch_hebbian<1, FC, 16, false, OVER>(g, preExt, postExt, dw, s);
   if (fits(1)) return launch_hebbian<1, FC, 32, false, OVER>(g, preExt, postExt, dw, s);
   if (fits(2)) return launch_hebbian<2, FC, 32, false, OVER>(g, preExt, postExt, dw, s);
   return launch_hebbian<8, FC, 16, false, OVER>(g, preExt, postExt, dw, s);
}

}  // namespace

extern "C" pvgpu_status pvgpu_transpose_weights(const pvgpu_conn_desc *conn, const float *preWeights,
                                                float *postWeights, void *stream) {
   if (!conn || !preWeights || !postWeights) return PVGPU_ERR_BAD_ARG;
   const pvgpu_loc &pre = conn->pre, &post = conn->post;
   if (!pvgpu::loc_valid(pre) || !pvgpu::loc_valid(post)) return PVGPU_ERR_BAD_ARG;
   if (!pvgpu::axis_legal(pre.nx, post.nx, conn->nxp) || !pvgpu::axis_legal(pre.ny, post.ny, conn->nyp))
      return PVGPU_ERR_ILLEGAL_GEOMETRY;
   TGeom g;
   g.nxp = conn->nxp;
   g.nyp = conn->nyp;
   g.nfp = post.nf;
   g.nkx = pre.nx > post.nx ? pre.nx / post.nx : 1;
   g.nky = pre.ny > post.ny ? pre.ny / post.ny : 1;
   g.nkf = pre.nf;
   g.xStride = g.nkx;
   g.yStride = g.nky;
   g.xTStride = post.nx > pre.nx ? post.nx / pre.nx : 1;
   g.yTStride = post.ny > pre.ny ? post.ny / pre.ny : 1;
   g.nxpPost = g.nxp * g.xStride / g.xTStride;
   g.nypPost = g.nyp * g.yStride / g.yTStride;
   g.nkxPost = g.xTStride;
   g.nkyPost = g.yTStride;
   g.nkfPost = post.nf;
   int64_t total = (int64_t)g.nkx * g.nky * g.nkf * g.nxp * g.nyp * g.nfp;
   transpose_kernel<<<(unsigned)((total + 255) / 256), 256, 0, pvgpu::as_stream(stream)>>>(g, preWeights, postWeights);
   PVGPU_CHECK_LAUNCH("transpose_weights");
   return PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_hebbian_dw(const pvgpu_conn_desc *conn, float dWMax, const float *preExt,
                                         const float *postExt, float *dw, void *stream) {
   if (!conn || !preExt || !postExt || !dw) return PVGPU_ERR_BAD_ARG;
   const pvgpu_loc &pre = conn->pre, &post = conn->post;
   if (!pvgpu::loc_valid(pre) || !pvgpu::loc_valid(post) || pre.nbatch != post.nbatch) return PVGPU_ERR_BAD_ARG;
   if (!pvgpu::axis_legal(pre.nx, post.nx, conn->nxp) || !pvgpu::axis_legal(pre.ny, post.ny, conn->nyp))
      return PVGPU_ERR_ILLEGAL_GEOMETRY;
   HGeom g;
   const Loc lpre = pvgpu::to_loc(pre), lpost = pvgpu::to_loc(post);
   g.ax = pvgpu::fast_axis(Axis{pre.nx, post.nx, conn->nxp, pre.halo.lt}, lpre.nxExt());
   g.ay = pvgpu::fast_axis(Axis{pre.ny, post.ny, conn->nyp, pre.halo.dn}, lpre.nyExt());
   g.nPreExt = lpre.numExt();
   g.nPostExt = lpost.numExt();
   g.nb = pre.nbatch;
   g.preNf = pre.nf;
   g.preNxExt = lpre.nxExt();
   g.postNx = post.nx;
   g.postNy = post.ny;
   g.postNf = post.nf;
   g.postNxExt = lpost.nxExt();
   g.postDn = post.halo.dn;
   g.nxp = conn->nxp;
   g.nyp = conn->nyp;
   g.patchSize = conn->nxp * conn->nyp * post.nf;
   g.nkx = pre.nx > post.nx ? pre.nx / post.nx : 1;
   g.nky = pre.ny > post.ny ? pre.ny / post.ny : 1;
   g.dWMax = dWMax;
   cudaStream_t s = pvgpu::as_stream(stream);
   if (g.nPostExt * g.nb > 0x7fffffffLL) return launch_hebbian<4, 1, 16, true>(g, preExt, postExt, dw, s);
   // features per CTA: as many as share a 32-byte sector, fewer while that leaves SMs without a CTA
   int fc = 8;
   while (fc > 1 && ((int64_t)g.nkx * g.nky * ((pre.nf + fc - 1) / fc) < 128 || fc >= 2 * pre.nf)) fc >>= 1;
   const bool over = g.nxp > g.postNx || g.nyp > g.postNy;
   auto launch = [&](auto n) {
      constexpr int FC = decltype(n)::value;
      return over ? launch_hebbian_ept<FC, true>(g, preExt, postExt, dw, s) : launch_hebbian_ept<FC, false>(g, preExt, postExt, dw, s);
   };
   return fc == 8   ? launch(std::integral_constant<int, 8>())
          : fc == 4 ? launch(std::integral_constant<int, 4>())
          : fc == 2 ? launch(std::integral_constant<int, 2>())
                    : launch(std::integral_constant<int, 1>());
}

// ---- MomentumUpdater (weightupdaters/MomentumUpdater.cpp:291-345) ----------------------------
// applyMomentum then prev_dW = dW then HebbianUpdater::updateWeights (W += dW), one thread per
// weight, every operation separately rounded as the reference's loop does.
namespace {
__global__ void momentum_weights_kernel(int64_t n, float dwFactor, float wFactor, float *__restrict__ dw,
                                        float *__restrict__ prevDw, float *__restrict__ w) {
   const float keep = __fadd_rn(1.0f, -dwFactor);
   for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
      float d = __fmul_rn(dw[k], keep);
      d = __fadd_rn(d, __fmul_rn(dwFactor, prevDw[k]));
      const float wk = w[k];
      d = __fadd_rn(d, -__fmul_rn(wFactor, wk));
      dw[k] = d;
      prevDw[k] = d;
      w[k] = __fadd_rn(wk, d);
   }
}
}  // namespace

extern "C" pvgpu_status pvgpu_momentum_factors(char method, float tau, float decay, float dWMax, float *dwFactor,
                                               float *wFactor) {
   if (!dwFactor || !wFactor) return PVGPU_ERR_BAD_ARG;
   switch (method) {
      case 'v':  // viscosity: exp(-1/tau), 0 when tau is 0 (host expf, as the reference)
         *dwFactor = tau != 0.0f ? std::exp(-1.0f / tau) : 0.0f;
         *wFactor = decay;
         return PVGPU_OK;
      case 's':
         *dwFactor = tau;
         *wFactor = decay;
         return PVGPU_OK;
      case 'a':
         *dwFactor = tau;
         *wFactor = decay * dWMax;
         return PVGPU_OK;
      default: return PVGPU_ERR_BAD_ARG;
   }
}

extern "C" pvgpu_status pvgpu_momentum_update_weights(int64_t n, float dwFactor, float wFactor, float *dw,
                                                      float *prevDw, float *w, void *stream) {
   if (n < 0 || (n > 0 && (!dw || !prevDw || !w))) return PVGPU_ERR_BAD_ARG;
   if (n == 0) return PVGPU_OK;
   const int64_t blocks = (n + 255) / 256;
   momentum_weights_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, pvgpu::as_stream(stream)>>>(
         n, dwFactor, wFactor, dw, prevDw, w);
   PVGPU_CHECK_LAUNCH("momentum_update_weights");
   return PVGPU_OK;
}
