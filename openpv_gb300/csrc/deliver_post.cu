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
#include "fp32_gemm.cuh"

namespace {

using pvgpu::Axis;
using pvgpu::Loc;

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

// FAST mode: the delivery as a problem of fp32_gemm.cuh, phase = kernel phase.
struct PostProblem {
   PostGeom g;
   int64_t M;  // rows per phase
   int N, K, stride;
   int64_t sy;
   const float *a;
   const float *W;
   float *gsyn;
   struct At {
      int b0, r0, nxPh, perImg;
   };
   using Old = float;
   __device__ __forceinline__ At begin(int, int64_t m0) const {
      At t;
      t.nxPh = g.tgt.nx / g.nkx;
      t.perImg = t.nxPh * (g.tgt.ny / g.nky);
      t.b0 = (int)(m0 / t.perImg);
      t.r0 = (int)(m0 - (int64_t)t.b0 * t.perImg);
      return t;
   }
   __device__ __forceinline__ void row(const At &t, int phase, int64_t, int i, int64_t *base, int64_t *out) const {
      const uint32_t q = (uint32_t)t.r0 + i, db = q / (uint32_t)t.perImg, p = q - db * t.perImg;
      const uint32_t yp = p / (uint32_t)t.nxPh;
      const int x = phase % g.nkx + g.nkx * (int)(p - yp * t.nxPh), y = phase / g.nkx + g.nky * (int)yp;
      *base = (int64_t)(t.b0 + db) * g.src.numExt() + src_start(g, x, y);
      *out = (int64_t)(t.b0 + db) * g.tgt.numRes() + ((int64_t)y * g.tgt.nx + x) * g.tgt.nf;
   }
   __device__ __forceinline__ const float *b(int phase) const {
      return W + (size_t)post_kernel(g, phase % g.nkx, phase / g.nkx, 0) * K;
   }
   __device__ __forceinline__ float old(int64_t out, int n) const { return gsyn[out + n]; }
   __device__ __forceinline__ void store(int64_t out, int n, float v, float o) const { gsyn[out + n] = fmaf(g.dtf, v, o); }
};

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
   const PostProblem p = {g, M, g.nkf, g.K, g.numPerStride, g.sy, aExt, postWeights, gsyn};
   const int phases = g.nkx * g.nky;
   if (aligned(4)) return pvgpu::fp32_gemm::run<4>(p, phases, s, "deliver_post");
   if (aligned(2)) return pvgpu::fp32_gemm::run<2>(p, phases, s, "deliver_post");
   return pvgpu::fp32_gemm::run<1>(p, phases, s, "deliver_post");
}
