// lca_solver_fp32.cu -- the plain FP32 form of the batched LCA solver: FP32 SIMT GEMMs (fp32_gemm.cuh)
// and FP32 activity.  It is the baseline the BF16 tensor-core form is measured against.
//
// Three kernels per timestep, each over the whole batch:
//   recon   D[pos][k] = sum_f A[pos][f] W[f][k], k = (ky*P + kx)*C + c;
//   fold    residual r = x - sum of the patches of D that cover a pixel, positions in ascending
//           (y, x) order, into the padded layout that the BF16 form's kernel R writes (zero border);
//   drive   G[pos][f] = sum_k r[window of pos][k] W[f][k], the windows read in place from the padded
//           residual, and the LCA update of those neurons as the GEMM's epilogue.
//
// 32 images of 32x32x3, 512 features: 108 us a timestep (48 + 5 + 55), against 237 us with a CTA per 128 positions for
// the reconstruction (64 of them, 145 us) and residual windows rebuilt by every feature tile's CTA
// (93 us).
#include "fp32_gemm.cuh"
#include "lca_common.cuh"

namespace {

using pvgpu::LcaGeom;

struct ReconProblem {
   int64_t M;
   int N, K, stride;  // K = stride = F
   int64_t sy;
   const float *a, *Wt;
   float *D;
   struct At {};
   struct Old {};
   __device__ __forceinline__ At begin(int, int64_t) const { return At(); }
   __device__ __forceinline__ void row(const At &, int, int64_t m0, int i, int64_t *base, int64_t *out) const {
      *base = (m0 + i) * K;
      *out = (m0 + i) * N;
   }
   __device__ __forceinline__ const float *b(int) const { return Wt; }
   __device__ __forceinline__ Old old(int64_t, int) const { return Old(); }
   __device__ __forceinline__ void store(int64_t out, int n, float v, Old) const { D[out + n] = v; }
};

// SIMPLE: no ceiling and no width (LcaGeom::simple), A = V < VThresh ? AMin : V - AShift
template <bool SIMPLE>
struct DriveProblem {
   LcaGeom g;
   int C, S, RP, padPerImage;
   int64_t M;
   int N, K, stride;
   int64_t sy;
   const float *a, *W;
   float *V, *A32;
   struct At {};
   using Old = float;
   __device__ __forceinline__ At begin(int, int64_t) const { return At(); }
   __device__ __forceinline__ void row(const At &, int, int64_t m0, int i, int64_t *base, int64_t *out) const {
      const uint32_t m = (uint32_t)(m0 + i), b = m / (uint32_t)g.Npos, pos = m - b * g.Npos;
      const uint32_t y = pos / (uint32_t)g.v1Nx, x = pos - y * g.v1Nx;
      *base = (int64_t)b * padPerImage + (int64_t)(S * y) * RP + S * x * C;
      *out = m;
   }
   __device__ __forceinline__ const float *b(int) const { return W; }
   // v_index of position row m (m = b * Npos + pos, Npos a multiple of 128)
   __device__ __forceinline__ size_t v_at(int64_t m, int f) const {
      const int r = (int)(m & 127);
      return ((size_t)(m >> 7) * (g.F >> 6) + (f >> 6)) * 8192 + ((f >> 5) & 1) * 4096 + r * 32 +
             ((((f >> 2) & 7) ^ (r & 7)) << 2) + (f & 3);
   }
   __device__ __forceinline__ float old(int64_t m, int f) const { return V[v_at(m, f)]; }
   __device__ __forceinline__ float threshold(float v) const {
      if (SIMPLE) return v < g.VThresh ? g.AMin : __fadd_rn(v, -g.AShift);
      return pvgpu::lca_thresh(v, g);
   }
   // HyPerLCAInternalStateBuffer.kpp:52-61 and the threshold, rounded as the CPU path rounds
   __device__ __forceinline__ void store(int64_t m, int f, float drive, float vo) const {
      const float ao = threshold(vo);
      const float vn = __fadd_rn(__fmul_rn(g.e, vo), __fmul_rn(__fadd_rn(1.0f, -g.e), __fadd_rn(drive, __fmul_rn(g.si, ao))));
      V[v_at(m, f)] = vn;
      A32[(size_t)m * g.F + f] = threshold(vn);
   }
};

// One thread per value of the padded residual.  Every pixel is covered by at most (P/S)^2 positions;
// their loads are independent and summed in order.
template <int S, int P, int C>
__global__ void __launch_bounds__(128) fold_residual_kernel(LcaGeom g, int rowsPad, int RP,
                                                                 const float *__restrict__ x,
                                                                 const float *__restrict__ D,
                                                                 float *__restrict__ rpad, float *__restrict__ recOut) {
   constexpr int KP = P * P * C, E = (P - S) / 2, Q = P / S;
   const int yp = blockIdx.y, b = blockIdx.x;
   const int col = blockIdx.z * blockDim.x + threadIdx.x;
   if (col >= RP) return;
   const int iy = yp - E, j = col - E * C, ix = j / C, c = j - ix * C;
   float r = 0.0f;
   if (iy >= 0 && iy < g.inNy && j >= 0 && ix < g.inNx) {
      // the last position covering the pixel, and the tap there; earlier ones are S taps further on
      const int py1 = (iy + E) / S, px1 = (ix + E) / S, ky1 = iy + E - S * py1, kx1 = ix + E - S * px1;
      const float *d = D + (size_t)b * g.Npos * KP;
      float t[Q][Q];
#pragma unroll
      for (int qy = 0; qy < Q; qy++)
#pragma unroll
         for (int qx = 0; qx < Q; qx++) {
            const int py = py1 - (Q - 1 - qy), px = px1 - (Q - 1 - qx);
            const int k = ((ky1 + S * (Q - 1 - qy)) * P + kx1 + S * (Q - 1 - qx)) * C + c;
            t[qy][qx] = py >= 0 && py < g.v1Ny && px >= 0 && px < g.v1Nx
                              ? __ldg(d + (size_t)(py * g.v1Nx + px) * KP + k)
                              : 0.0f;
         }
      float rec = 0.0f;
#pragma unroll
      for (int qy = 0; qy < Q; qy++)
#pragma unroll
         for (int qx = 0; qx < Q; qx++) rec += t[qy][qx];
      const size_t at = ((size_t)b * g.inNy + iy) * g.inNx * C + j;
      r = x[at] - rec;
      if (recOut) recOut[at] = rec;
   }
   rpad[((size_t)b * rowsPad + yp) * RP + col] = r;
}

template <int S, int P, int C>
pvgpu_status step(const LcaGeom &g, const float *x, const float *W32, const float *Wt32, float *D, int imagesPerD, float *rpad,
                  float *rec, float *V, float *A32, cudaStream_t st, cudaEvent_t mid) {
   constexpr int KP = P * P * C, E = (P - S) / 2;
   const int64_t M = (int64_t)g.nb * g.Npos;
   const int RP = ((g.inNx + 2 * E) * C + 3) & ~3, rowsPad = g.inNy + 2 * E;
   const size_t nPix = (size_t)g.inNx * g.inNy * C;
   if (M > 0x7fffffff) return PVGPU_ERR_UNSUPPORTED_SHAPE;
   for (int b0 = 0; b0 < g.nb; b0 += imagesPerD) {  // as many images as D holds
      LcaGeom part = g;
      part.nb = std::min(imagesPerD, g.nb - b0);
      const ReconProblem rp = {(int64_t)part.nb * g.Npos, KP, g.F, g.F, 0, A32 + (size_t)b0 * g.Npos * g.F, Wt32, D};
      const pvgpu_status r = pvgpu::fp32_gemm::run<4>(rp, 1, st, "lca32 recon");
      if (r != PVGPU_OK) return r;
      const dim3 fg(part.nb, rowsPad, (RP + 127) / 128);
      fold_residual_kernel<S, P, C><<<fg, 128, 0, st>>>(part, rowsPad, RP, x + b0 * nPix, D, rpad + (size_t)b0 * rowsPad * RP,
                                                       rec ? rec + b0 * nPix : nullptr);
      PVGPU_CHECK_LAUNCH("lca32 fold");
   }
   if (mid) cudaEventRecord(mid, st);
   // windows start at multiples of S * C floats, their rows of P * C values RP (a multiple of 4) apart
   constexpr int VW = S * C % 4 == 0 ? 4 : 2;
   if (g.simple) {
      const DriveProblem<true> dp = {g, C, S, RP, rowsPad * RP, M, g.F, KP, P * C, RP, rpad, W32, V, A32};
      return pvgpu::fp32_gemm::run<VW>(dp, 1, st, "lca32 drive");
   }
   const DriveProblem<false> dp = {g, C, S, RP, rowsPad * RP, M, g.F, KP, P * C, RP, rpad, W32, V, A32};
   return pvgpu::fp32_gemm::run<VW>(dp, 1, st, "lca32 drive");
}

}  // namespace

namespace pvgpu {

// D: room for the reconstruction GEMM of imagesPerD images; rec: the step's reconstruction W^T a (what the energy
// probe subtracts from the image it is given), or null
pvgpu_status lca_fp32_step(int S, int P, int C, const LcaGeom &g, const float *x, const float *W32, const float *Wt32,
                           float *D, int imagesPerD, float *rpad, float *rec, float *V, float *A32, cudaStream_t st,
                           cudaEvent_t mid) {
   if (S == 2 && P == 8 && C == 1) return step<2, 8, 1>(g, x, W32, Wt32, D, imagesPerD, rpad, rec, V, A32, st, mid);
   if (S == 2 && P == 8 && C == 3) return step<2, 8, 3>(g, x, W32, Wt32, D, imagesPerD, rpad, rec, V, A32, st, mid);
   if (S == 4 && P == 16 && C == 1) return step<4, 16, 1>(g, x, W32, Wt32, D, imagesPerD, rpad, rec, V, A32, st, mid);
   return PVGPU_ERR_UNSUPPORTED_SHAPE;
}

}  // namespace pvgpu
