// lca_grad.cu -- the gradient of unrolled LCA (differentiable dictionary learning) on the device,
// behind the C ABI: L(W) = 0.5 ||x - W^T a_T||^2 + lambda ||a_T||_1 after T LCA timesteps from
// V = 0, with the soft threshold a = T(V) = max(V - VThresh, 0) (ANNActivityBuffer with AMin = 0,
// AShift = VThresh, VWidth = 0), V' = e V + (1 - e)(W r + a), r = x - W^T a, e = exp(-dt/tau)
// (HyPerLCAInternalStateBuffer.kpp:18-63 with selfInteract), and dL/dW.  The reference learns its
// dictionaries with the Hebbian rule (weightupdaters/HebbianUpdater.cpp:476-629): the gradient of
// the loss of a fixed activity a is minus that update (dWMax = 1); here the whole unrolled solve is
// differentiated, with a checkpoint every K timesteps.
//
// Both deliveries are GEMMs over the im2col'd operands.  Row-major, M = nbatch * positions:
//   recon:  D[M][KP] = A[M][F] . W[F][KP],  y = fold(D)   (patch k of position p adds to pixel
//           (S*py - E + ky, S*px - E + kx, c), E = (P - S) / 2 -- PatchGeometry's one-to-many start)
//   drive:  R[M][KP] = im2col(x - y),  Z[M][F] = R . W^T
// and their adjoints (the transpose delivery and the pre (x) post-error correlation):
//   gR = (1 - e) g . W,  gr = fold(gR),  gD = -im2col(gr),  gA = gD . W^T,
//   g <- e g + [V >= VThresh] ((1 - e) g + gA),   dW += (1 - e) g^T R + A^T gD
// where g = dL/dV of the later step; on the library path below the correlations of a whole segment run as two
// GEMMs over all its steps' positions (K = steps x positions).  The final loss seeds g_T = [V_T >= VThresh](-Z_T + lambda [a_T > 0])
// and dW = -A_T^T R_T.
//
// Where v1Nf and KP are multiples of 8 the GEMMs are the split-plane ones of split_gemm.cuh (tcgen05, six
// BF16 plane products per FP32 product) and the passes between them are folded in: a timestep is
//   recon GEMM (planes of a x planes of W^T -> D),
//   fold_im2col (residual windows gathered from D, their im2col written as planes),
//   drive GEMM, whose epilogue updates V and writes the planes of the new activity,
// and an adjoint step the same three plus the correlations of that step's positions, added into one
// partial dW per range of positions.  Measured for 32 x 64x64x1 -> 16x16x256, 100 steps: 10.7 ms against
// 16.8 ms with library GEMMs (14.4 us each, nine plane products) and separate fold, im2col and update
// passes (31 us a step); dW's median error against FP64 over 40 inputs 2.1e-7 against 6.0e-7.  The last
// segment's states are kept from the forward pass.
//
// Other sizes, and runs whose buffers fit in no other way, go through cuBLAS in FP32 emulated on the BF16 tensor cores
// (CUBLAS_COMPUTE_32F_EMULATED_16BFX9: each operand split in three BF16 parts, FP32 accuracy), or
// in plain FP32 where that mode is refused.  cuBLAS is loaded at the first create that needs it.
// Everything else -- fold, im2col, the update and its adjoint,
// the threshold mask, the loss -- is the kernels below.  A run is one CUDA graph (captured once
// per set of pointers, replayed on the caller's stream).
#include "split_gemm.cuh"

#include <cublas_v2.h>
#include <dlfcn.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

namespace {

constexpr int kThreads = 256;

struct Geo {
   int nb, iny, inx, C, vy, vx, F, P, S, E, KP, Np;
   int64_t M;  // nb * Np
};

__device__ __forceinline__ float soft(float v, float vt) { return v >= vt ? v - vt : 0.0f; }

__global__ void threshold_kernel(int64_t n, float vt, const float *__restrict__ v, float *__restrict__ a) {
   for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
      a[i] = soft(v[i], vt);
}

// out[b][iy][ix][c] = (x ? x : 0) + sign * sum over the positions whose patch covers the pixel of
// D[b, p][k] (positions ascending in y, then x: a fixed order, no atomics).
__global__ void fold_kernel(Geo g, const float *__restrict__ D, const float *__restrict__ x, float sign,
                            float *__restrict__ out) {
   const int n = g.nb * g.iny * g.inx * g.C;
   for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const int c = i % g.C;
      const int ix = (i / g.C) % g.inx;
      const int iy = (i / (g.C * g.inx)) % g.iny;
      const int b = i / (g.C * g.inx * g.iny);
      // positions py with 0 <= iy - (S*py - E) < P
      const int pyLo = max(0, (iy + g.E - g.P + g.S) / g.S), pyHi = min(g.vy - 1, (iy + g.E) / g.S);
      const int pxLo = max(0, (ix + g.E - g.P + g.S) / g.S), pxHi = min(g.vx - 1, (ix + g.E) / g.S);
      float s = 0.0f;
      for (int py = pyLo; py <= pyHi; py++) {
         const int ky = iy - (g.S * py - g.E);
         for (int px = pxLo; px <= pxHi; px++) {
            const int kx = ix - (g.S * px - g.E);
            s += D[((int64_t)b * g.Np + py * g.vx + px) * g.KP + (ky * g.P + kx) * g.C + c];
         }
      }
      out[i] = (x ? x[i] : 0.0f) + sign * s;
   }
}

// R[b, p][k] = sign * img[b][S*py - E + ky][S*px - E + kx][c], 0 outside the image.  One block
// per row (b, p); the threads walk k.
__global__ void im2col_kernel(Geo g, const float *__restrict__ img, float sign, float *__restrict__ R) {
   const int row = blockIdx.x;
   const int p = row % g.Np, b = row / g.Np;
   const int iy0 = g.S * (p / g.vx) - g.E, ix0 = g.S * (p % g.vx) - g.E;
   const float *ib = img + (size_t)b * g.iny * g.inx * g.C;
   float *out = R + (size_t)row * g.KP;
   const int PC = g.P * g.C;
   for (int k = threadIdx.x; k < g.KP; k += blockDim.x) {
      const int ky = k / PC, r = k - ky * PC, kx = r / g.C, c = r - kx * g.C;
      const int iy = iy0 + ky, ix = ix0 + kx;
      float v = 0.0f;
      if (iy >= 0 && iy < g.iny && ix >= 0 && ix < g.inx) v = ib[(iy * g.inx + ix) * g.C + c];
      out[k] = sign * v;
   }
}

// WT[k][f] = W[f][k] (the weights as the K-major operand of the reconstruction GEMM).
__global__ void transpose_kernel(int F, int KP, const float *__restrict__ W, float *__restrict__ WT) {
   __shared__ float tile[32][33];
   const int f0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
   for (int j = threadIdx.y; j < 32; j += blockDim.y)
      if (f0 + j < F && k0 + threadIdx.x < KP) tile[j][threadIdx.x] = W[(size_t)(f0 + j) * KP + k0 + threadIdx.x];
   __syncthreads();
   for (int j = threadIdx.y; j < 32; j += blockDim.y)
      if (k0 + j < KP && f0 + threadIdx.x < F) WT[(size_t)(k0 + j) * F + f0 + threadIdx.x] = tile[threadIdx.x][j];
}

// V' = e V + (1 - e)(Z + A), A' = T(V')
__global__ void update_kernel(int n, float e, float vt, const float *__restrict__ v, const float *__restrict__ a,
                              const float *__restrict__ z, float *__restrict__ vOut, float *__restrict__ aOut) {
   const float om = 1.0f - e;
   for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const float vn = e * v[i] + om * (z[i] + a[i]);
      vOut[i] = vn;
      aOut[i] = soft(vn, vt);
   }
}

// gOut = e g + [V >= vt] ((1 - e) g + gA)
__global__ void adjoint_update_kernel(int n, float e, float vt, const float *__restrict__ v,
                                      const float *__restrict__ gA, const float *__restrict__ g,
                                      float *__restrict__ gOut) {
   const float om = 1.0f - e;
   for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const float gv = g[i];
      gOut[i] = e * gv + (v[i] >= vt ? om * gv + gA[i] : 0.0f);
   }
}

// g_T = [V_T >= vt] (lambda [A_T > 0] - Z_T)
__global__ void seed_kernel(int64_t n, float vt, float lambda, const float *__restrict__ v,
                            const float *__restrict__ a, const float *__restrict__ z, float *__restrict__ gV) {
   for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
      gV[i] = v[i] >= vt ? (a[i] > 0.0f ? lambda : 0.0f) - z[i] : 0.0f;
}

// Per-block partial sums of 0.5 r^2 (r: nr values) + lambda |a| (a: na values), in FP64; then
// one block adds the partials in block order (deterministic).
constexpr int kLossBlocks = 256;
__global__ void loss_partial_kernel(int64_t nr, const float *__restrict__ r, int64_t na, const float *__restrict__ a,
                                    double lambda, double *__restrict__ partial) {
   double s = 0.0;
   for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nr; i += (int64_t)gridDim.x * blockDim.x)
      s += 0.5 * (double)r[i] * (double)r[i];
   for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < na; i += (int64_t)gridDim.x * blockDim.x)
      s += lambda * fabs((double)a[i]);
   __shared__ double red[kThreads];
   red[threadIdx.x] = s;
   __syncthreads();
   for (int w = kThreads / 2; w > 0; w >>= 1) {
      if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
      __syncthreads();
   }
   if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void loss_final_kernel(const double *__restrict__ partial, int n, double *__restrict__ out) {
   if (threadIdx.x == 0 && blockIdx.x == 0) {
      double s = 0.0;
      for (int i = 0; i < n; i++) s += partial[i];
      *out = s;
   }
}

// ---- the split-plane path ------------------------------------------------------------------
using pvgpu::split::bf16;
using pvgpu::split::split2;
using pvgpu::split::split_store4;
using pvgpu::split::split_store8;
using pvgpu::tc::griddep_launch_dependents;
using pvgpu::tc::griddep_wait;

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, const float4 &v) { *reinterpret_cast<float4 *>(p) = v; }
template <typename F>
__device__ __forceinline__ float4 each4(const float4 &a, const float4 &b, F f) {
   return make_float4(f(a.x, b.x), f(a.y, b.y), f(a.z, b.z), f(a.w, b.w));
}

// The GEMMs' epilogues, four neighbouring values at offset `at` of a [rows][columns] matrix.
struct EpiStore {
   float alpha;
   float *D;
   struct Regs {};
   __device__ __forceinline__ void load(Regs &, size_t) const {}
   __device__ __forceinline__ void late(Regs &, size_t) const {}
   __device__ __forceinline__ void finish(const Regs &, const float4 &z, size_t at) const {
      st4(D + at, make_float4(alpha * z.x, alpha * z.y, alpha * z.z, alpha * z.w));
   }
};

// The forward state is held in two parts, V = hi + lo (lo a BF16 below half an ulp of hi: 32 bits of V in
// all), because the 2^-24 that each of the T updates would round off V decides whether values near the
// threshold lie above it, and every value that falls on the other side of it than in exact arithmetic
// shows in dW.  hi >= vt exactly where V >= vt; below: the largest value less than vt.
__device__ __forceinline__ float soft2(float hi, float lo, float vt) { return hi >= vt ? __fadd_rn(__fadd_rn(hi, -vt), lo) : 0.0f; }

// V' = e V + (1 - e)(Z + T(V)) = V + (1 - e)(Z - min(V, vt)), the sum compensated
__device__ __forceinline__ void step2(float &hi, float &lo, float z, float om, float vt, float below) {
   const float d = __fmul_rn(om, __fadd_rn(z, -fminf(hi, vt)));
   const float s = __fadd_rn(hi, d), t = __fadd_rn(s, -hi);
   const float r = __fadd_rn(__fadd_rn(__fadd_rn(hi, -__fadd_rn(s, -t)), __fadd_rn(d, -t)), lo);
   hi = __fadd_rn(s, r);
   lo = __fadd_rn(r, -__fadd_rn(hi, -s));
   if (hi == vt && lo < 0.0f) {
      hi = below;
      lo = __fadd_rn(lo, __fadd_rn(vt, -below));
   }
}

__device__ __forceinline__ float bf16_at(const uint2 &u, int i) {
   const uint32_t w = i < 2 ? u.x : u.y;
   return __uint_as_float(i & 1 ? w & 0xffff0000u : w << 16);
}
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
   return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(b)) << 16);
}

// V' and the planes of A' = T(V')
struct EpiForward {
   float om, vt, below;
   const float *v;
   const bf16 *vLo;
   float *vOut;
   bf16 *vLoOut;
   bf16 *a;
   size_t plane;
   struct Regs {
      float4 v;
      uint2 lo;
   };
   __device__ __forceinline__ void load(Regs &r, size_t at) const { r.v = ld4(v + at); }
   __device__ __forceinline__ void late(Regs &r, size_t at) const { r.lo = *reinterpret_cast<const uint2 *>(vLo + at); }
   __device__ __forceinline__ void finish(const Regs &r, const float4 &z, size_t at) const {
      float hi[4] = {r.v.x, r.v.y, r.v.z, r.v.w}, lo[4], x[4];
      const float zi[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
         lo[i] = bf16_at(r.lo, i);
         step2(hi[i], lo[i], zi[i], om, vt, below);
         x[i] = soft2(hi[i], lo[i], vt);
      }
      st4(vOut + at, make_float4(hi[0], hi[1], hi[2], hi[3]));
      *reinterpret_cast<uint2 *>(vLoOut + at) = make_uint2(bf16_pair(lo[0], lo[1]), bf16_pair(lo[2], lo[3]));
      split_store4(make_float4(x[0], x[1], x[2], x[3]), a + at, plane);
   }
};

// g <- e g + [V >= vt]((1 - e) g + gA), in place, and its planes
struct EpiAdjoint {
   float e, vt;
   const float *v;
   float *g;
   bf16 *gp;
   size_t plane;
   struct Regs {
      float4 g;
      bool on[4];
   };
   __device__ __forceinline__ void load(Regs &r, size_t at) const {
      r.g = ld4(g + at);
      const float4 x = ld4(v + at);
      r.on[0] = x.x >= vt;
      r.on[1] = x.y >= vt;
      r.on[2] = x.z >= vt;
      r.on[3] = x.w >= vt;
   }
   __device__ __forceinline__ void late(Regs &, size_t) const {}
   __device__ __forceinline__ void finish(const Regs &r, const float4 &z, size_t at) const {
      const float om = 1.0f - e;
      auto next = [&](float gi, float zi, bool on) { return e * gi + (on ? om * gi + zi : 0.0f); };
      const float4 n = make_float4(next(r.g.x, z.x, r.on[0]), next(r.g.y, z.y, r.on[1]), next(r.g.z, z.z, r.on[2]),
                                   next(r.g.w, z.w, r.on[3]));
      st4(g + at, n);
      split_store4(n, gp + at, plane);
   }
};

// g_T = [V_T >= vt](lambda [A_T > 0] - Z_T) and its planes
struct EpiSeed {
   float vt, lambda;
   const float *v;
   float *g;
   bf16 *gp;
   size_t plane;
   struct Regs {
      float4 v;
   };
   __device__ __forceinline__ void load(Regs &r, size_t at) const { r.v = ld4(v + at); }
   __device__ __forceinline__ void late(Regs &, size_t) const {}
   __device__ __forceinline__ void finish(const Regs &r, const float4 &z, size_t at) const {
      const float4 n = each4(
            r.v, z, [&](float vi, float zi) { return vi >= vt ? (soft(vi, vt) > 0.0f ? lambda : 0.0f) - zi : 0.0f; });
      st4(g + at, n);
      split_store4(n, gp + at, plane);
   }
};

// Planes of W [F][KP] and of its transpose [KP][F].
__global__ void split_weights_kernel(int F, int KP, const float *__restrict__ W, bf16 *__restrict__ Wp,
                                     bf16 *__restrict__ WTp) {
   griddep_launch_dependents();
   griddep_wait();
   const size_t n = (size_t)F * KP;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
      const size_t f = i / KP, k = i - f * KP;
      uint32_t p[3];
      split2(W[i], 0.0f, p);
#pragma unroll
      for (int q = 0; q < 3; q++) Wp[q * n + i] = WTp[q * n + k * F + f] = __ushort_as_bfloat16((unsigned short)p[q]);
   }
}

// Planes of T(V), eight values per thread.
__global__ void split_activity_kernel(int64_t n8, float vt, const float *__restrict__ v, const bf16 *__restrict__ vLo,
                                      bf16 *__restrict__ a, size_t plane) {
   griddep_launch_dependents();
   griddep_wait();
   for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n8; i += (int64_t)gridDim.x * blockDim.x) {
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; q++) x[q] = soft2(v[i * 8 + q], __bfloat162float(vLo[i * 8 + q]), vt);
      split_store8(x, a + i * 8, plane);
   }
}

// The residual windows of BR rows of positions and their im2col, in one pass: window = base * x +
// signImg * fold(D), each pixel gathered from the positions that cover it in ascending (y, x) order (as
// fold_kernel), staged in shared memory, then every position's patch written as planes times signOut.
// Neighbouring bands gather the P - S rows they share twice, from L2; in exchange the image and the
// FP32 im2col never go to memory and the pass is one launch (23 us for the two before, 11 now).
// SS, PP, CC: the geometry as constants, or 0.  Any other geometry takes xPer positions of a row at a time: its
// gather is a chain of loads per pixel, so where bands are few and patches large a row is divided (3 x 56x76x3 ->
// 14x19x8, 16x16 patches, 16 steps: 2.49 ms with whole rows, now 1.65; the library path 1.25).
constexpr int kMaxBandRows = 2, kFoldThreads = 384;
template <int SS, int PP, int CC>
__global__ void __launch_bounds__(kFoldThreads, 2) fold_im2col_kernel(Geo g, int bandRows, int xPer, const float *__restrict__ D,
                                                                      const float *__restrict__ x, float signImg, float signOut,
                                                                      bf16 *__restrict__ out, size_t plane) {
   extern __shared__ __align__(16) float win[];
   const int S = SS ? SS : g.S, P = PP ? PP : g.P, C = CC ? CC : g.C, E = (P - S) / 2, PC = P * C, KP = P * PC;
   const int bands = (g.vy + bandRows - 1) / bandRows;
   const int b = blockIdx.x / bands, y0 = (blockIdx.x % bands) * bandRows, rows = min(bandRows, g.vy - y0);
   const int x0 = SS ? 0 : blockIdx.y * xPer, xn = SS ? g.vx : min(xPer, g.vx - x0);  // positions of a row
   const int WP = ((SS ? g.inx + 2 * E : S * (xn - 1) + P) * C + 3) & ~3, WR = S * (rows - 1) + P;
   griddep_launch_dependents();
   griddep_wait();
   const float *Db = D + (size_t)b * g.Np * KP;
   if constexpr (SS != 0) {
      // in groups of S pixels that the same positions cover, whose S * C values are neighbours in D: all of
      // a group's loads are independent vector loads
      constexpr int Q = PP / (SS ? SS : 1), G = SS * CC, VW = G % 4 == 0 ? 4 : 2;
      const int groups = WP / G + (WP % G != 0);
      for (int i = threadIdx.x; i < WR * groups; i += blockDim.x) {
         const int yy = i / groups, q = i - yy * groups;
         const int v = S * y0 + yy, iy = v - E;  // v: row in the zero-bordered image
         float sum[G];
#pragma unroll
         for (int j = 0; j < G; j++) sum[j] = 0.0f;
         // positions in ascending (y, x) order; the loads of up to two rows of them in flight
#pragma unroll 2
         for (int ty = Q - 1; ty >= 0; ty--) {
            float t[Q][G];
#pragma unroll
            for (int tx = 0; tx < Q; tx++) {
               const int py = v / S - ty, px = q - tx;
               const bool on = py >= 0 && py < g.vy && px >= 0 && px < g.vx && iy >= 0 && iy < g.iny;
               const float *d = Db + ((size_t)py * g.vx + px) * KP + ((v % S + S * ty) * P + S * tx) * C;
#pragma unroll
               for (int j = 0; j < G; j += VW) {
                  if constexpr (VW == 4) {
                     const float4 f = on ? __ldg(reinterpret_cast<const float4 *>(d + j)) : make_float4(0, 0, 0, 0);
                     t[tx][j] = f.x;
                     t[tx][j + 1] = f.y;
                     t[tx][j + 2] = f.z;
                     t[tx][j + 3] = f.w;
                  } else {
                     const float2 f = on ? __ldg(reinterpret_cast<const float2 *>(d + j)) : make_float2(0, 0);
                     t[tx][j] = f.x;
                     t[tx][j + 1] = f.y;
                  }
               }
            }
#pragma unroll
            for (int tx = Q - 1; tx >= 0; tx--)
#pragma unroll
               for (int j = 0; j < G; j++) sum[j] += t[tx][j];
         }
#pragma unroll
         for (int j = 0; j < G; j++) {
            const int col = q * G + j, xc = col - E * C;  // xc: value in the image's row
            const bool in = iy >= 0 && iy < g.iny && xc >= 0 && xc < g.inx * C;
            if (col < WP)
               win[yy * WP + col] = in ? (x ? x[((size_t)b * g.iny + iy) * g.inx * C + xc] : 0.0f) + signImg * sum[j] : 0.0f;
         }
      }
   } else {
      for (int i = threadIdx.x; i < WR * WP; i += blockDim.x) {
         const int yy = i / WP, col = i - yy * WP;
         const int iy = S * y0 - E + yy, j = col + (S * x0 - E) * C;
         float r = 0.0f;
         if (iy >= 0 && iy < g.iny && j >= 0 && j < g.inx * C) {
            const int ix = j / C, c = j - ix * C;
            const int pyLo = max(0, (iy + E - P + S) / S), pyHi = min(g.vy - 1, (iy + E) / S);
            const int pxLo = max(0, (ix + E - P + S) / S), pxHi = min(g.vx - 1, (ix + E) / S);
            float s = 0.0f;
            for (int py = pyLo; py <= pyHi; py++) {
               const float *d = Db + ((size_t)py * g.vx + pxLo) * KP + ((iy + E - S * py) * P + ix + E - S * pxLo) * C + c;
#pragma unroll 4
               for (int px = pxLo; px <= pxHi; px++, d += KP - S * C) s += __ldg(d);
            }
            r = (x ? x[((size_t)b * g.iny + iy) * g.inx * C + j] : 0.0f) + signImg * s;
         }
         win[i] = r;
      }
   }
   __syncthreads();
   const int k8 = KP / 8, items = rows * xn * k8;
   bf16 *o = out + ((size_t)b * g.Np + (size_t)y0 * g.vx + x0) * KP;
   for (int i = threadIdx.x; i < items; i += blockDim.x) {
      const int p = i / k8, k = (i - p * k8) * 8, yl = p / xn, xl = p - yl * xn;
      const float *w = win + (S * yl) * WP + S * xl * C;
      int ky = k / PC, rem = k - ky * PC;
      float v[8];
      if constexpr (SS * CC % 4 == 0 && SS != 0 && PP * CC % 8 == 0) {  // two aligned quads of one patch row
         const float4 *w4 = reinterpret_cast<const float4 *>(w + ky * WP + rem);
#pragma unroll
         for (int q = 0; q < 2; q++) {
            v[4 * q] = signOut * w4[q].x;
            v[4 * q + 1] = signOut * w4[q].y;
            v[4 * q + 2] = signOut * w4[q].z;
            v[4 * q + 3] = signOut * w4[q].w;
         }
      } else {
#pragma unroll
         for (int q = 0; q < 8; q++) {
            v[q] = signOut * w[ky * WP + rem];
            if (++rem == PC) {
               rem = 0;
               ky++;
            }
         }
      }
      split_store8(v, o + (size_t)(yl * g.vx + xl) * KP + k, plane);
   }
}

// dW = om * sum of the first pair's partial correlations + sum of the second's, splits in order; NaN (and the
// loss) if a bounded device wait of the run's GEMMs gave up.
__global__ void corr_sum_kernel(int n, int splits, float om, const float *__restrict__ P, const int *__restrict__ err,
                                float *__restrict__ dW, double *__restrict__ loss) {
   griddep_launch_dependents();
   griddep_wait();
   const bool bad = *err != 0;
   if (bad && blockIdx.x == 0 && threadIdx.x == 0) *loss = nan("");
   for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      float s[2] = {0.0f, 0.0f};
      for (int h = 0; h < 2; h++)
         for (int k = 0; k < splits; k++) s[h] += P[((size_t)h * splits + k) * n + i];
      dW[i] = bad ? nanf("") : om * s[0] + s[1];
   }
}

// The pipeline without its copies: nothing ever arrives.
__global__ void __launch_bounds__(pvgpu::split::kThreads, 1) gemm_expiry_kernel(int chunks, int *err, long long *out) {
   using namespace pvgpu::split;
   extern __shared__ uint8_t smem_raw[];
   __shared__ __align__(8) uint64_t bars[bars_of<kMaxStages>()];
   __shared__ uint32_t tmemBase;
   const uint64_t t0 = global_ns();
   pipeline<32, stages_of(32)>(
         align1024(smem_raw), 3 * (kPlaneA + 32 * 128), chunks, err, &tmemBase, bars, [](int, uint8_t *, uint64_t *) {},
         [](uint32_t, int, int, uint32_t, uint32_t) {}, [] {}, [] {}, [&](const float *, int) { out[1] = 1; });
   if (threadIdx.x == 0) out[0] = (long long)(global_ns() - t0);
}

// ---- cuBLAS, loaded at first use --------------------------------------------------------------
struct Blas {
   void *so = nullptr;
   cublasStatus_t (*create)(cublasHandle_t *) = nullptr;
   cublasStatus_t (*destroy)(cublasHandle_t) = nullptr;
   cublasStatus_t (*setStream)(cublasHandle_t, cudaStream_t) = nullptr;
   cublasStatus_t (*setWorkspace)(cublasHandle_t, void *, size_t) = nullptr;
   cublasStatus_t (*gemmEx)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int, const void *,
                            const void *, cudaDataType, int, const void *, cudaDataType, int, const void *, void *,
                            cudaDataType, int, cublasComputeType_t, cublasGemmAlgo_t) = nullptr;
   cublasStatus_t (*setSpecialValues)(cublasHandle_t, cudaEmulationSpecialValuesSupport) = nullptr;  // optional
   bool ok = false;
};

Blas g_blas;
std::once_flag g_blas_once;

void load_blas() {
   const char *env = getenv("PVGPU_CUBLAS");
   const char *names[] = {env, "libcublas.so.13", "/usr/local/cuda/lib64/libcublas.so.13",
                          "/usr/local/cuda/lib64/libcublas.so", "libcublas.so"};
   for (const char *n : names) {
      if (!n) continue;
      g_blas.so = dlopen(n, RTLD_NOW | RTLD_GLOBAL);
      if (g_blas.so) break;
   }
   if (!g_blas.so) return;
   g_blas.create = reinterpret_cast<decltype(g_blas.create)>(dlsym(g_blas.so, "cublasCreate_v2"));
   g_blas.destroy = reinterpret_cast<decltype(g_blas.destroy)>(dlsym(g_blas.so, "cublasDestroy_v2"));
   g_blas.setStream = reinterpret_cast<decltype(g_blas.setStream)>(dlsym(g_blas.so, "cublasSetStream_v2"));
   g_blas.setWorkspace = reinterpret_cast<decltype(g_blas.setWorkspace)>(dlsym(g_blas.so, "cublasSetWorkspace_v2"));
   g_blas.gemmEx = reinterpret_cast<decltype(g_blas.gemmEx)>(dlsym(g_blas.so, "cublasGemmEx"));
   g_blas.setSpecialValues = reinterpret_cast<decltype(g_blas.setSpecialValues)>(
         dlsym(g_blas.so, "cublasSetEmulationSpecialValuesSupport"));
   g_blas.ok = g_blas.create && g_blas.destroy && g_blas.setStream && g_blas.setWorkspace && g_blas.gemmEx;
}

unsigned grid_for(int64_t n) {
   int64_t b = (n + kThreads - 1) / kThreads;
   return (unsigned)(b > 152 * 32 ? 152 * 32 : (b < 1 ? 1 : b));
}

}  // namespace

struct pvgpu_lca_grad {
   pvgpu_lca_grad_desc d;
   Geo g;
   float e = 0.f;
   int nseg = 0;
   cublasHandle_t blas = nullptr;
   cublasComputeType_t compute = CUBLAS_COMPUTE_32F_EMULATED_16BFX9;
   void *blasWs = nullptr;
   size_t blasWsBytes = 0;
   // device buffers (FP32 unless noted)
   float *V[2] = {nullptr, nullptr}, *A[2] = {nullptr, nullptr};  // forward ping-pong [M][F]
   float *ck = nullptr;                  // checkpoints: V at the start of each segment [nseg][M][F]
   float *sV = nullptr, *sA = nullptr;   // one segment's states [K][M][F]
   float *sR = nullptr;                  // one segment's im2col'd residuals [K][M][KP]
   float *sG = nullptr;                  // one segment's adjoints dL/dV of the later state [K][M][F]
   float *sGD = nullptr;                 // one segment's -im2col(fold(gR)) [K][M][KP]
   float *WT = nullptr;                  // W transposed [KP][F]
   float *D = nullptr, *R = nullptr, *Z = nullptr, *img = nullptr;
   float *gV = nullptr, *gR = nullptr, *gD = nullptr, *gA = nullptr, *gImg = nullptr;
   double *lossPartial = nullptr;
   // the split-plane path: states of one segment (V in FP32, planes of A, R, g, gD), W's planes
   bool tc = false;
   bf16 *pA = nullptr, *pR = nullptr, *pG = nullptr, *pGD = nullptr, *pW = nullptr, *pWT = nullptr;
   size_t planeA = 0, planeR = 0;  // values of one plane of pA (K slots) and of pR (K + 1 slots)
   bf16 *ckLo = nullptr, *vLo = nullptr, *sVLo = nullptr;  // the low parts of ck, V[0] and sV
   float *P = nullptr;             // partial correlations
   int splits = 0, bn = 128, bandRows = kMaxBandRows, xPer = 1;
   int *err = nullptr;
   CUtensorMap mA, mR, mG, mGD, mW, mWT;        // operands of the GEMMs (W's as B)
   CUtensorMap cA, cR, cG, cGD;                 // the same planes as operands of the correlations
   cudaStream_t capStream = nullptr;
   cudaGraphExec_t graph = nullptr;
   const float *gW = nullptr, *gX = nullptr;
   float *gDW = nullptr;
   double *gLoss = nullptr;
};

namespace {

// C[M][N] = alpha A[M][K] . op(B) + beta C, all row-major FP32.  transB: B is [N][K] (so op(B) =
// B^T), else [K][N].  cuBLAS is column-major: C^T = op(B)^T A^T.
pvgpu_status gemm_rm(pvgpu_lca_grad *s, cudaStream_t st, int64_t M, int64_t N, int64_t K, float alpha,
                     const float *Am, const float *B, bool transB, float beta, float *Cm) {
   (void)st;
   const cublasStatus_t r =
         g_blas.gemmEx(s->blas, transB ? CUBLAS_OP_T : CUBLAS_OP_N, CUBLAS_OP_N, (int)N, (int)M, (int)K, &alpha, B,
                       CUDA_R_32F, transB ? (int)K : (int)N, Am, CUDA_R_32F, (int)K, &beta, Cm, CUDA_R_32F, (int)N,
                       s->compute, CUBLAS_GEMM_DEFAULT);
   return r == CUBLAS_STATUS_SUCCESS ? PVGPU_OK : pvgpu::record_message(PVGPU_ERR_LAUNCH, "lca_grad: cublasGemmEx failed");
}

// C[M][N] = alpha A^T . B + beta C with A [K][M], B [K][N] row-major (the correlation over K):
// C^T = B^T A in column-major terms.
pvgpu_status gemm_tn(pvgpu_lca_grad *s, int64_t M, int64_t N, int64_t K, float alpha, const float *Am,
                     const float *B, float beta, float *Cm) {
   const cublasStatus_t r =
         g_blas.gemmEx(s->blas, CUBLAS_OP_N, CUBLAS_OP_T, (int)N, (int)M, (int)K, &alpha, B, CUDA_R_32F, (int)N, Am,
                       CUDA_R_32F, (int)M, &beta, Cm, CUDA_R_32F, (int)N, s->compute, CUBLAS_GEMM_DEFAULT);
   return r == CUBLAS_STATUS_SUCCESS ? PVGPU_OK : pvgpu::record_message(PVGPU_ERR_LAUNCH, "lca_grad: cublasGemmEx failed");
}

#define PVGPU_TRY(x)                   \
   do {                                \
      pvgpu_status st_ = (x);          \
      if (st_ != PVGPU_OK) return st_; \
   } while (0)

// One forward timestep from (v, a) to (vOut, aOut); the im2col'd residual goes to Rout.
pvgpu_status forward_step(pvgpu_lca_grad *s, cudaStream_t st, const float *W, const float *x, const float *v,
                          const float *a, float *vOut, float *aOut, float *Rout) {
   const Geo &g = s->g;
   PVGPU_TRY(gemm_rm(s, st, g.M, g.KP, g.F, 1.0f, a, s->WT, true, 0.0f, s->D));  // D = A . W
   const int64_t nImg = (int64_t)g.nb * g.iny * g.inx * g.C;
   fold_kernel<<<grid_for(nImg), kThreads, 0, st>>>(g, s->D, x, -1.0f, s->img);  // r = x - fold(D)
   im2col_kernel<<<(unsigned)g.M, kThreads, 0, st>>>(g, s->img, 1.0f, Rout);
   PVGPU_TRY(gemm_rm(s, st, g.M, g.F, g.KP, 1.0f, Rout, W, true, 0.0f, s->Z));  // Z = R . W^T
   update_kernel<<<grid_for(g.M * g.F), kThreads, 0, st>>>((int)(g.M * g.F), s->e, s->d.VThresh, v, a, s->Z, vOut,
                                                           aOut);
   PVGPU_CHECK_LAUNCH("lca_grad forward");
   return PVGPU_OK;
}

pvgpu_status enqueue(pvgpu_lca_grad *s, const float *W, const float *x, float *dW, double *loss, cudaStream_t st) {
   const Geo &g = s->g;
   const int T = s->d.steps, K = s->d.checkpointEvery;
   const int64_t nV = g.M * g.F, nRk = g.M * g.KP;
   const float vt = s->d.VThresh, e = s->e;
   transpose_kernel<<<dim3((g.KP + 31) / 32, (g.F + 31) / 32), dim3(32, 8), 0, st>>>(g.F, g.KP, W, s->WT);
   // ---- forward, V = 0, checkpoint V at the start of every segment ----
   PVGPU_CUDA(cudaMemsetAsync(s->V[0], 0, nV * sizeof(float), st), "lca_grad zero");
   PVGPU_CUDA(cudaMemsetAsync(s->A[0], 0, nV * sizeof(float), st), "lca_grad zero");
   int cur = 0;
   for (int t = 0; t < T; t++) {
      if (t % K == 0)
         PVGPU_CUDA(cudaMemcpyAsync(s->ck + (size_t)(t / K) * nV, s->V[cur], nV * sizeof(float), cudaMemcpyDeviceToDevice,
                                    st),
                    "lca_grad checkpoint");
      PVGPU_TRY(forward_step(s, st, W, x, s->V[cur], s->A[cur], s->V[1 - cur], s->A[1 - cur], s->R));
      cur = 1 - cur;
   }
   // ---- the loss at a_T, and the seed of the adjoint ----
   PVGPU_TRY(gemm_rm(s, st, g.M, g.KP, g.F, 1.0f, s->A[cur], s->WT, true, 0.0f, s->D));
   const int64_t nImg = (int64_t)g.nb * g.iny * g.inx * g.C;
   fold_kernel<<<grid_for(nImg), kThreads, 0, st>>>(g, s->D, x, -1.0f, s->img);  // r_T
   im2col_kernel<<<(unsigned)g.M, kThreads, 0, st>>>(g, s->img, 1.0f, s->R);     // R_T
   PVGPU_TRY(gemm_rm(s, st, g.M, g.F, g.KP, 1.0f, s->R, W, true, 0.0f, s->Z));  // Z_T = R_T . W^T
   loss_partial_kernel<<<kLossBlocks, kThreads, 0, st>>>(nImg, s->img, nV, s->A[cur], (double)s->d.lambda1,
                                                         s->lossPartial);
   loss_final_kernel<<<1, 32, 0, st>>>(s->lossPartial, kLossBlocks, loss);
   seed_kernel<<<grid_for(nV), kThreads, 0, st>>>(nV, vt, s->d.lambda1, s->V[cur], s->A[cur], s->Z, s->gV);
   PVGPU_TRY(gemm_tn(s, g.F, g.KP, g.M, -1.0f, s->A[cur], s->R, 0.0f, dW));  // dW = -A_T^T R_T
   PVGPU_CHECK_LAUNCH("lca_grad loss");
   // ---- segments in reverse: recompute the segment's states, then its adjoint steps ----
   for (int seg = s->nseg - 1; seg >= 0; seg--) {
      const int t0 = seg * K, t1 = t0 + K < T ? t0 + K : T, n = t1 - t0;
      PVGPU_CUDA(cudaMemcpyAsync(s->sV, s->ck + (size_t)seg * nV, nV * sizeof(float), cudaMemcpyDeviceToDevice, st),
                 "lca_grad restore");
      threshold_kernel<<<grid_for(nV), kThreads, 0, st>>>(nV, vt, s->sV, s->sA);
      for (int i = 0; i < n; i++) {
         // state i + 1 goes to slot i + 1; the segment's last output is not needed
         float *vo = i + 1 < n ? s->sV + (size_t)(i + 1) * nV : s->V[0];
         float *ao = i + 1 < n ? s->sA + (size_t)(i + 1) * nV : s->A[0];
         PVGPU_TRY(forward_step(s, st, W, x, s->sV + (size_t)i * nV, s->sA + (size_t)i * nV, vo, ao,
                                s->sR + (size_t)i * nRk));
      }
      // the adjoint steps: g of step i lives in sG[i]; step i writes dL/dV_t into sG[i - 1], or
      // into gV for the segment before
      PVGPU_CUDA(cudaMemcpyAsync(s->sG + (size_t)(n - 1) * nV, s->gV, nV * sizeof(float), cudaMemcpyDeviceToDevice, st),
                 "lca_grad adjoint carry");
      for (int i = n - 1; i >= 0; i--) {
         const float *Vt = s->sV + (size_t)i * nV, *gi = s->sG + (size_t)i * nV;
         float *gDi = s->sGD + (size_t)i * nRk;
         PVGPU_TRY(gemm_rm(s, st, g.M, g.KP, g.F, 1.0f - e, gi, s->WT, true, 0.0f, s->gR));  // gR = (1-e) g . W
         fold_kernel<<<grid_for(nImg), kThreads, 0, st>>>(g, s->gR, nullptr, 1.0f, s->gImg);  // gr = fold(gR)
         im2col_kernel<<<(unsigned)g.M, kThreads, 0, st>>>(g, s->gImg, -1.0f, gDi);         // gD = -im2col(gr)
         PVGPU_TRY(gemm_rm(s, st, g.M, g.F, g.KP, 1.0f, gDi, W, true, 0.0f, s->gA));        // gA = gD . W^T
         adjoint_update_kernel<<<grid_for(nV), kThreads, 0, st>>>((int)nV, e, vt, Vt, s->gA, gi,
                                                                  i > 0 ? s->sG + (size_t)(i - 1) * nV : s->gV);
         PVGPU_CHECK_LAUNCH("lca_grad adjoint");
      }
      // the segment's correlations, each one GEMM over all its steps' positions:
      // dW += (1 - e) sum_i g_i^T R_i + sum_i A_i^T gD_i
      PVGPU_TRY(gemm_tn(s, g.F, g.KP, (int64_t)n * g.M, 1.0f - e, s->sG, s->sR, 1.0f, dW));
      PVGPU_TRY(gemm_tn(s, g.F, g.KP, (int64_t)n * g.M, 1.0f, s->sA, s->sGD, 1.0f, dW));
   }
   return PVGPU_OK;
}

// ---- the split-plane run -------------------------------------------------------------------
template <typename Kernel, typename... Args>
pvgpu_status launch_pdl(Kernel kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
   cudaLaunchAttribute attr[1];
   attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   attr[0].val.programmaticStreamSerializationAllowed = 1;
   cudaLaunchConfig_t c = {};
   c.gridDim = grid;
   c.blockDim = dim3(threads);
   c.dynamicSmemBytes = smem;
   c.stream = st;
   c.attrs = attr;
   c.numAttrs = 1;
   PVGPU_CUDA(cudaLaunchKernelEx(&c, kernel, args...), "lca_grad launch");
   return PVGPU_OK;
}

constexpr size_t gemm_smem(int bn) { return pvgpu::split::stages_of(bn) * 3 * (pvgpu::split::kPlaneA + (size_t)bn * 128) + 1024; }
constexpr size_t kCorrSmem = 2 * 6 * (size_t)pvgpu::split::kPlaneA + 1024;

// A band of windows takes at most this much shared memory.  The limit that a launch is checked against belongs to
// the kernel, not to a handle, so it is set to the bound and never to one handle's size.
constexpr size_t kBandSmem = 200 * 1024;

size_t band_smem(const Geo &g, int xPer) {
   return sizeof(float) * (size_t)(g.S * (kMaxBandRows - 1) + g.P) * (((g.S * (xPer - 1) + g.P) * g.C + 3) & ~3);
}

template <typename Epi>
pvgpu_status gemm_tc(pvgpu_lca_grad *s, cudaStream_t st, const CUtensorMap &a, int aSlot, const CUtensorMap &b, int N, int K,
                     const Epi &epi) {
   using namespace pvgpu::split;
   const dim3 grid((N + s->bn - 1) / s->bn, (unsigned)((s->g.M + 127) / 128));
   if (s->bn == 128)
      return launch_pdl(gemm_kernel<128, Epi>, grid, pvgpu::split::kThreads, gemm_smem(128), st, a, b, aSlot, (int)s->g.M, N, K, epi, s->err);
   if (s->bn == 64)
      return launch_pdl(gemm_kernel<64, Epi>, grid, pvgpu::split::kThreads, gemm_smem(64), st, a, b, aSlot, (int)s->g.M, N, K, epi, s->err);
   return launch_pdl(gemm_kernel<32, Epi>, grid, pvgpu::split::kThreads, gemm_smem(32), st, a, b, aSlot, (int)s->g.M, N, K, epi, s->err);
}

template <typename Epi>
bool gemm_attrs() {
   using namespace pvgpu::split;
   return cudaFuncSetAttribute(gemm_kernel<128, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(128)) == cudaSuccess &&
          cudaFuncSetAttribute(gemm_kernel<64, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(64)) == cudaSuccess &&
          cudaFuncSetAttribute(gemm_kernel<32, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(32)) == cudaSuccess;
}

bool special_geometry(const Geo &g) {
   return (g.S == 4 && g.P == 16 && g.C == 1) || (g.S == 2 && g.P == 8 && (g.C == 1 || g.C == 3));
}

template <typename Fn>
auto with_geometry(const Geo &g, Fn &&fn) {
   if (g.S == 4 && g.P == 16 && g.C == 1) return fn(fold_im2col_kernel<4, 16, 1>);
   if (g.S == 2 && g.P == 8 && g.C == 1) return fn(fold_im2col_kernel<2, 8, 1>);
   if (g.S == 2 && g.P == 8 && g.C == 3) return fn(fold_im2col_kernel<2, 8, 3>);
   return fn(fold_im2col_kernel<0, 0, 0>);
}

pvgpu_status fold_im2col(pvgpu_lca_grad *s, cudaStream_t st, const float *x, float signImg, float signOut, bf16 *out,
                         size_t plane) {
   const Geo &g = s->g;
   const dim3 grid((unsigned)(g.nb * ((g.vy + s->bandRows - 1) / s->bandRows)), (g.vx + s->xPer - 1) / s->xPer);
   return with_geometry(g, [&](auto kernel) {
      return launch_pdl(kernel, grid, kFoldThreads, band_smem(g, s->xPer), st, g, s->bandRows, s->xPer, (const float *)s->D, x, signImg,
                        signOut, out, plane);
   });
}

pvgpu_status correlate(pvgpu_lca_grad *s, cudaStream_t st, int slot, bool both) {
   using namespace pvgpu::split;
   CorrArgs a;
   a.slotA[0] = 0;       // g^T R of the step
   a.slotB[0] = slot;
   a.slotA[1] = slot;    // A^T gD
   a.slotB[1] = 0;
   a.pair0 = both ? 0 : 1;
   a.M = (int)s->g.M;
   a.F = s->g.F;
   a.KP = s->g.KP;
   a.mt = (a.F + 127) / 128;
   a.nt = (a.KP + 127) / 128;
   a.splits = s->splits;
   a.P = s->P;
   return launch_pdl(corr_kernel, dim3((both ? 2 : 1) * a.mt * a.nt * a.splits), pvgpu::split::kThreads, kCorrSmem, st, s->cG, s->cR, s->cA,
                     s->cGD, a, s->err);
}

pvgpu_status enqueue_tc(pvgpu_lca_grad *s, const float *W, const float *x, float *dW, double *loss, cudaStream_t st) {
   const Geo &g = s->g;
   const int T = s->d.steps, K = s->d.checkpointEvery, F = g.F, KP = g.KP;
   const int64_t nV = g.M * F, nRk = g.M * KP;
   const float vt = s->d.VThresh, e = s->e;
   const int t0Last = (s->nseg - 1) * K;  // the last segment's states stay from the forward pass
   const size_t nW = (size_t)F * KP;
   PVGPU_CUDA(cudaMemsetAsync(s->P, 0, 2 * (size_t)s->splits * nW * sizeof(float), st), "lca_grad zero");
   PVGPU_CUDA(cudaMemsetAsync(s->err, 0, sizeof(int), st), "lca_grad zero");
   PVGPU_CUDA(cudaMemsetAsync(s->ck, 0, nV * sizeof(float), st), "lca_grad zero");  // V = 0
   PVGPU_CUDA(cudaMemsetAsync(s->ckLo, 0, nV * sizeof(bf16), st), "lca_grad zero");
   for (int q = 0; q < 3; q++)
      PVGPU_CUDA(cudaMemsetAsync(s->pA + q * s->planeA, 0, nV * sizeof(bf16), st), "lca_grad zero");
   split_weights_kernel<<<grid_for((int64_t)nW), kThreads, 0, st>>>(F, KP, W, s->pW, s->pWT);
   PVGPU_CHECK_LAUNCH("lca_grad weights");
   // R of one step's activity (slot sa) into R's slot sr
   auto residual = [&](int sa, int sr) -> pvgpu_status {
      PVGPU_TRY(gemm_tc(s, st, s->mA, sa, s->mWT, KP, F, EpiStore{1.0f, s->D}));       // D = A . W
      return fold_im2col(s, st, x, -1.0f, 1.0f, s->pR + (size_t)sr * nRk, s->planeR);  // R = im2col(x - fold(D))
   };
   // V and A's planes of the next step from R's slot sr
   struct State {
      float *hi;
      bf16 *lo;
   };
   const float below = std::nextafter(vt, -INFINITY);
   auto update = [&](int sr, const State &v, const State &out, int aOut) {
      return gemm_tc(s, st, s->mR, sr, s->mW, F, KP,
                     EpiForward{1.0f - e, vt, below, v.hi, v.lo, out.hi, out.lo, s->pA + (size_t)aOut * nV, s->planeA});
   };
   auto ck = [&](int seg) { return State{s->ck + (size_t)seg * nV, s->ckLo + (size_t)seg * nV}; };
   auto slot = [&](int i) { return State{s->sV + (size_t)i * nV, s->sVLo + (size_t)i * nV}; };
   // ---- forward: V of each segment's start into ck; A's planes in slot 0, and the last segment's
   // states in the slots of a segment ----
   State v = ck(0);
   for (int t = 0; t < T; t++) {
      const int i = t - t0Last;
      const State out = i >= 0 ? slot(i + 1) : (t + 1) % K == 0 ? ck((t + 1) / K) : State{s->V[0], s->vLo};
      PVGPU_TRY(residual(std::max(i, 0), std::max(i, 0)));
      PVGPU_TRY(update(std::max(i, 0), v, out, i >= 0 ? i + 1 : 0));
      v = out;
   }
   const int nLast = T - t0Last;
   // ---- the loss at a_T, the seed of the adjoint and dW = -A_T^T R_T ----
   PVGPU_TRY(gemm_tc(s, st, s->mA, nLast, s->mWT, KP, F, EpiStore{1.0f, s->D}));
   const int64_t nImg = (int64_t)g.nb * g.iny * g.inx * g.C;
   fold_kernel<<<grid_for(nImg), kThreads, 0, st>>>(g, s->D, x, -1.0f, s->img);  // r_T
   threshold_kernel<<<grid_for(nV), kThreads, 0, st>>>(nV, vt, v.hi, s->A[0]);
   loss_partial_kernel<<<kLossBlocks, kThreads, 0, st>>>(nImg, s->img, nV, s->A[0], (double)s->d.lambda1, s->lossPartial);
   loss_final_kernel<<<1, 32, 0, st>>>(s->lossPartial, kLossBlocks, loss);
   PVGPU_CHECK_LAUNCH("lca_grad loss");
   PVGPU_TRY(fold_im2col(s, st, x, -1.0f, 1.0f, s->pR + (size_t)K * nRk, s->planeR));  // R_T, a slot of its own
   PVGPU_TRY(gemm_tc(s, st, s->mR, K, s->mW, F, KP, EpiSeed{vt, s->d.lambda1, v.hi, s->gV, s->pG, (size_t)nV}));
   PVGPU_TRY(fold_im2col(s, st, x, -1.0f, -1.0f, s->pGD, (size_t)nRk));  // -R_T in gD's place
   PVGPU_TRY(correlate(s, st, nLast, false));
   // ---- segments in reverse ----
   for (int seg = s->nseg - 1; seg >= 0; seg--) {
      const int n = std::min(K, T - seg * K);
      const State v0 = ck(seg);
      if (seg < s->nseg - 1) {
         PVGPU_TRY(launch_pdl(split_activity_kernel, dim3(grid_for(nV / 8)), kThreads, 0, st, (int64_t)(nV / 8), vt,
                              (const float *)v0.hi, (const bf16 *)v0.lo, s->pA, s->planeA));
         for (int i = 0; i < n; i++) {
            PVGPU_TRY(residual(i, i));
            if (i + 1 < n) PVGPU_TRY(update(i, i ? slot(i) : v0, slot(i + 1), i + 1));
         }
      }
      for (int i = n - 1; i >= 0; i--) {
         PVGPU_TRY(gemm_tc(s, st, s->mG, 0, s->mWT, KP, F, EpiStore{1.0f - e, s->D}));  // gR = (1-e) g . W
         PVGPU_TRY(fold_im2col(s, st, nullptr, 1.0f, -1.0f, s->pGD, (size_t)nRk));      // gD = -im2col(fold(gR))
         PVGPU_TRY(correlate(s, st, i, true));                                         // g^T R_i and A_i^T gD
         PVGPU_TRY(gemm_tc(s, st, s->mGD, 0, s->mW, F, KP,
                           EpiAdjoint{e, vt, i ? slot(i).hi : v0.hi, s->gV, s->pG, (size_t)nV}));
      }
   }
   return launch_pdl(corr_sum_kernel, dim3(grid_for((int64_t)nW)), kThreads, 0, st, (int)nW, s->splits, 1.0f - e,
                     (const float *)s->P, (const int *)s->err, dW, loss);
}

void free_all(pvgpu_lca_grad *s) {
   if (!s) return;
   if (s->graph) cudaGraphExecDestroy(s->graph);
   if (s->capStream) cudaStreamDestroy(s->capStream);
   if (s->blas) g_blas.destroy(s->blas);
   void *bufs[] = {s->V[0], s->V[1], s->A[0], s->A[1], s->ck, s->sV, s->sA, s->sR, s->sG, s->sGD, s->WT, s->D, s->R,
                   s->Z, s->img, s->gV, s->gR, s->gD, s->gA, s->gImg, s->lossPartial, s->blasWs, s->pA, s->pR, s->pG, s->pGD, s->pW,
                   s->pWT, s->P, s->err, s->ckLo, s->vLo, s->sVLo};
   for (void *p : bufs)
      if (p) cudaFree(p);
   delete s;
}

}  // namespace

extern "C" pvgpu_status pvgpu_lca_grad_create(const pvgpu_lca_grad_desc *d, pvgpu_lca_grad **out) {
   if (!d || !out) return PVGPU_ERR_BAD_ARG;
   *out = nullptr;
   if (d->nbatch <= 0 || d->inNx <= 0 || d->inNy <= 0 || d->inNf <= 0 || d->v1Nx <= 0 || d->v1Ny <= 0 ||
       d->v1Nf <= 0 || d->nxp <= 0 || d->steps <= 0 || d->checkpointEvery <= 0 || !(d->tau > 0.0f) ||
       !(d->dt > 0.0f))
      return PVGPU_ERR_BAD_ARG;
   if (d->inNx % d->v1Nx || d->inNy % d->v1Ny || d->inNx / d->v1Nx != d->inNy / d->v1Ny)
      return pvgpu::record_message(PVGPU_ERR_UNSUPPORTED_SHAPE, "lca_grad: V1 must tile the input with one stride");
   const int S = d->inNx / d->v1Nx;
   if (d->nxp < S || (d->nxp - S) % 2)
      return pvgpu::record_message(PVGPU_ERR_ILLEGAL_GEOMETRY, "lca_grad: patch must exceed the stride by an even amount");
   pvgpu_lca_grad *s = new (std::nothrow) pvgpu_lca_grad();
   if (!s) return PVGPU_ERR_OOM;
   s->d = *d;
   Geo &g = s->g;
   g.nb = d->nbatch;
   g.iny = d->inNy;
   g.inx = d->inNx;
   g.C = d->inNf;
   g.vy = d->v1Ny;
   g.vx = d->v1Nx;
   g.F = d->v1Nf;
   g.P = d->nxp;
   g.S = S;
   g.E = (d->nxp - S) / 2;
   g.KP = g.P * g.P * g.C;
   g.Np = g.vy * g.vx;
   g.M = (int64_t)g.nb * g.Np;
   s->e = (float)std::exp(-(double)d->dt / (double)d->tau);
   const int K = d->checkpointEvery;
   s->nseg = (d->steps + K - 1) / K;
   const size_t nV = (size_t)g.M * g.F, nR = (size_t)g.M * g.KP, nImg = (size_t)g.nb * g.iny * g.inx * g.C;
   bool ok = true;
   auto alloc = [&](void **p, size_t bytes) {
      if (ok && cudaMalloc(p, bytes) != cudaSuccess) ok = false;
   };
   auto f32 = [&](float **p, size_t n) { alloc(reinterpret_cast<void **>(p), n * 4); };
   f32(&s->D, nR);
   f32(&s->img, nImg);
   f32(&s->gV, nV);
   alloc(reinterpret_cast<void **>(&s->lossPartial), kLossBlocks * sizeof(double));
   f32(&s->ck, (size_t)s->nseg * nV);
   // the split-plane path: T(0) = 0, rows of whole 16-byte groups, 32-bit matrix sizes, a band of windows in
   // shared memory
   bool noRoom = false;
   s->tc = ok && d->VThresh >= 0.0f && g.F % 8 == 0 && g.KP % 8 == 0 && g.M <= 0x7fffff00LL && (g.M + 127) / 128 <= 65535 &&
           (int64_t)g.nb * g.vy <= 0x7fffffff && band_smem(g, g.vx) <= kBandSmem &&
           (size_t)g.F * g.KP <= 0x7fffffff && pvgpu::encode_tiled_fn() != nullptr;
   if (s->tc) {
      auto planes = [&](bf16 **p, size_t n) { alloc(reinterpret_cast<void **>(p), 3 * n * sizeof(bf16)); };
      const size_t nW = (size_t)g.F * g.KP;
      s->planeA = (size_t)(K + 1) * nV;  // slot K: the activity after the last segment
      s->planeR = (size_t)(K + 1) * nR;  // slot K: R_T
      f32(&s->V[0], nV);
      f32(&s->A[0], nV);
      f32(&s->sV, (size_t)(K + 1) * nV);
      alloc(reinterpret_cast<void **>(&s->ckLo), (size_t)s->nseg * nV * sizeof(bf16));
      alloc(reinterpret_cast<void **>(&s->vLo), nV * sizeof(bf16));
      alloc(reinterpret_cast<void **>(&s->sVLo), (size_t)(K + 1) * nV * sizeof(bf16));
      planes(&s->pA, s->planeA);
      planes(&s->pR, s->planeR);
      planes(&s->pG, nV);
      planes(&s->pGD, nR);
      planes(&s->pW, nW);
      planes(&s->pWT, nW);
      const int tiles = ((g.F + 127) / 128) * ((g.KP + 127) / 128), sms = pvgpu::num_sms();
      // ranges of positions: as many as give every SM a CTA of the two pairs' tiles, of a chunk at least
      s->splits = std::max(1, (int)std::min<int64_t>(sms / (2 * tiles), (g.M + 63) / 64));
      f32(&s->P, 2 * (size_t)s->splits * nW);
      alloc(reinterpret_cast<void **>(&s->err), sizeof(int));
      // columns per tile: the fewest whose tiles still fit in one wave of the SMs (M = 512, F = 224, 66
      // steps in segments of 5: 4.2 ms with 32 columns, 4.8 with 64; M = 5120, F = 256, 20 steps: 1.9 ms with
      // 128 columns, 2.3 in two waves of 64)
      const int64_t mTiles = (g.M + 127) / 128, n = std::max(g.F, g.KP);
      s->bn = 128;
      for (int bn = 64; bn >= 32 && mTiles * ((n + bn - 1) / bn) <= sms; bn /= 2) s->bn = bn;
      s->bandRows = (int64_t)g.nb * ((g.vy + 1) / 2) < sms / 2 ? 1 : 2;
      // positions of a row per CTA: whole rows, but where these leave half of the SMs idle and a thread more than
      // ten loads of the gather in a row, as few (two at least) as give every SM two CTAs.  Over 230 geometries:
      // 5 to 25 % of a run there; elsewhere the overlap of the parts' windows costs 2 to 18 %.
      s->xPer = g.vx;
      const int64_t bands = (int64_t)g.nb * ((g.vy + s->bandRows - 1) / s->bandRows);
      const double loads = (double)band_smem(g, g.vx) / 4 / kFoldThreads * (g.P / S) * (g.P / S);
      if (!special_geometry(g) && bands < sms / 2 && loads >= 10) {
         const int64_t parts = std::min<int64_t>((2 * sms + bands - 1) / bands, (g.vx + 1) / 2);
         s->xPer = (int)((g.vx + parts - 1) / parts);
      }
      using pvgpu::split::make_map;
      const uint64_t M = (uint64_t)g.M, F = g.F, KP = g.KP;
      if (ok && !(make_map(&s->mA, s->pA, s->planeA, K + 1, M, F, 128) && make_map(&s->mR, s->pR, s->planeR, K + 1, M, KP, 128) &&
                  make_map(&s->mG, s->pG, nV, 1, M, F, 128) && make_map(&s->mGD, s->pGD, nR, 1, M, KP, 128) &&
                  make_map(&s->mW, s->pW, nW, 1, F, KP, s->bn) && make_map(&s->mWT, s->pWT, nW, 1, KP, F, s->bn) &&
                  make_map(&s->cA, s->pA, s->planeA, K + 1, M, F, 64) && make_map(&s->cR, s->pR, s->planeR, K + 1, M, KP, 64) &&
                  make_map(&s->cG, s->pG, nV, 1, M, F, 64) && make_map(&s->cGD, s->pGD, nR, 1, M, KP, 64) &&
                  gemm_attrs<EpiStore>() && gemm_attrs<EpiForward>() && gemm_attrs<EpiAdjoint>() && gemm_attrs<EpiSeed>() &&
                  cudaFuncSetAttribute(pvgpu::split::corr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kCorrSmem) == cudaSuccess &&
                  with_geometry(g, [&](auto kernel) {
                     return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBandSmem) == cudaSuccess;
                  }))) {
         cudaGetLastError();
         free_all(s);
         return pvgpu::record_message(PVGPU_ERR_LAUNCH, "lca_grad: tensor maps");
      }
      if (ok) {
         cudaMemset(s->err, 0, sizeof(int));
         if (cudaStreamCreateWithFlags(&s->capStream, cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            s->capStream = nullptr;
         }
         *out = s;
         return PVGPU_OK;
      }
      // The low parts of the checkpoints are half as much again (100 steps with a checkpoint before each: 644 bytes a
      // neuron against 440): where only the library path's buffers fit, that path runs.
      cudaGetLastError();
      void **mine[] = {(void **)&s->V[0], (void **)&s->A[0], (void **)&s->sV,  (void **)&s->ckLo, (void **)&s->vLo,
                       (void **)&s->sVLo, (void **)&s->pA,   (void **)&s->pR,  (void **)&s->pG,   (void **)&s->pGD,
                       (void **)&s->pW,   (void **)&s->pWT,  (void **)&s->P,   (void **)&s->err};
      for (void **p : mine) {
         if (*p) cudaFree(*p);
         *p = nullptr;
      }
      s->tc = false;
      ok = noRoom = true;
   }
   std::call_once(g_blas_once, load_blas);
   if (!g_blas.ok) {
      free_all(s);
      return noRoom ? PVGPU_ERR_OOM
                    : pvgpu::record_message(PVGPU_ERR_UNSUPPORTED_SHAPE, "lca_grad: cuBLAS could not be loaded");
   }
   for (int i = 0; i < 2; i++) {
      alloc(reinterpret_cast<void **>(&s->V[i]), nV * 4);
      alloc(reinterpret_cast<void **>(&s->A[i]), nV * 4);
   }
   alloc(reinterpret_cast<void **>(&s->sV), (size_t)K * nV * 4);
   alloc(reinterpret_cast<void **>(&s->sA), (size_t)K * nV * 4);
   alloc(reinterpret_cast<void **>(&s->sR), (size_t)K * nR * 4);
   alloc(reinterpret_cast<void **>(&s->sG), (size_t)K * nV * 4);
   alloc(reinterpret_cast<void **>(&s->sGD), (size_t)K * nR * 4);
   alloc(reinterpret_cast<void **>(&s->WT), (size_t)g.F * g.KP * 4);
   alloc(reinterpret_cast<void **>(&s->R), nR * 4);
   constexpr int kProbe = 16;  // the probe below multiplies two kProbe x kProbe blocks within Z
   alloc(reinterpret_cast<void **>(&s->Z), std::max<size_t>(nV, 2 * kProbe * kProbe) * 4);
   alloc(reinterpret_cast<void **>(&s->gR), nR * 4);
   alloc(reinterpret_cast<void **>(&s->gD), nR * 4);
   alloc(reinterpret_cast<void **>(&s->gA), nV * 4);
   alloc(reinterpret_cast<void **>(&s->gImg), nImg * 4);
   s->blasWsBytes = 64u << 20;  // cuBLAS takes this instead of allocating (also inside a capture)
   alloc(&s->blasWs, s->blasWsBytes);
   if (!ok) {
      cudaGetLastError();
      free_all(s);
      return PVGPU_ERR_OOM;
   }
   if (g_blas.create(&s->blas) != CUBLAS_STATUS_SUCCESS ||
       g_blas.setWorkspace(s->blas, s->blasWs, s->blasWsBytes) != CUBLAS_STATUS_SUCCESS) {
      s->blas = nullptr;
      free_all(s);
      return pvgpu::record_message(PVGPU_ERR_LAUNCH, "lca_grad: cuBLAS handle");
   }
   // the operands are finite (a run with an inf or NaN in W or x has no meaningful gradient), so the
   // emulated GEMMs skip their scans for special values
   if (g_blas.setSpecialValues) g_blas.setSpecialValues(s->blas, CUDA_EMULATION_SPECIAL_VALUES_SUPPORT_NONE);
   if (cudaStreamCreateWithFlags(&s->capStream, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      s->capStream = nullptr;
   }
   // FP32 emulated on the BF16 tensor cores where cuBLAS takes it, else plain FP32: one probe GEMM
   {
      float *p = s->Z;
      const float one = 1.0f, zero = 0.0f;
      g_blas.setStream(s->blas, nullptr);
      if (g_blas.gemmEx(s->blas, CUBLAS_OP_N, CUBLAS_OP_N, kProbe, kProbe, kProbe, &one, p, CUDA_R_32F, kProbe, p, CUDA_R_32F,
                        kProbe, &zero, p + kProbe * kProbe, CUDA_R_32F, kProbe, CUBLAS_COMPUTE_32F_EMULATED_16BFX9,
                        CUBLAS_GEMM_DEFAULT) != CUBLAS_STATUS_SUCCESS)
         s->compute = CUBLAS_COMPUTE_32F;
      cudaDeviceSynchronize();
      cudaGetLastError();
   }
   *out = s;
   return PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_lca_grad_destroy(pvgpu_lca_grad *s) {
   if (!s) return PVGPU_ERR_BAD_ARG;
   free_all(s);
   return PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_lca_grad_info(const pvgpu_lca_grad *s, int *emulatedFp32) {
   if (!s || !emulatedFp32) return PVGPU_ERR_BAD_ARG;
   *emulatedFp32 = s->tc || s->compute == CUBLAS_COMPUTE_32F_EMULATED_16BFX9 ? 1 : 0;
   return PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_lca_grad_error_flag(const pvgpu_lca_grad *s, int *hostFlag) {
   if (!s || !hostFlag) return PVGPU_ERR_BAD_ARG;
   *hostFlag = 0;
   if (s->err) PVGPU_CUDA(cudaMemcpy(hostFlag, s->err, sizeof(int), cudaMemcpyDeviceToHost), "lca_grad error flag");
   return PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_selftest_gemm_expiry(int chunks, long long *hostOut4, void *stream) {
   if (!hostOut4 || chunks < 1 || chunks > 64) return PVGPU_ERR_BAD_ARG;
   cudaStream_t s = pvgpu::as_stream(stream);
   constexpr size_t kWords = 8;  // error word, then each kernel's time and whether it wrote
   long long host[kWords] = {}, *d = nullptr;
   PVGPU_CUDA(cudaFuncSetAttribute(gemm_expiry_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(32)),
              "selftest_gemm_expiry");
   PVGPU_CUDA(cudaMallocAsync(&d, sizeof(host), s), "selftest_gemm_expiry");
   cudaError_t e = cudaMemsetAsync(d, 0, sizeof(host), s);
   for (int k = 0; k < 2 && e == cudaSuccess; k++) {
      gemm_expiry_kernel<<<1, pvgpu::split::kThreads, gemm_smem(32), s>>>(chunks, reinterpret_cast<int *>(d), d + 2 + 2 * k);
      e = cudaGetLastError();
      if (e == cudaSuccess && k == 0) e = cudaMemcpyAsync(host + 6, d, sizeof(int), cudaMemcpyDeviceToHost, s);
   }
   if (e == cudaSuccess) e = cudaMemcpyAsync(host, d, 6 * sizeof(long long), cudaMemcpyDeviceToHost, s);
   const cudaError_t f = cudaFreeAsync(d, s);
   if (e == cudaSuccess) e = f;
   if (e == cudaSuccess) e = cudaStreamSynchronize(s);
   if (e != cudaSuccess) return pvgpu::record_cuda_error(e, "selftest_gemm_expiry");
   hostOut4[0] = (int)host[6];
   hostOut4[1] = host[2];
   hostOut4[2] = host[4];
   hostOut4[3] = host[3] || host[5];
   return hostOut4[0] ? PVGPU_ERR_TIMEOUT : PVGPU_OK;
}

extern "C" pvgpu_status pvgpu_lca_grad_run(pvgpu_lca_grad *s, const float *W, const float *x, float *dW,
                                           double *loss, void *stream) {
   if (!s || !W || !x || !dW || !loss) return PVGPU_ERR_BAD_ARG;
   cudaStream_t st = pvgpu::as_stream(stream);
   if (!s->capStream) {  // no capture stream: enqueue directly on the caller's stream
      if (s->tc) return enqueue_tc(s, W, x, dW, loss, st);
      if (g_blas.setStream(s->blas, st) != CUBLAS_STATUS_SUCCESS)
         return pvgpu::record_message(PVGPU_ERR_LAUNCH, "lca_grad: cublasSetStream");
      return enqueue(s, W, x, dW, loss, st);
   }
   if (!s->graph || s->gW != W || s->gX != x || s->gDW != dW || s->gLoss != loss) {
      if (s->graph) cudaGraphExecDestroy(s->graph);
      s->graph = nullptr;
      if (!s->tc && g_blas.setStream(s->blas, s->capStream) != CUBLAS_STATUS_SUCCESS)
         return pvgpu::record_message(PVGPU_ERR_LAUNCH, "lca_grad: cublasSetStream");
      PVGPU_CUDA(cudaStreamBeginCapture(s->capStream, cudaStreamCaptureModeThreadLocal), "lca_grad capture");
      pvgpu_status r = s->tc ? enqueue_tc(s, W, x, dW, loss, s->capStream) : enqueue(s, W, x, dW, loss, s->capStream);
      cudaGraph_t gr = nullptr;
      cudaError_t ee = cudaStreamEndCapture(s->capStream, &gr);
      if (r != PVGPU_OK || ee != cudaSuccess) {
         if (gr) cudaGraphDestroy(gr);
         return r != PVGPU_OK ? r : pvgpu::record_cuda_error(ee, "lca_grad capture");
      }
      cudaError_t ei = cudaGraphInstantiate(&s->graph, gr, 0);
      cudaGraphDestroy(gr);
      if (ei != cudaSuccess) {
         s->graph = nullptr;
         return pvgpu::record_cuda_error(ei, "lca_grad instantiate");
      }
      s->gW = W;
      s->gX = x;
      s->gDW = dW;
      s->gLoss = loss;
   }
   PVGPU_CUDA(cudaGraphLaunch(s->graph, st), "lca_grad launch");
   return PVGPU_OK;
}
