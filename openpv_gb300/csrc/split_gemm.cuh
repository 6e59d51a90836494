// split_gemm.cuh -- FP32 GEMMs on the BF16 tensor cores: every operand is three BF16 planes whose sum
// is its FP32 value (x = p0 + p1 + p2, each the rounded remainder of the ones before), and a product
// takes the six plane products down to 2^-16 of the largest (p0 q0; p0 q1, p1 q0; p1 q1, p0 q2, p2 q0);
// what is left out is below 2^-24.
//
// The tensor core adds into its FP32 accumulator rounding toward zero, so a long chain loses half an
// ulp per instruction with the accumulator's sign: two chains of eight instructions (K = 256) biased a
// product by 1.2e-7, as much as FP32 rounding costs in all, and persistently, step after step.  The p0 q0
// products therefore run in chains of two instructions (K = 32) into two alternating accumulators, which
// the epilogue warps add up in registers, rounding to nearest, while the next chain runs; the five small
// products have an accumulator of their own (2^-8 of the size).
//
// Planes lie [plane][slot][row][col] (BF16, col contiguous and a multiple of 8); rows and columns beyond a
// slot's matrix read as zero.
#pragma once

#include "pvgpu_internal.cuh"
#include "tc_ptx.cuh"
#include "tmap.cuh"

namespace pvgpu {
namespace split {

using namespace pvgpu::tc;
using bf16 = __nv_bfloat16;

// Tensor map of an operand's three planes [3][slots][rows][cols], box = 64 columns x boxRows of one slot
// in all three planes (one copy lands as three tiles, plane after plane), 128-byte swizzle.
inline bool make_map(CUtensorMap *m, const bf16 *base, size_t planeStride, uint64_t slots, uint64_t rows, uint64_t cols,
                     uint32_t boxRows) {
   EncodeTiledFn enc = encode_tiled_fn();
   if (!enc || cols % 8 || planeStride % 8 || boxRows == 0 || boxRows > 256) return false;
   cuuint64_t dims[4] = {cols, rows, slots, 3};
   cuuint64_t strides[3] = {cols * 2, rows * cols * 2, planeStride * 2};
   cuuint32_t box[4] = {64, boxRows, 1, 3}, estr[4] = {1, 1, 1, 1};
   return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16 *>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

__device__ __forceinline__ void load_planes(void *dst, const CUtensorMap *map, uint64_t *bar, int col, int row, int slot) {
   asm volatile(
         "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
         "[%6];" ::"r"(smem_u32(dst)),
         "l"(reinterpret_cast<uint64_t>(map)), "r"(col), "r"(row), "r"(slot), "r"(0), "r"(smem_u32(bar))
         : "memory");
}

// Two values into their planes' packed pairs (the first in the low half).
__device__ __forceinline__ void split2(float a, float b, uint32_t *p) {
#pragma unroll
   for (int i = 0; i < 3; i++) {
      const bf16 x = __float2bfloat16_rn(a), y = __float2bfloat16_rn(b);
      a -= __bfloat162float(x);
      b -= __bfloat162float(y);
      p[i] = (uint32_t)__bfloat16_as_ushort(x) | ((uint32_t)__bfloat16_as_ushort(y) << 16);
   }
}

// Four values into 8 bytes of each plane (dst 8-byte aligned).
__device__ __forceinline__ void split_store4(const float4 &v, bf16 *dst, size_t planeStride) {
   uint32_t w[2][3];
   split2(v.x, v.y, w[0]);
   split2(v.z, v.w, w[1]);
#pragma unroll
   for (int i = 0; i < 3; i++) *reinterpret_cast<uint2 *>(dst + i * planeStride) = make_uint2(w[0][i], w[1][i]);
}

// Eight values into 16 bytes of each plane (dst 16-byte aligned).
__device__ __forceinline__ void split_store8(const float *v, bf16 *dst, size_t planeStride) {
   uint32_t w[4][3];
#pragma unroll
   for (int i = 0; i < 4; i++) split2(v[2 * i], v[2 * i + 1], w[i]);
#pragma unroll
   for (int i = 0; i < 3; i++)
      *reinterpret_cast<uint4 *>(dst + i * planeStride) = make_uint4(w[0][i], w[1][i], w[2][i], w[3][i]);
}

constexpr int kEpiWarps = 8;    // warps 0-7 epilogue: TMEM lane quarter = warp % 4, half of the columns = warp / 4
constexpr int kThreads = 32 * (kEpiWarps + 2);  // warp 8 loads, warp 9 MMA
constexpr int kMaxStages = 3;
constexpr int stages_of(int bn) { return bn <= 64 ? 3 : 2; }  // what fits beside a 128-row operand's planes
constexpr uint32_t kPlaneA = 128 * 128;  // bytes of a 128-row, 64-deep operand plane

// The six plane products, largest first.
__device__ constexpr int kPa[6] = {0, 0, 1, 1, 0, 2}, kPb[6] = {0, 1, 0, 1, 2, 0};

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) {
   const uint32_t a = smem_u32(p);
   return p + ((1024u - (a & 1023u)) & 1023u);
}

// A wait of a kernel of a run: at most kWaitNs, and no longer than a look at the run's error word where it is set,
// so that a run whose first wait gave up ends at once and not after a limit for each of its kernels.
__device__ __forceinline__ bool run_wait(uint64_t *bar, uint32_t parity, const int *err) {
   if (mbar_try_wait(bar, parity)) return true;
   const uint64_t t0 = global_ns();
   for (;;) {
      for (int i = 0; i < 64; i++)
         if (mbar_try_wait(bar, parity)) return true;
      if (*reinterpret_cast<const volatile int *>(err) || global_ns() - t0 > kWaitNs) return false;
   }
}

// The loads, MMAs and epilogue that the two kernels below share: `chunks` stages of operand planes, loaded
// by load(chunk, stage base, full barrier), each multiplied in two halves of K: mma(stage base, half, product,
// accumulator, accumulate).  TMEM columns: the two p0 q0 accumulators, then the small products'.
// early() runs in the epilogue warps while the first products do: it loads what rows() reads beside them;
// late() once the sums have left the registers: it loads what did not fit beside them.
// The sums are staged in shared memory and rows(z) runs over them row by row, so that what the epilogue
// reads and writes in global memory is coalesced (a thread per row cost 11 us more than the GEMM on
// 8192 x 256).  Every wait is bounded; on expiry *err is set, the copies in flight land and the results are
// not written.
template <int kStages>
constexpr int bars_of() {
   return 2 * kStages + 5;
}

template <int BN, int kStages, typename Load, typename Mma, typename Early, typename Late, typename Rows>
__device__ __forceinline__ void pipeline(uint8_t *smem, uint32_t stageBytes, int chunks, int *err, uint32_t *tmemBase,
                                         uint64_t *bars, Load load, Mma mma, Early early, Late late, Rows rows) {
   uint64_t *full = bars, *empty = full + kStages, *accFull = empty + kStages, *accEmpty = accFull + 2, *done = accEmpty + 2;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   // A run that has failed loads nothing more.  The word is read here and looked at by the load lane only, so that
   // the set-up hides the latency (a failure of the kernel just before may go unseen).
   int failed = 0;
   if (warp == kEpiWarps && lane == 0) asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(failed) : "l"(err));
   bool ok = true;
   if (threadIdx.x == 0) {
      for (int i = 0; i < bars_of<kStages>(); i++)
         mbar_init(&bars[i], &bars[i] == accEmpty || &bars[i] == accEmpty + 1 ? kEpiWarps : 1);
      fence_mbar_init();
   }
   if (warp == 0) tmem_alloc(tmemBase, 512);
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem = *tmemBase;
   griddep_launch_dependents();
   griddep_wait();
   constexpr int HALF = BN / 2, RUN = HALF < 32 ? HALF : 32;  // an epilogue warp's columns, columns per TMEM load
   auto load_run = [](uint32_t at, float *v) {
      if constexpr (RUN == 32) tmem_ld32(at, v);
      else tmem_ld16(at, v);
   };
   float acc[HALF];
   if (warp == kEpiWarps) {
      if (lane == 0) {
         ok = failed == 0;
         int issued = 0;
         for (int c = 0; c < chunks && ok; c++) {
            const int s = c % kStages, u = c / kStages;
            if (u > 0 && !(ok = run_wait(&empty[s], (uint32_t)((u - 1) & 1), err))) break;
            mbar_arrive_expect_tx(&full[s], stageBytes);
            load(c, smem + s * stageBytes, &full[s]);
            issued = c + 1;
         }
         if (!ok) mbar_land(full, kStages, issued);  // copies in flight land before the CTA may exit
      }
   } else if (warp == kEpiWarps + 1) {
      if (lane == 0) {
         for (int c = 0; c < chunks && ok; c++) {
            const int s = c % kStages;
            if (!(ok = run_wait(&full[s], (uint32_t)((c / kStages) & 1), err))) break;
            tc_fence_after();
            const uint32_t st = smem_u32(smem + s * stageBytes);
#pragma unroll
            for (int h = 0; h < 2; h++) {
               // chain 2 c + h, accumulator h, once the epilogue has read the chain before in it
               if (c > 0 && !(ok = run_wait(&accEmpty[h], (uint32_t)((c - 1) & 1), err))) break;
               tc_fence_after();
               mma(st, 2 * h, 0, tmem + h * BN, 0u);
               mma(st, 2 * h + 1, 0, tmem + h * BN, 1u);
               mma_commit(&accFull[h]);
#pragma unroll
               for (int k = 0; k < 2; k++)
#pragma unroll
                  for (int q = 1; q < 6; q++) mma(st, 2 * h + k, q, tmem + 2 * BN, (uint32_t)((c | h | k | (q - 1)) != 0));
            }
            if (!ok) break;
            mma_commit(&empty[s]);
         }
         mma_commit(done);
      }
   } else {
      early();
#pragma unroll
      for (int j = 0; j < HALF; j++) acc[j] = 0.0f;
      const uint32_t t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * HALF;
#pragma unroll 1
      for (int d = 0; d < 2 * chunks && ok; d++) {
         if (!(ok = __all_sync(0xffffffffu, run_wait(&accFull[d & 1], (uint32_t)((d >> 1) & 1), err)))) break;
         tc_fence_after();
#pragma unroll
         for (int c = 0; c < HALF; c += RUN) {
            float v[RUN];
            load_run(t + (d & 1) * BN + c, v);
#pragma unroll
            for (int j = 0; j < RUN; j++) acc[c + j] += v[j];
         }
         tc_fence_before();
         __syncwarp();
         if (lane == 0) mbar_arrive(&accEmpty[d & 1]);
      }
   }
   __syncwarp();
   const bool good = __syncthreads_and(ok && mbar_wait(done, 0));
   tc_fence_after();
   constexpr int LZ = BN + 4;
   float *z = reinterpret_cast<float *>(smem);  // the stages are free: every MMA is done
   if (!good) {
      if (threadIdx.x == 0) atomicExch(err, 1);
      if (warp == kEpiWarps && lane == 0 && ok) mbar_land(full, kStages, chunks);
   } else if (warp < kEpiWarps) {
      const uint32_t t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 2 * BN + (warp >> 2) * HALF;
      float *zr = z + (size_t)((warp & 3) * 32 + lane) * LZ + (warp >> 2) * HALF;
#pragma unroll
      for (int c = 0; c < HALF; c += RUN) {
         float v[RUN];
         load_run(t + c, v);
#pragma unroll
         for (int j = 0; j < RUN; j += 4)
            *reinterpret_cast<float4 *>(zr + c + j) = make_float4(acc[c + j] + v[j], acc[c + j + 1] + v[j + 1],
                                                                  acc[c + j + 2] + v[j + 2], acc[c + j + 3] + v[j + 3]);
      }
   }
   if (good && warp < kEpiWarps) late();
   __syncthreads();
   if (good && warp < kEpiWarps) rows(z, LZ);
   tc_fence_before();
   __syncthreads();
   if (warp == 0) tmem_dealloc(tmem, 512);
}

// C[m][n] = sum_k A[m][k] B[n][k]: 128 x BN per CTA, K in chunks of 64.  The epilogue gets four
// neighbouring values of a row at a time (load() what it needs, then finish()).
//
// What bounds it: the operand planes' way from L2 (96 KB per chunk at BN = 128) and the MMAs (1,536
// cycles a chunk) about equally.
template <int BN, typename Epi>
__global__ void __launch_bounds__(kThreads, 1)
      gemm_kernel(const __grid_constant__ CUtensorMap a, const __grid_constant__ CUtensorMap b, int aSlot, int M, int N, int K,
                  Epi epi, int *__restrict__ err) {
   extern __shared__ uint8_t smem_raw[];
   __shared__ __align__(8) uint64_t bars[bars_of<kMaxStages>()];
   __shared__ uint32_t tmemBase;
   constexpr uint32_t planeB = BN * 128, stageBytes = 3 * (kPlaneA + planeB);
   const int m0 = blockIdx.y * 128, n0 = blockIdx.x * BN;
   const int chunks = (K + 63) / 64;
   // an epilogue thread: four columns of every STEP-th row
   constexpr int PER = BN / 4, STEP = 32 * kEpiWarps / PER, ROWS = 128 / STEP;
   const int col = (threadIdx.x % PER) * 4, r0 = threadIdx.x / PER;
   typename Epi::Regs q[ROWS];
   pipeline<BN, stages_of(BN)>(
         align1024(smem_raw), stageBytes, chunks, err, &tmemBase, bars,
         [&](int c, uint8_t *st, uint64_t *bar) {
            load_planes(st, &a, bar, c * 64, m0, aSlot);
            load_planes(st + 3 * kPlaneA, &b, bar, c * 64, n0, 0);
         },
         [&](uint32_t st, int k, int q, uint32_t d, uint32_t accumulate) {
            mma_bf16(d, sdesc_sw128(st + kPa[q] * kPlaneA + k * 32), sdesc_sw128(st + 3 * kPlaneA + kPb[q] * planeB + k * 32),
                     idesc_bf16(128, BN), accumulate);
         },
         [&]() {
            if (n0 + col >= N) return;
#pragma unroll
            for (int i = 0; i < ROWS; i++)
               if (m0 + r0 + i * STEP < M) epi.load(q[i], (size_t)(m0 + r0 + i * STEP) * N + n0 + col);
         },
         [&]() {
            if (n0 + col >= N) return;
#pragma unroll
            for (int i = 0; i < ROWS; i++)
               if (m0 + r0 + i * STEP < M) epi.late(q[i], (size_t)(m0 + r0 + i * STEP) * N + n0 + col);
         },
         [&](const float *z, int lz) {
            if (n0 + col >= N) return;
#pragma unroll
            for (int i = 0; i < ROWS; i++) {
               const int r = r0 + i * STEP;
               if (m0 + r < M)
                  epi.finish(q[i], *reinterpret_cast<const float4 *>(z + r * lz + col), (size_t)(m0 + r) * N + n0 + col);
            }
         });
}

// P[s][f][k] += sum over positions m of split s of A[m][f] B[m][k]: the correlation over positions, both
// operands read MN-major from their [position][column] planes.  CTA = (128 f) x (128 k) of one of `pairs`
// operand pairs and one of `splits` ranges of positions; each adds its own partial matrix, so the sum's
// order is fixed.
struct CorrArgs {
   int slotA[2], slotB[2];
   int pair0;             // first operand pair of this launch
   int M, F, KP, mt, nt, splits;
   float *P;              // [2 pairs][splits][F][KP]
};

__global__ void __launch_bounds__(kThreads, 1)
      corr_kernel(const __grid_constant__ CUtensorMap a0, const __grid_constant__ CUtensorMap b0,
                  const __grid_constant__ CUtensorMap a1, const __grid_constant__ CUtensorMap b1, CorrArgs g,
                  int *__restrict__ err) {
   extern __shared__ uint8_t smem_raw[];
   __shared__ __align__(8) uint64_t bars[bars_of<kMaxStages>()];
   __shared__ uint32_t tmemBase;
   // a stage: two column halves of A, then of B, each three planes of 64 positions x 64 columns
   constexpr uint32_t kBox = 64 * 128, kHalf = 3 * kBox;
   int u = blockIdx.x;
   const int ks = u % g.splits;
   u /= g.splits;
   const int nt = u % g.nt;
   u /= g.nt;
   const int mt = u % g.mt, pair = g.pair0 + u / g.mt;
   const int all = (g.M + 63) / 64, c0 = (int)((int64_t)all * ks / g.splits), chunks = (int)((int64_t)all * (ks + 1) / g.splits) - c0;
   if (chunks == 0) return;  // CTA-uniform, before any barrier
   const CUtensorMap *A = pair ? &a1 : &a0, *B = pair ? &b1 : &b0;
   const int slotA = g.slotA[pair], slotB = g.slotB[pair];
   // an epilogue thread: four columns of every eighth row of the partial matrix
   static_assert(kEpiWarps == 8, "eight rows per step");
   const int col = (threadIdx.x & 31) * 4, r0 = threadIdx.x >> 5;
   float *out = g.P + (((size_t)pair * g.splits + ks) * g.F + mt * 128) * g.KP + nt * 128 + col;
   float4 o[16];
   pipeline<128, 2>(
         align1024(smem_raw), 4 * kHalf, chunks, err, &tmemBase, bars,
         [&](int c, uint8_t *st, uint64_t *bar) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
               load_planes(st + h * kHalf, A, bar, mt * 128 + h * 64, (c0 + c) * 64, slotA);
               load_planes(st + (2 + h) * kHalf, B, bar, nt * 128 + h * 64, (c0 + c) * 64, slotB);
            }
         },
         [&](uint32_t st, int k, int q, uint32_t d, uint32_t accumulate) {
            constexpr uint32_t idesc = idesc_bf16(128, 128) | (1u << 15) | (1u << 16);  // both operands MN-major
            mma_bf16(d, sdesc_sw128_mn(st + kPa[q] * kBox + k * 2048, kHalf),
                     sdesc_sw128_mn(st + 2 * kHalf + kPb[q] * kBox + k * 2048, kHalf), idesc, accumulate);
         },
         [&]() {
            if (nt * 128 + col >= g.KP) return;
#pragma unroll
            for (int i = 0; i < 16; i++)
               if (mt * 128 + r0 + i * 8 < g.F) o[i] = *reinterpret_cast<const float4 *>(out + (size_t)(r0 + i * 8) * g.KP);
         },
         [] {},
         [&](const float *z, int lz) {
            if (nt * 128 + col >= g.KP) return;
#pragma unroll
            for (int i = 0; i < 16; i++) {
               const int r = r0 + i * 8;
               if (mt * 128 + r < g.F) {
                  const float4 v = *reinterpret_cast<const float4 *>(z + r * lz + col);
                  *reinterpret_cast<float4 *>(out + (size_t)r * g.KP) =
                        make_float4(o[i].x + v.x, o[i].y + v.y, o[i].z + v.z, o[i].w + v.w);
               }
            }
         });
}

}  // namespace split
}  // namespace pvgpu
