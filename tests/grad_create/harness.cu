// pvgpu_lca_grad_create on the host: device allocations come from a counter with a budget (nothing is touched),
// cuBLAS is tests/grad_create/fake_cublas.cpp, which asks this program whether each operand lies in one
// allocation.  Reads lines "budgetMB nb inNx inNy inNf v1Nx v1Ny v1Nf nxp VThresh steps every", prints per line
// "status bad peakMB left path": operands outside their allocation, the most allocated, allocations left after
// destroy, 1 for the split-plane path, 0 for library GEMMs.
#include "pvgpu_internal.cuh"
#include "tmap.cuh"

#include <algorithm>
#include <cstdio>
#include <map>

namespace {
std::map<uintptr_t, size_t> g_blocks;
size_t g_used = 0, g_peak = 0, g_budget = 0;
uintptr_t g_next = 1u << 20;
int g_bad = 0;

cudaError_t host_malloc(void **p, size_t n) {
   if (g_used + n > g_budget) return cudaErrorMemoryAllocation;
   g_blocks[g_next] = n;
   *p = reinterpret_cast<void *>(g_next);
   g_next += (n + 4095) / 4096 * 4096 + 4096;
   g_used += n;
   g_peak = std::max(g_peak, g_used);
   return cudaSuccess;
}
template <typename T>
cudaError_t host_malloc(T **p, size_t n) {
   return host_malloc(reinterpret_cast<void **>(p), n);
}
cudaError_t host_free(void *p) {
   auto it = g_blocks.find(reinterpret_cast<uintptr_t>(p));
   if (it == g_blocks.end()) {
      g_bad++;
      return cudaErrorInvalidValue;
   }
   g_used -= it->second;
   g_blocks.erase(it);
   return cudaSuccess;
}
}  // namespace

extern "C" void harness_operand(const void *p, size_t bytes) {
   const uintptr_t a = reinterpret_cast<uintptr_t>(p);
   auto it = g_blocks.upper_bound(a);
   if (it == g_blocks.begin()) {
      g_bad++;
      return;
   }
   --it;
   if (a + bytes > it->first + it->second) g_bad++;
}

namespace pvgpu {
pvgpu_status record_cuda_error(cudaError_t, const char *) { return PVGPU_ERR_LAUNCH; }
pvgpu_status record_message(pvgpu_status s, const char *) { return s; }
int num_sms() { return 152; }
inline EncodeTiledFn host_encode_tiled_fn() {
   return [](CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
             CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; };
}
}  // namespace pvgpu

#define encode_tiled_fn host_encode_tiled_fn
#define cudaMalloc host_malloc
#define cudaFree host_free
#define cudaFuncSetAttribute(...) cudaSuccess
#include "lca_grad.cu"

int main() {
   double budget, vt;
   pvgpu_lca_grad_desc d;
   while (std::scanf("%lf %d %d %d %d %d %d %d %d %lf %d %d", &budget, &d.nbatch, &d.inNx, &d.inNy, &d.inNf, &d.v1Nx, &d.v1Ny,
                     &d.v1Nf, &d.nxp, &vt, &d.steps, &d.checkpointEvery) == 12) {
      d.VThresh = (float)vt;
      d.lambda1 = 0.1f;
      d.tau = 100.0f;
      d.dt = 1.0f;
      g_budget = (size_t)(budget * 1e6);
      g_bad = 0;
      g_peak = g_used;
      pvgpu_lca_grad *h = nullptr;
      const pvgpu_status st = pvgpu_lca_grad_create(&d, &h);
      const int emulated = h ? (int)h->tc : -1;
      const double peak = g_peak / 1e6;
      if (h) pvgpu_lca_grad_destroy(h);
      std::printf("%d %d %.1f %zu %d\n", (int)st, g_bad, peak, g_blocks.size(), emulated);
   }
}
