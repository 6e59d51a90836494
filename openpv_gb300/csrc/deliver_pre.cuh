// deliver_pre.cuh -- geometry shared by the presynaptic delivery kernels: the reference-order tile
// kernel (deliver_pre.cu) and the FAST kernels (deliver_pre_fast.cu).
#pragma once

#include "pvgpu_internal.cuh"

namespace pvgpu {

struct PreGeom {
   Loc pre, post;
   Axis ax, ay;
   int nxp, nyp, nfp;
   int nkx, nky, nkf;
   int patchSize;
   int TX, FT;  // tile columns, tile features (the tile kernel)
   float dtf;
};

// FAST mode; PVGPU_ERR_UNSUPPORTED_SHAPE for a shape that neither FAST kernel takes.
pvgpu_status deliver_pre_fast(const PreGeom &g, const pvgpu_entry *entries, const int64_t *numActive,
                              const float *aExt, const float *W, float *gsyn, cudaStream_t s);

}  // namespace pvgpu
