// Device helpers shared by the projection kernels (gg_project.cu,
// gg_fp_tile.cu, gg_adjoint.cu).
#pragma once

#include "gg_common.cuh"

namespace gg {

// Sample point of pixel (di, dj) (offsets from the image centre) in the CAS
// volume frame: the reference's nx*di + ny*dj + volCenter
// (gpuForwardProject.cu:53-55) as its build evaluates it, fma(nx, di, ny*dj) +
// vc, written with round-to-nearest intrinsics so the grouping cannot change.
// Shared by the forward and adjoint kernels so both see identical bits.
__device__ __forceinline__ float sample_coord(float n_x, float n_y, int di, int dj, int vc)
{
    return __fadd_rn(__fmaf_rn(n_x, (float)di, __fmul_rn(n_y, (float)dj)), (float)vc);
}

// Table lookup of the reference's nearest-index KB rule,
// ker[roundf(fma(r, kerScale, kerCenter))], as floor(fma(r, kerScale,
// kerCenter + 1/2)): equal for every float r in [-2, 2] (checked
// exhaustively) and one conversion instead of a roundf and a conversion.
// Callers pass r in [-2, 2]; the clamp only keeps a NaN or infinite
// coordinate (bad axes) inside the table.  Entry k is read at sker[k * rep]
// (rep interleaved copies).
__device__ __forceinline__ float kb_weight(const float *sker, float r, float kerScale, float kerCenterHalf, int kerSize,
                                           int rep = 1)
{
    return sker[min(max(__float2int_rd(__fmaf_rn(r, kerScale, kerCenterHalf)), 0), kerSize - 1) * rep];
}

__device__ __forceinline__ void load_table(float *sker, const float *ker, int kerSize)
{
    for (int t = threadIdx.x; t < kerSize; t += blockDim.x) sker[t] = __ldg(ker + t);
}

} // namespace gg
