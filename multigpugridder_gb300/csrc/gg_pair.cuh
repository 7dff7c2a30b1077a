// Precomp factors as float pairs (hi + lo = the FP64 value to 48 bits); their
// products keep the pair, so the one rounding to FP32 at the end is the FP64
// product's but for ties.
#pragma once

namespace gg {

struct FF {
    float h, l;
};
__device__ __forceinline__ FF ff_mul(FF a, FF b)
{
    const float p = __fmul_rn(a.h, b.h);
    const float e = __fmaf_rn(a.h, b.h, -p) + (a.h * b.l + a.l * b.h);
    const float s = __fadd_rn(p, e);
    return FF{s, __fsub_rn(e, __fsub_rn(s, p))};
}
__device__ __forceinline__ FF ff_at(const float2 *__restrict__ pc, int i)
{
    const float2 v = __ldg(pc + i);
    return FF{v.x, v.y};
}
// x * f, f a pair, rounded once
__device__ __forceinline__ float ff_scale(float x, FF f)
{
    const float p = __fmul_rn(x, f.h);
    return __fadd_rn(p, __fmaf_rn(x, f.h, -p) + x * f.l);
}

} // namespace gg
