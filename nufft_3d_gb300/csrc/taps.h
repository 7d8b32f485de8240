// The neighbour test and weight of one (sample, grid point) pair for the
// stored tables, from the signed distances per axis.  The distance is formed
// with explicitly rounded operations (never contracted into FMAs), so passes
// that are compiled separately (count and fill) take identical decisions.
#pragma once

#include "internal.h"

namespace nufft3d {

struct TapDist {
    float x2, y2, z2;
};

__device__ __forceinline__ TapDist tap_dist(float ex, float ey, float ez)
{
    return {__fmul_rn(ex, ex), __fmul_rn(ey, ey), __fmul_rn(ez, ez)};
}

__device__ __forceinline__ float tap_d2(const TapDist &t) { return __fadd_rn(__fadd_rn(t.z2, t.y2), t.x2); }

// nufft_3d.m:183-192: 4 dist2 <= J^2, or per axis for the separable kernel
__device__ __forceinline__ bool tap_inside(const TapDist &t, const KBParams &kb, int radial)
{
    const float h2 = kb.half2;
    return radial ? tap_d2(t) <= h2 : t.x2 <= h2 && t.y2 <= h2 && t.z2 <= h2;
}

__device__ __forceinline__ float tap_value(const TapDist &t, const KBParams &kb, int radial)
{
    if (radial) return kb_weight(tap_d2(t), kb);
    return __fmul_rn(__fmul_rn(kb_weight(t.z2, kb), kb_weight(t.y2, kb)), kb_weight(t.x2, kb));
}

}  // namespace nufft3d
