// stats.cuh -- reduction of the row pass's per-CTA statistics: compensated float-float sums
// (TwoSum) for the energies, maxima for the norms, in a fixed order.
#pragma once
#include "engine.h"

namespace fm {

namespace {

// butterfly all-reduce of a float-float value; every lane ends with the same bits
// because each level combines the pair in lane order
__device__ __forceinline__ void warp_ff_sum(float &h, float &l) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, h, o);
        const float ol = __shfl_xor_sync(0xffffffffu, l, o);
        const bool low = (threadIdx.x & o) == 0;
        float ah = low ? h : oh, al = low ? l : ol;
        const float bh = low ? oh : h, bl = low ? ol : l;
        ff_add(ah, al, bh);
        h = ah;
        l = al + bl;
    }
}
__device__ __forceinline__ float warp_maxf(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Statistic s of nblk CTAs by one warp: lanes stride over the CTAs, one butterfly.  The same
// bits whichever warp of whichever kernel runs it.
__device__ __forceinline__ void finalize_stat(const float2 *__restrict__ partials, int nblk, int s, double *out) {
    const int lane = threadIdx.x & 31;
    float h = 0.f, l = 0.f;
    for (int b = lane; b < nblk; b += 32) {
        const float2 v = __ldcg(partials + (size_t)s * nblk + b);
        if (s < 5) {
            ff_add(h, l, v.x);
            l += v.y;
        } else {
            h = fmaxf(h, v.x);
        }
    }
    if (s < 5) warp_ff_sum(h, l);
    else h = warp_maxf(h);
    if (lane == 0) out[s] = (double)h + (double)l;
}

}  // namespace

}  // namespace fm
