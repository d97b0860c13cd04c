// Per-pixel device code shared by the compositor kernels.
#pragma once

#include "common.cuh"

namespace gstex {

// Completes a Hit in the direct form, rebuilding the Gaussian's camera-space
// frame from its parameters (rare: splats at the camera plane and pixels within
// the reference's denominator clamp).
__device__ __forceinline__ void direct_hit(Hit& H, const float4* __restrict__ quats, const float3* __restrict__ means,
                                           const float* __restrict__ scales, float glob, const float2* __restrict__ uv0s,
                                           const float3* __restrict__ umaps, const float3* __restrict__ vmaps,
                                           const View& V, int gid, const PixelRay& P, float tvn) {
    const Axes A = quat_axes(quats[gid]);
    const float3 mc = V.xform(means[gid]);
    const float is1 = 1.f / (scales[3 * (size_t)gid] * glob), is2 = 1.f / (scales[3 * (size_t)gid + 1] * glob);
    const float2 uv0 = uv0s[gid];
    intersect_direct(H, P, tvn, mc, V.rot(A.a1), V.rot(A.a2), V.rot(A.a3), V.rot(umaps[gid]), V.rot(vmaps[gid]), is1,
                     is2, uv0.x, uv0.y);
}

// All channels of the 4 bilinear corners (C == 3 fast path).
template <int TEXMODE>
__device__ __forceinline__ void fetch3(const void* tex, const Bilerp& B, float c[4][3]) {
    const int rows[4] = { B.i00, B.i01, B.i10, B.i11 };
    if (TEXMODE == 1) {
        const uint2* t = (const uint2*)tex;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint2 raw = __ldg(t + rows[q]);
            const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
            const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
            c[q][0] = __low2float(lo);
            c[q][1] = __high2float(lo);
            c[q][2] = __low2float(hi);
        }
    } else {
        // (3 times a row passes 31 bits from 716M texels on)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float* t = (const float*)tex + 3 * (size_t)rows[q];
            c[q][0] = __ldg(t + 0);
            c[q][1] = __ldg(t + 1);
            c[q][2] = __ldg(t + 2);
        }
    }
}

template <typename T>
__device__ __forceinline__ T ld_or(const T* p, size_t i, T z) {
    return p ? p[i] : z;
}

// Blur moments -> world-space mean gradient (helpers.cuh:155-164, 114-121);
// p: the camera-space mean.
__device__ __forceinline__ float3 blur_mean_grad(const View& V, float3 p, float mx, float my) {
    const float rw = 1.f / (p.z + 1e-6f);
    const float vx = V.fx * mx, vy = V.fy * my;
    return V.rot_t(make_float3(vx * rw, vy * rw, -(vx * p.x + vy * p.y) * rw * rw));
}

}  // namespace gstex
