// Shared device code of the gstex_gb300 library (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <utility>
#include <cuda_bf16.h>
#include <stdint.h>

#include "../../include/gstex_gb300.h"

namespace gstex {

constexpr int kMaxChannels = 64;
constexpr int kMaxBlockWidth = 16;

// Reference float constants (csrc/texture.cu:198, 213-217; texture_helpers.cuh:305)
constexpr float kTNear = 0.01f;
constexpr float kTFar = 1000.0f;
constexpr float kAlphaMax = 0.99f;
constexpr float kAlphaMin = 1.f / 255.f;
constexpr float kTDone = 1e-4f;
constexpr float kDenomEps = 1e-6f;
constexpr float kBlurFsq = 2.0f;

// Host-side status helpers (defined in status.cu).
int check_launch(const char* what, int launches = 1);
void set_cuda_error(cudaError_t e, const char* what);

#define GSTEX_REQUIRE(cond)                         \
    do {                                            \
        if (!(cond)) return GSTEX_ERR_INVALID_ARGUMENT; \
    } while (0)

// (a >= 0; a + b - 1 could pass 31 bits)
__host__ __device__ inline int ceil_div(int a, int b) { return a / b + (a % b > 0); }

// ---------------------------------------------------------------------------
// quaternion (w, x, y, z) -> columns ax1, ax2, ax3 of the rotation
// (reference csrc/helpers.cuh:166-185)
// ---------------------------------------------------------------------------
struct Axes {
    float3 a1, a2, a3;
};

__device__ __forceinline__ Axes quat_axes(float4 q) {
    const float w = q.x, x = q.y, y = q.z, z = q.w;
    Axes A;
    A.a1 = make_float3(1.f - 2.f * (y * y + z * z), 2.f * (x * y + w * z), 2.f * (x * z - w * y));
    A.a2 = make_float3(2.f * (x * y - w * z), 1.f - 2.f * (x * x + z * z), 2.f * (y * z + w * x));
    A.a3 = make_float3(2.f * (x * z + w * y), 2.f * (y * z - w * x), 1.f - 2.f * (x * x + y * y));
    return A;
}

// d(R(q)) adjoint for gradients vR = columns (v_a1, v_a2, v_a3)
// (reference csrc/helpers.cuh:187-228)
__device__ __forceinline__ float4 quat_axes_vjp(float4 q, float3 c0, float3 c1, float3 c2) {
    const float w = q.x, x = q.y, y = q.z, z = q.w;
    const float r00 = c0.x, r01 = c0.y, r02 = c0.z;
    const float r10 = c1.x, r11 = c1.y, r12 = c1.z;
    const float r20 = c2.x, r21 = c2.y, r22 = c2.z;
    float4 o;
    o.x = 2.f * (x * (r12 - r21) + y * (r20 - r02) + z * (r01 - r10));
    o.y = 2.f * (-2.f * x * (r11 + r22) + y * (r01 + r10) + z * (r02 + r20) + w * (r12 - r21));
    o.z = 2.f * (x * (r01 + r10) - 2.f * y * (r00 + r22) + z * (r12 + r21) + w * (r20 - r02));
    o.w = 2.f * (x * (r02 + r20) + y * (r12 + r21) - 2.f * z * (r00 + r11) + w * (r01 - r10));
    return o;
}

__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 operator*(float s, float3 a) { return make_float3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }

// World->camera view transform (row-major 4x4, first 12 entries used).
struct View {
    float r[9];
    float t[3];
    float fx, fy, cx, cy;
    __device__ __forceinline__ float3 rot(float3 p) const {
        return make_float3(r[0] * p.x + r[1] * p.y + r[2] * p.z, r[3] * p.x + r[4] * p.y + r[5] * p.z,
                           r[6] * p.x + r[7] * p.y + r[8] * p.z);
    }
    __device__ __forceinline__ float3 rot_t(float3 p) const {
        return make_float3(r[0] * p.x + r[3] * p.y + r[6] * p.z, r[1] * p.x + r[4] * p.y + r[7] * p.z,
                           r[2] * p.x + r[5] * p.y + r[8] * p.z);
    }
    __device__ __forceinline__ float3 xform(float3 p) const {
        return make_float3(r[0] * p.x + r[1] * p.y + r[2] * p.z + t[0], r[3] * p.x + r[4] * p.y + r[5] * p.z + t[1],
                           r[6] * p.x + r[7] * p.y + r[8] * p.z + t[2]);
    }
};

__device__ __forceinline__ View load_view(const float* viewmat, float fx, float fy, float cx, float cy) {
    View v;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        v.r[3 * i + 0] = viewmat[4 * i + 0];
        v.r[3 * i + 1] = viewmat[4 * i + 1];
        v.r[3 * i + 2] = viewmat[4 * i + 2];
        v.t[i] = viewmat[4 * i + 3];
    }
    v.fx = fx; v.fy = fy; v.cx = cx; v.cy = cy;
    return v;
}

// ---------------------------------------------------------------------------
// Per-view, per-Gaussian record staged in shared memory by the compositor.
//
// The reference intersects every pixel ray with the splat plane in world
// space (texture_helpers.cuh:302-313 then texture.cu:171-181).  Here the same
// intersection is evaluated in camera space relative to the projected centre
// d0 = mu_c / mu_c.z: for a pixel direction d = d0 + e (e = (du/fx, dv/fy, 0))
//   den   = n_c . d                 = g + nu*du + nv*dv
//   t_cam = (n_c . mu_c) / den      = tvn / den         (camera z of the hit)
//   delta = t_cam d - mu_c          = mu_z (g e - (n_c.e) d0) / den
//   l_k   = a_k . delta             = (Pku*du + Pkv*dv) / den
// which has no cancellation between the camera distance and the splat size.
// Gaussians with mu_z <= 0.01 (only reachable through the reference's
// zero-slot entries) and pixels whose ray is within the reference's 1e-6
// denominator clamp use the direct camera-space form instead.
//
// The record also carries a conservative screen box of the region where the
// splat can reach alpha >= 1/255: sigma <= ln(255 * opacity) is an ellipse
// in the splat plane, inside the rectangle +-a*s1*ax1 +-a*s2*ax2 with
// a = sqrt(2 ln(255 opacity)) (inflated slightly; a parallelogram for a
// quaternion that is not of unit length); when all four corners are
// in front of the camera the projected rectangle, hence the box of its
// projected corners, contains every pixel whose ray meets the ellipse.  A
// pixel outside the box is a pixel the reference skips (alpha < 1/255).
//
// Fields are grouped by how often the per-pixel loop reads them.
// ---------------------------------------------------------------------------
struct RecHot {   // every (pixel, Gaussian) pair
    float4 box;   // screen box of alpha >= 1/255: x0, x1, y0, y1 (one load for the per-visit test)
    float4 org;   // px0, py0, g, tvn
    float4 lc;    // p1u, p1v, p2u, p2v (scaled by 1 / (scale * glob_scale))
    float4 nop;   // nu, nv, opacity, flags (int bits; bit 0: direct form only)
};
struct RecWarm {  // pairs that pass the alpha test
    float4 uvm;   // uu, uv_, vu, vv: texture uv numerators
    float4 uvs;   // uv0.x, uv0.y, blur centre x, blur centre y
    float4 col;   // colour rgb, 1 / (scale_x * glob_scale)
    float4 nrm;   // world normal (axis 3), 1 / (scale_y * glob_scale)
    int4 tex;     // chart h, w, start, Gaussian id
};
struct RecCold {  // the backward's ray terms and the blur adjoint
    float4 mu;    // camera-space mean, a1 . mean
    float4 dt;    // a2 . mean, umap . mean, vmap . mean (camera space), unused
};
constexpr int kRecBytes = sizeof(RecHot) + sizeof(RecWarm) + sizeof(RecCold);

// The alpha >= 1/255 region of a splat as pixel rows see it: at height y, with
// u = (y - yc) / hy, the region lies inside xc + m (y - yc) +- s sqrt(1 - u^2)
// (an ellipse) or xc +- s (a box), and only rows with |u| <= 1 meet it.  The
// image of the ellipse sigma <= ln(255 opacity) is an ellipse when the splat's
// rectangle is in front of the camera; where that form does not apply (an
// infinite screen box, blur, a strong perspective) the screen box takes its
// place, and a region that no pixel meets has s < 0.  16 bytes, one load: s
// and 1 / hy are rounded to bfloat16 such that the region only grows; m, whose
// error would move a sliver's ends sideways, keeps all but its last bit.
struct RecCull {
    float xc, yc;
    uint32_t ms;  // m (upper half), s
    uint32_t hk;  // 1 / hy, m (lower half but for its last bit), 1 for an ellipse
};

// One (view, Gaussian) record as it is stored in device memory: built once per
// view by the record kernel (where the near-edge-on solve runs in double), then
// read by every tile the splat touches.  224 bytes, in 16-byte chunks ordered
// by who reads them, so that each reader takes whole 32-byte sectors: the cull
// test chunk 0, the block kernels' forward 2-8 and backward 2-9.
enum RecChunk {
    kChunkCull = 0,   // RecCull (chunk 1 is unused)
    kChunkOrg = 2,    // px0, py0, g (NaN: direct form only), tvn
    kChunkLc = 3,     // p1u, p1v, p2u, p2v
    kChunkNop = 4,    // nu, nv, opacity, chart start (31 bits) and kCoarseChart
    kChunkUvm = 5,    // texture uv numerators
    kChunkUvs = 6,    // uv0.x, uv0.y, chart h, w (ints)
    kChunkCol = 7,    // colour, 1 / (scale_x glob)
    kChunkNrm = 8,    // world normal, 1 / (scale_y glob)
    kChunkRay = 9,    // a1.mu / s1, a2.mu / s2, umap.mu, vmap.mu (camera space)
    kChunkMisc = 10,  // blur centre x, y, flags, Gaussian id (ints)
    kChunkBox = 11,   // screen box
    kChunkMu = 12,    // camera-space mean, a1 . mean
    kChunkDt = 13,    // a2 . mean, umap . mean, vmap . mean
    kRecChunks = 14
};
// Set where a texel of the chart is kCoarsePixels wide or more: the pixels of a
// block then mostly share their four texels, and the backward adds up their
// gradients before it touches memory.  Backward of a full-HD view with 48 pixels
// a texel, 800x800 with 1x1 charts (2 to 15 pixels), 32 views with 1.7 pixels:
// never 27.4 ms, 122 us, 25.4 ms; from 24 pixels on 14.8, 122, 25.4; from 12 on
// 13.8, 138, 25.4; from 6 on 13.7, 166, 25.4; from 3 on 13.7, 185, 28.8.
constexpr uint32_t kCoarseChart = 0x80000000u;
constexpr float kCoarsePixels = 16.f;
struct __align__(16) RecAll {
    float4 c[kRecChunks];
};
static_assert(sizeof(RecAll) == 224, "record layout");

struct Recs {
    RecHot* hot;
    RecWarm* warm;
    RecCold* cold;
    RecCull* cull;  // null when the kernel does not stage it
    __device__ __forceinline__ static Recs carve(unsigned char* smem, int n, bool with_cull) {
        Recs r;
        r.hot = reinterpret_cast<RecHot*>(smem);
        r.warm = reinterpret_cast<RecWarm*>(smem + sizeof(RecHot) * n);
        r.cold = reinterpret_cast<RecCold*>(smem + (sizeof(RecHot) + sizeof(RecWarm)) * n);
        r.cull = with_cull ? reinterpret_cast<RecCull*>(smem + (size_t)kRecBytes * n) : nullptr;
        return r;
    }
};

__device__ __forceinline__ float4 f4(float3 v, float w) { return make_float4(v.x, v.y, v.z, w); }
__device__ __forceinline__ float3 f3(float4 v) { return make_float3(v.x, v.y, v.z); }

// Pairs of fp32 values in one instruction (the f32x2 add / mul / fma of this
// GPU): each half is the IEEE fp32 operation, rounded to nearest; fma2 is a
// fused multiply-add per half.
__device__ __forceinline__ unsigned long long pack2(float2 a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r) {
    float2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)), "l"(pack2(c)));
    return unpack2(r);
}
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }

// Near-edge-on splats (|n_c . d0| < kEdgeOn): the plane coefficients in
// double.  Writes H.org, H.nop.x/.y, H.lc and Wm.uvm.
constexpr float kEdgeOn = 0.05f;
__device__ __forceinline__ void edge_on_solve(RecHot& H, RecWarm& Wm, const View& V, float3 mc, float3 a1c,
                                              float3 a2c, float3 nc, float3 umc, float3 vmc, float is1, float is2,
                                              float tvn) {
    const double mz = mc.z, imz = 1.0 / mz;
    const double u0 = (double)mc.x * imz, v0 = (double)mc.y * imz;
    const double g = (double)nc.x * u0 + (double)nc.y * v0 + nc.z;
    const double ifx = 1.0 / V.fx, ify = 1.0 / V.fy;
    const double a1d = a1c.x * u0 + a1c.y * v0 + a1c.z, a2d = a2c.x * u0 + a2c.y * v0 + a2c.z;
    const double umd = umc.x * u0 + umc.y * v0 + umc.z, vmd = vmc.x * u0 + vmc.y * v0 + vmc.z;
    H.org = make_float4((float)(V.fx * u0 + V.cx), (float)(V.fy * v0 + V.cy), (float)g, tvn);
    H.nop.x = (float)(nc.x * ifx);
    H.nop.y = (float)(nc.y * ify);
    H.lc = make_float4((float)(mz * (g * a1c.x - a1d * nc.x) * ifx * is1),
                      (float)(mz * (g * a1c.y - a1d * nc.y) * ify * is1),
                      (float)(mz * (g * a2c.x - a2d * nc.x) * ifx * is2),
                      (float)(mz * (g * a2c.y - a2d * nc.y) * ify * is2));
    Wm.uvm = make_float4((float)(mz * (g * umc.x - umd * nc.x) * ifx), (float)(mz * (g * umc.y - umd * nc.y) * ify),
                         (float)(mz * (g * vmc.x - vmd * nc.x) * ifx), (float)(mz * (g * vmc.y - vmd * nc.y) * ify));
}

// s rounded away from zero, ih towards zero.
__device__ __forceinline__ RecCull pack_cull(float xc, float yc, float m, float s, float ih, bool ellipse) {
    RecCull c;
    c.xc = xc;
    c.yc = yc;
    c.ms = (__float_as_uint(m) & 0xffff0000u) | ((__float_as_uint(s) + 0xffffu) >> 16);
    c.hk = (__float_as_uint(ih) & 0xffff0000u) | (__float_as_uint(m) & 0xfffeu) | (ellipse ? 1u : 0u);
    return c;
}

// Rows of the screen box x0..x1, y0..y1 (infinite or empty ones included).
__device__ __forceinline__ RecCull cull_box(float x0, float x1, float y0, float y1) {
    if (x0 > x1) return pack_cull(0.f, 0.f, 0.f, -1.f, 0.f, false);
    if (!(fabsf(x0) < 1e30f && fabsf(x1) < 1e30f && fabsf(y0) < 1e30f && fabsf(y1) < 1e30f))
        return pack_cull(0.f, 0.f, 0.f, INFINITY, 0.f, false);
    // (the half sizes cover the rounding of the middle)
    const float mx = 1e-3f + 1e-6f * (fabsf(x0) + fabsf(x1)), my = 1e-3f + 1e-6f * (fabsf(y0) + fabsf(y1));
    return pack_cull(0.5f * (x0 + x1), 0.5f * (y0 + y1), 0.f, 0.5f * (x1 - x0) + mx, 0.99999f / (0.5f * (y1 - y0) + my),
                     false);
}

// Image of the plane ellipse mu + e1 cos(t) a1 + e2 sin(t) a2 (for any two a).  With u_i the
// homogeneous images of the axes relative to the projected centre (px0, py0),
// its tangent lines satisfy l^T D l = 0, D = e1^2 u1 u1^T + e2^2 u2 u2^T -
// u0 u0^T, u0 = (0, 0, z); scaled to D_zz = -1, D is [S - c c^T, -c; -c^T, -1]
// with the ellipse's centre c and its second moments S, sums of squares
// without cancellation.  S is widened so that the region grows by at least
// `eps` pixels on every side: the per-pixel evaluation rounds the projected
// centre to single precision, a thin sliver's half width may be less.
// Returns false where a corner comes near the camera plane (D_zz cancels).
__device__ __forceinline__ bool cull_ellipse(RecCull& c, const View& V, float3 mc, float u0, float v0, float3 a1,
                                             float3 a2, float e1, float e2) {
    const float x1 = e1 * V.fx * (a1.x - u0 * a1.z), y1 = e1 * V.fy * (a1.y - v0 * a1.z), z1 = e1 * a1.z;
    const float x2 = e2 * V.fx * (a2.x - u0 * a2.z), y2 = e2 * V.fy * (a2.y - v0 * a2.z), z2 = e2 * a2.z;
    const float k = mc.z * mc.z - (z1 * z1 + z2 * z2);
    if (!(k > 0.05f * mc.z * mc.z)) return false;
    const float ik = 1.f / k;
    const float cx = -(x1 * z1 + x2 * z2) * ik, cy = -(y1 * z1 + y2 * z2) * ik;
    float sxx = (x1 * x1 + x2 * x2) * ik + cx * cx, syy = (y1 * y1 + y2 * y2) * ik + cy * cy;
    const float sxy = (x1 * y1 + x2 * y2) * ik + cx * cy;
    const float px0 = V.fx * u0 + V.cx, py0 = V.fy * v0 + V.cy;
    const float reach = sqrtf(sxx + syy);
    const float eps = 5e-4f + 5e-7f * (fabsf(px0) + fabsf(py0)) + 2e-6f * reach;
    const float grow = 2.f * reach * eps + eps * eps;
    sxx += grow;
    syy += grow;
    const float m = sxy / syy, w = sxx - sxy * m, hy = sqrtf(syy);
    if (!(w > 0.f && sxx < 1e12f && syy < 1e12f)) return false;
    c = pack_cull(px0 + cx, py0 + cy, m, sqrtf(w) * 1.0001f, 0.9999f / hy, true);
    return true;
}

// One row of a region: its middle and half width there; false if the region
// does not meet the row.
__device__ __forceinline__ bool cull_span(const RecCull& c, float y, float& mid, float& half) {
    const float dy = y - c.yc, u = dy * __uint_as_float(c.hk & 0xffff0000u);
    const float q = 1.f - u * u;
    mid = c.xc + __uint_as_float((c.ms & 0xffff0000u) | (c.hk & 0xfffeu)) * dy;
    half = __uint_as_float(c.ms << 16) * sqrtf((c.hk & 1u) ? fmaxf(q, 0.f) : 1.f) + 1e-3f;
    return q >= 0.f;
}

// Columns [0, 8) of one row that a region can reach, as a bit mask: x0 is the
// centre of column 0, y the row's centre.
__device__ __forceinline__ unsigned cull_row(const RecCull& c, float x0, float y) {
    float mid, half;
    const bool meets = cull_span(c, y, mid, half);
    mid -= x0;
    const int lo = min(max(__float2int_ru(mid - half), 0), 8), hi = min(max(__float2int_rd(mid + half), -1), 7) + 1;
    const unsigned bits = ((1u << hi) - 1u) & ~((1u << lo) - 1u);
    return meets ? bits : 0u;
}

__device__ __forceinline__ bool make_record(RecHot& H, RecWarm& Wm, RecCold& Cd, int gid, const View& V,
                                            const float3 mean, const float4 quat, const float2 scale,
                                            float glob_scale, float opac, float3 color, float2 uv0, float3 umap,
                                            float3 vmap, int3 dims, bool use_blur, bool allow_double = true,
                                            RecCull* E = nullptr, bool cull = true) {
    const Axes A = quat_axes(quat);
    const float3 mc = V.xform(mean);
    const float3 a1c = V.rot(A.a1), a2c = V.rot(A.a2), nc = V.rot(A.a3);
    const float3 umc = V.rot(umap), vmc = V.rot(vmap);
    const float is1 = 1.f / (scale.x * glob_scale), is2 = 1.f / (scale.y * glob_scale);
    const float tvn = dot3(nc, mc);
    // blur centre exactly as the reference projects it (helpers.cuh:145-152)
    const float rwb = 1.f / (mc.z + 1e-6f);
    const float bx = mc.x * rwb * V.fx + V.cx, by = mc.y * rwb * V.fy + V.cy;
    Cd.mu = f4(mc, dot3(a1c, mc));
    Cd.dt = make_float4(dot3(a2c, mc), dot3(umc, mc), dot3(vmc, mc), 0.f);
    Wm.uvs = make_float4(uv0.x, uv0.y, bx, by);
    Wm.col = f4(color, is1);
    Wm.nrm = f4(A.a3, is2);
    Wm.tex = make_int4(dims.x, dims.y, dims.z, gid);

    // screen box of alpha >= 1/255 (empty when the splat can never reach it)
    float x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;
    const float smax = __logf(255.f * opac);
    int flags = 0;
    if (!(mc.z > kTNear)) flags = 1;
    bool oval = false;
    if (smax > 0.f) {
        const float a = sqrtf(2.f * smax + 1e-3f) * 1.002f;
        const float e1 = a / is1, e2 = a / is2;
        // The point of the plane with l_k = a_k . delta is delta = l1 b1 + l2 b2, where b is
        // dual to a in the plane.  b_k = a_k for a rotation; the axes of a quaternion that
        // is not of unit length are oblique.
        float3 b1 = cross3(a2c, nc), b2 = cross3(nc, a1c);
        const float det = dot3(a1c, b1), idet = 1.f / det;
        b1 = idet * b1;
        b2 = idet * b2;
        bool front = !flags && fabsf(det) > 1e-6f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float s1 = (k & 1) ? -e1 : e1, s2 = (k & 2) ? -e2 : e2;
            const float3 c = make_float3(mc.x + s1 * b1.x + s2 * b2.x, mc.y + s1 * b1.y + s2 * b2.y,
                                         mc.z + s1 * b1.z + s2 * b2.z);
            front = front && c.z > 1e-3f;
            const float iz = 1.f / c.z;
            const float px = V.fx * c.x * iz + V.cx, py = V.fy * c.y * iz + V.cy;
            x0 = fminf(x0, px); x1 = fmaxf(x1, px);
            y0 = fminf(y0, py); y1 = fmaxf(y1, py);
        }
        if (front) {
            const float mx = 1e-2f + 1e-5f * (fabsf(x0) + fabsf(x1)), my = 1e-2f + 1e-5f * (fabsf(y0) + fabsf(y1));
            x0 -= mx; x1 += mx; y0 -= my; y1 += my;
            if (E && !use_blur && cull) oval = cull_ellipse(*E, V, mc, mc.x / mc.z, mc.y / mc.z, b1, b2, e1, e2);
        } else {
            x0 = y0 = -INFINITY;
            x1 = y1 = INFINITY;
        }
        if (use_blur) {
            const float r = sqrtf(smax) * 1.002f + 1e-2f;
            x0 = fminf(x0, bx - r); x1 = fmaxf(x1, bx + r);
            y0 = fminf(y0, by - r); y1 = fmaxf(y1, by + r);
        }
    } else if (opac != opac) {
        // a NaN opacity gives alpha = fminf(0.99, NaN) = 0.99 in the reference: never cull it
        x0 = y0 = -INFINITY;
        x1 = y1 = INFINITY;
    }
    if (!cull) {
        // alpha-visualisation mode sets alpha without the opacity: no box
        x0 = y0 = -INFINITY;
        x1 = y1 = INFINITY;
    }
    if (E && !oval) *E = cull_box(x0, x1, y0, y1);

    H.box = make_float4(x0, x1, y0, y1);
    if (flags) {
        H.org = make_float4(V.cx, V.cy, 0.f, tvn);
        H.lc = make_float4(0.f, 0.f, 0.f, 0.f);
        H.nop = make_float4(0.f, 0.f, opac, __int_as_float(flags));
        Wm.uvm = make_float4(0.f, 0.f, 0.f, 0.f);
        return false;
    }
    const float u0f = mc.x / mc.z, v0f = mc.y / mc.z;
    const float gf = nc.x * u0f + nc.y * v0f + nc.z;
    const bool edge_on = fabsf(gf) < kEdgeOn;
    if (edge_on && allow_double) {
        edge_on_solve(H, Wm, V, mc, a1c, a2c, nc, umc, vmc, is1, is2, tvn);
    } else {
        const float mz = mc.z, ifx = 1.f / V.fx, ify = 1.f / V.fy;
        const float a1d = a1c.x * u0f + a1c.y * v0f + a1c.z, a2d = a2c.x * u0f + a2c.y * v0f + a2c.z;
        const float umd = umc.x * u0f + umc.y * v0f + umc.z, vmd = vmc.x * u0f + vmc.y * v0f + vmc.z;
        H.org = make_float4(V.fx * u0f + V.cx, V.fy * v0f + V.cy, gf, tvn);
        H.nop.x = nc.x * ifx;
        H.nop.y = nc.y * ify;
        H.lc = make_float4(mz * (gf * a1c.x - a1d * nc.x) * ifx * is1, mz * (gf * a1c.y - a1d * nc.y) * ify * is1,
                          mz * (gf * a2c.x - a2d * nc.x) * ifx * is2, mz * (gf * a2c.y - a2d * nc.y) * ify * is2);
        Wm.uvm = make_float4(mz * (gf * umc.x - umd * nc.x) * ifx, mz * (gf * umc.y - umd * nc.y) * ify,
                             mz * (gf * vmc.x - vmd * nc.x) * ifx, mz * (gf * vmc.y - vmd * nc.y) * ify);
    }
    H.nop.z = opac;
    H.nop.w = __int_as_float(flags);
    return edge_on && !allow_double;
}

__device__ __forceinline__ RecCull unpack_cull(float4 c) {
    RecCull e;
    e.xc = c.x;
    e.yc = c.y;
    e.ms = __float_as_uint(c.z);
    e.hk = __float_as_uint(c.w);
    return e;
}

// A record as it is stored (RecChunk).  The block kernels read "direct form
// only" from a NaN in g, which makes the plane denominator NaN.
__device__ __forceinline__ void pack_record(RecAll& r, const RecHot& h, const RecWarm& w, const RecCold& c,
                                            const RecCull& e) {
    const int flags = __float_as_int(h.nop.w);
    const float du = (float)w.tex.x * sqrtf(w.uvm.x * w.uvm.x + w.uvm.y * w.uvm.y);
    const float dv = (float)w.tex.y * sqrtf(w.uvm.z * w.uvm.z + w.uvm.w * w.uvm.w);
    const bool coarse = !flags && kCoarsePixels * fmaxf(du, dv) <= fabsf(h.org.z);
    const uint32_t start = (uint32_t)w.tex.z | (coarse ? kCoarseChart : 0u);
    r.c[kChunkCull] = make_float4(e.xc, e.yc, __uint_as_float(e.ms), __uint_as_float(e.hk));
    r.c[kChunkCull + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    r.c[kChunkOrg] = make_float4(h.org.x, h.org.y, flags ? __int_as_float(0x7fffffff) : h.org.z, h.org.w);
    r.c[kChunkLc] = h.lc;
    r.c[kChunkNop] = make_float4(h.nop.x, h.nop.y, h.nop.z, __uint_as_float(start));
    r.c[kChunkUvm] = w.uvm;
    r.c[kChunkUvs] = make_float4(w.uvs.x, w.uvs.y, __int_as_float(w.tex.x), __int_as_float(w.tex.y));
    r.c[kChunkCol] = w.col;
    r.c[kChunkNrm] = w.nrm;
    r.c[kChunkRay] = make_float4(w.col.w * c.mu.w, w.nrm.w * c.dt.x, c.dt.y, c.dt.z);
    r.c[kChunkMisc] = make_float4(w.uvs.z, w.uvs.w, h.nop.w, __int_as_float(w.tex.w));
    r.c[kChunkBox] = h.box;
    r.c[kChunkMu] = c.mu;
    r.c[kChunkDt] = c.dt;
}

// Per-pixel constants: pixel centre, camera direction d = (u, v, 1), |d|.
struct PixelRay {
    float px, py;
    float u, v;
    float dn;    // |d|
    float idn;   // 1/|d| = the reference's view_depth
};

__device__ __forceinline__ PixelRay make_pixel(const View& V, int i, int j) {
    PixelRay P;
    P.px = (float)j + 0.5f;
    P.py = (float)i + 0.5f;
    P.u = (P.px - V.cx) / V.fx;
    P.v = (P.py - V.cy) / V.fy;
    P.dn = sqrtf(P.u * P.u + P.v * P.v + 1.f);
    P.idn = 1.f / P.dn;
    return P;
}

__device__ __forceinline__ bool outside_box(const RecHot& H, const PixelRay& P) {
    return P.px < H.box.x || P.px > H.box.y || P.py < H.box.z || P.py > H.box.w;
}

// Intersection of a pixel ray with a staged splat.
struct Hit {
    float t;         // ray parameter along the unit ray (reference t)
    float tcam;      // camera z of the hit (reference t * view_depth)
    float l1s, l2s;  // plane coordinates divided by the scales
    float du, dv;    // pixel offset from the projected centre (fast form)
    float inv;       // d t_cam / d tvn: 1 / den (fast form), idn / den_ref (direct form)
    float nd;        // n_c . d, the sign of ray . normal
    float tu, tv;    // texture uv before clamping (direct form only)
    bool direct;
};

__device__ __forceinline__ float clamp_denom(float d) {
    if (0.f <= d && d < kDenomEps) return kDenomEps;
    if (-kDenomEps < d && d <= 0.f) return -kDenomEps;
    return d;
}

// Fast form of the intersection; sets H.direct when the pixel needs the
// direct form (computed by the caller from the Gaussian's parameters).
__device__ __forceinline__ Hit intersect(const RecHot& Hr, const PixelRay& P) {
    Hit H;
    const float2 d = sub2(make_float2(P.px, P.py), make_float2(Hr.org.x, Hr.org.y));
    H.du = d.x;
    H.dv = d.y;
    const float den = Hr.org.z + Hr.nop.x * H.du + Hr.nop.y * H.dv;
    H.nd = den;
    H.direct = __float_as_int(Hr.nop.w) != 0 || !(fabsf(den) >= kDenomEps * P.dn);
    const float inv = __fdividef(1.f, den);
    H.inv = inv;
    H.tcam = Hr.org.w * inv;
    H.t = H.tcam * P.dn;
    const float2 l = mul2(fma2(make_float2(Hr.lc.y, Hr.lc.w), dup2(H.dv),
                               mul2(make_float2(Hr.lc.x, Hr.lc.z), dup2(H.du))), dup2(inv));
    H.l1s = l.x;
    H.l2s = l.y;
    return H;
}

// Direct camera-space form with the reference's denominator clamp, from the
// camera-space frame of the Gaussian.
__device__ __forceinline__ void intersect_direct(Hit& H, const PixelRay& P, float tvn, float3 mc, float3 a1c,
                                                 float3 a2c, float3 nc, float3 umc, float3 vmc, float is1, float is2,
                                                 float uv0x, float uv0y) {
    const float3 d = make_float3(P.u, P.v, 1.f);
    H.nd = dot3(nc, d);
    const float dref = clamp_denom(H.nd * P.idn);
    const float t = tvn / dref;
    const float3 delta = t * (P.idn * d) - mc;
    H.inv = P.idn / dref;
    H.t = t;
    H.tcam = t * P.idn;
    H.l1s = dot3(a1c, delta) * is1;
    H.l2s = dot3(a2c, delta) * is2;
    H.tu = uv0x + dot3(umc, delta);
    H.tv = uv0y + dot3(vmc, delta);
}

// Texture coordinates of the hit (before clamping).
__device__ __forceinline__ float2 hit_uv(const Hit& H, const RecWarm& Wm) {
    if (!H.direct) {
        const float2 t = fma2(make_float2(Wm.uvm.y, Wm.uvm.w), dup2(H.dv),
                              mul2(make_float2(Wm.uvm.x, Wm.uvm.z), dup2(H.du)));
        return fma2(t, dup2(H.inv), make_float2(Wm.uvs.x, Wm.uvs.y));
    }
    return make_float2(H.tu, H.tv);
}

__device__ __forceinline__ float clamp01(float x) {
    // texture_helpers.cuh:37-51
    if (x <= 0.f) x = 0.f;
    if (x >= 1.f) x = 1.f;
    return x;
}

// Bilinear corner indices (texel rows) and weights inside chart (h, w, start)
// (texture_helpers.cuh:162-215).  Indices are texel rows, not element offsets.
struct Bilerp {
    int i00, i01, i10, i11;
    float w00, w01, w10, w11;
    float fx, fy;  // fractional parts (for the uv gradient)
};

__device__ __forceinline__ Bilerp bilerp(int h, int w, int start, float u, float v, bool bilinear) {
    Bilerp B;
    const float2 tc = mul2(make_float2((float)h, (float)w), make_float2(u, v));
    const float tcx = tc.x, tcy = tc.y;
    int iix = __float2int_rz(tcx), iiy = __float2int_rz(tcy);
    const int jjx = min(iix + 1, h - 1), jjy = min(iiy + 1, w - 1);
    const float wx = tcx - (float)iix, wy = tcy - (float)iiy;
    iix = min(iix, h - 1);
    iiy = min(iiy, w - 1);
    B.fx = wx; B.fy = wy;
    const float2 wyy = make_float2(1.f - wy, wy);
    const float2 w0 = mul2(dup2(1.f - wx), wyy), w1 = mul2(dup2(wx), wyy);
    const float w00 = w0.x, w01 = w0.y, w10 = w1.x, w11 = w1.y;
    B.i00 = start + iix * w + iiy;
    B.i01 = start + iix * w + jjy;
    B.i10 = start + jjx * w + iiy;
    B.i11 = start + jjx * w + jjy;
    if (bilinear) {
        B.w00 = w00; B.w01 = w01; B.w10 = w10; B.w11 = w11;
    } else {
        B.w00 = B.w01 = B.w10 = B.w11 = 0.f;
        if (w00 >= w01 && w00 >= w10 && w00 >= w11) B.w00 = 1.f;
        else if (w01 >= w00 && w01 >= w10 && w01 >= w11) B.w01 = 1.f;
        else if (w10 >= w00 && w10 >= w01 && w10 >= w11) B.w10 = 1.f;
        else B.w11 = 1.f;
    }
    return B;
}

// A chain of short kernels: launch_chained lets a kernel be set up while the one
// before it in the stream still runs; chain_wait, before it reads or writes
// anything that kernel may touch, waits for its end (and that of all before it).
// Then the next one of the chain may be set up in turn.  Binning of four small
// views (17 launches) 157 -> 138 us, of eight large ones 422 -> 382; a 32-bit
// sort of 100k items 46 -> 32, of 780k 74 -> 50.  Not for the compositor: blocks
// set up around those of the kernel before are spread unevenly over the
// multiprocessors (forward of a 720p view 354 -> 388 us).
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);  // (errors: check_launch)
}

}  // namespace gstex
