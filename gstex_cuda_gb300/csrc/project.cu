// Per-Gaussian projection work: screen AABB, tile counts, prefix sum, SH.
//
// Built with -fmad=false and IEEE division so that the AABB and tile counts
// are reproducible bit for bit by a CPU restatement of the same operations.
#include <algorithm>

#include "common.cuh"
#include "project.cuh"

namespace gstex {

// Reference: csrc/get_aabb_2d.cu:11-89
__global__ void aabb_kernel(int n, const float3* __restrict__ means, const float* __restrict__ scales,
                            float glob_scale, const float4* __restrict__ quats, const float* __restrict__ viewmat,
                            float fx, float fy, float cx, float cy, float2* __restrict__ centers,
                            float2* __restrict__ extents) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float m[12];
#pragma unroll
    for (int k = 0; k < 12; k++) m[k] = viewmat[k];
    float2 c, e;
    float z;
    aabb_2d(m, fx, fy, cx, cy, means[i], quats[i], scales[3 * (size_t)i], scales[3 * (size_t)i + 1], glob_scale, c, e, z);
    centers[i] = c;
    extents[i] = e;
}

// gstex_cuda/get_aabb_2d.py:70-91 in float32: floor((c-e)/bw), floor((c+e)/bw + 1),
// clamped to the tile grid.
__global__ void tiles_hit_kernel(int n, const float2* __restrict__ centers, const float2* __restrict__ extents,
                                 int tiles_x, int tiles_y, float fbw, int32_t* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = tiles_hit(centers[i], extents[i], tiles_x, tiles_y, fbw);
}

// project_points (gstex_cuda/get_aabb_2d.py:22-32) in one launch instead of a
// matrix product and eleven elementwise operations (174 -> 25 us of host time a
// call, which is what a small view's pass consists of): the product's
// accumulation order (for more than 16 points) and the operations' rounding are
// kept.
__global__ void project_points_kernel(int n, const float3* __restrict__ points, const float* __restrict__ viewmat,
                                      float fx, float fy, float cx, float cy, float2* __restrict__ pix,
                                      float* __restrict__ depths) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 p = points[i];
    float v[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
        v[c] = __fadd_rn(__fmaf_rn(p.z, viewmat[4 * c + 2], __fmaf_rn(p.y, viewmat[4 * c + 1],
                                                                     __fmul_rn(p.x, viewmat[4 * c]))),
                         viewmat[4 * c + 3]);
    const float rw = __fdiv_rn(1.f, __fadd_rn(v[2], 1e-6f));
    pix[i] = make_float2(__fadd_rn(__fmul_rn(__fmul_rn(v[0], rw), fx), cx),
                         __fadd_rn(__fmul_rn(__fmul_rn(v[1], rw), fy), cy));
    depths[i] = v[2];
}

// ---------------------------------------------------------------------------
// Inclusive int32 scan (decomposed: block sums, scan of sums, block scan)
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    total = warp_sums[(blockDim.x >> 5) - 1];
    const int before = warp > 0 ? warp_sums[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

// order: sums in[order[i]] and keeps these in `picked`.
__global__ void scan_block_sums(int n, const int32_t* __restrict__ in, const int32_t* __restrict__ order,
                                int32_t* __restrict__ picked, int64_t* __restrict__ sums) {
    chain_wait();
    __shared__ long long part[kScanThreads / 32];
    const int base = blockIdx.x * kScanTile;
    long long s = 0;  // (a block's counts may pass 31 bits, and the caller has to see it)
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const unsigned idx = base + k * kScanThreads + threadIdx.x;  // (may pass 31 bits)
        if (idx < (unsigned)n) {
            const int v = in[order ? order[idx] : idx];
            if (order) picked[idx] = v;
            s += v;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = 0;
#pragma unroll
        for (int w = 0; w < kScanThreads / 32; w++) s += part[w];
        sums[blockIdx.x] = s;
    }
}

// single block: exclusive scan of the block sums (64-bit to detect overflow)
__global__ void scan_sums(int nb, int64_t* __restrict__ sums, int64_t* __restrict__ total) {
    chain_wait();
    __shared__ long long carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += blockDim.x) {
        const int i = base + threadIdx.x;
        long long v = i < nb ? sums[i] : 0;
        // warp-serial inclusive scan over the block (small nb)
        __shared__ long long buf[1024];
        buf[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < (int)blockDim.x; o <<= 1) {
            long long y = threadIdx.x >= (unsigned)o ? buf[threadIdx.x - o] : 0;
            __syncthreads();
            buf[threadIdx.x] += y;
            __syncthreads();
        }
        if (i < nb) sums[i] = carry + buf[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += buf[threadIdx.x];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// total: `offsets` still holds the sums of the blocks (at most one per thread),
// and each block adds up those before it.
__global__ void scan_apply(int n, const int32_t* __restrict__ in, const int64_t* __restrict__ offsets,
                           int64_t* __restrict__ total_out, int32_t* __restrict__ out) {
    chain_wait();
    __shared__ int ws[32];
    __shared__ long long before[kScanThreads / 32];
    long long offset = 0;
    if (total_out) {
        long long x = threadIdx.x < blockIdx.x ? offsets[threadIdx.x] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) before[threadIdx.x >> 5] = x;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kScanThreads / 32; w++) offset += before[w];
        if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = offset + offsets[blockIdx.x];
    } else {
        offset = offsets[blockIdx.x];
    }
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const int idx = base + k;
        v[k] = idx < n ? in[idx] : 0;
        s += v[k];
    }
    int total;
    int run = block_exclusive_scan(s, ws, total) + (int)offset;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        run += v[k];
        const int idx = base + k;
        if (idx < n) out[idx] = run;
    }
}

// ---------------------------------------------------------------------------
// Spherical harmonics (csrc/sh.cuh:46-253; basis of gstex_cuda/_torch_impl.py:62-113)
// ---------------------------------------------------------------------------
// Templated on the degree in use (DTU), so the basis stays in registers; the
// coefficient stride follows the stored degree.
template <int DTU>
__global__ void sh_forward_kernel(int n, int degree, const float3* __restrict__ dirs,
                                  const float* __restrict__ coeffs, float* __restrict__ colors) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    constexpr int NB = (DTU + 1) * (DTU + 1);
    float Y[25];
    sh_basis(DTU, dirs[i], Y);
    const float* k = coeffs + (size_t)i * sh_bases(degree) * 3;
    float c0 = 0.f, c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        c0 += Y[b] * k[3 * b + 0];
        c1 += Y[b] * k[3 * b + 1];
        c2 += Y[b] * k[3 * b + 2];
    }
    colors[3 * (size_t)i] = c0;
    colors[3 * (size_t)i + 1] = c1;
    colors[3 * (size_t)i + 2] = c2;
}

template <int DTU>
__global__ void sh_backward_kernel(int n, int degree, const float3* __restrict__ dirs,
                                   const float* __restrict__ v_colors, float* __restrict__ v_coeffs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    constexpr int NB = (DTU + 1) * (DTU + 1);
    float Y[25];
    sh_basis(DTU, dirs[i], Y);
    const int B = sh_bases(degree);
    const float v0 = v_colors[3 * (size_t)i], v1 = v_colors[3 * (size_t)i + 1], v2 = v_colors[3 * (size_t)i + 2];
    float* o = v_coeffs + (size_t)i * B * 3;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        o[3 * b + 0] = Y[b] * v0;
        o[3 * b + 1] = Y[b] * v1;
        o[3 * b + 2] = Y[b] * v2;
    }
    for (int b = NB; b < B; b++) {
        o[3 * b + 0] = 0.f;
        o[3 * b + 1] = 0.f;
        o[3 * b + 2] = 0.f;
    }
}

// The same with all stored bases in use, the rows moved through shared memory
// (RowStage).  500k Gaussians of degree 3: forward 55 -> 28 us, backward 138 ->
// 17 us (both move about 100 MB: 16 us).
template <int DTU>
__global__ void __launch_bounds__(RowStage<1>::kRows) sh_forward_rows_kernel(int n, const float3* __restrict__ dirs,
                                                                             const float* __restrict__ coeffs,
                                                                             float* __restrict__ colors) {
    constexpr int NB = (DTU + 1) * (DTU + 1);
    __shared__ RowStage<3 * NB> rows;
    const int i0 = blockIdx.x * rows.kRows, i = i0 + threadIdx.x;
    rows.load(coeffs, i0, min(n - i0, rows.kRows));
    if (i >= n) return;
    float Y[25];
    sh_basis(DTU, dirs[i], Y);
    const float* k = rows.row();
    float c0 = 0.f, c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        c0 += Y[b] * k[3 * b + 0];
        c1 += Y[b] * k[3 * b + 1];
        c2 += Y[b] * k[3 * b + 2];
    }
    colors[3 * (size_t)i] = c0;
    colors[3 * (size_t)i + 1] = c1;
    colors[3 * (size_t)i + 2] = c2;
}

template <int DTU>
__global__ void __launch_bounds__(RowStage<1>::kRows) sh_backward_rows_kernel(int n, const float3* __restrict__ dirs,
                                                                              const float* __restrict__ v_colors,
                                                                              float* __restrict__ v_coeffs) {
    constexpr int NB = (DTU + 1) * (DTU + 1);
    __shared__ RowStage<3 * NB> rows;
    const int i0 = blockIdx.x * rows.kRows, i = i0 + threadIdx.x;
    if (i < n) {
        float Y[25];
        sh_basis(DTU, dirs[i], Y);
        const float v0 = v_colors[3 * (size_t)i], v1 = v_colors[3 * (size_t)i + 1], v2 = v_colors[3 * (size_t)i + 2];
        float* o = rows.row();
#pragma unroll
        for (int b = 0; b < NB; b++) {
            o[3 * b + 0] = Y[b] * v0;
            o[3 * b + 1] = Y[b] * v1;
            o[3 * b + 2] = Y[b] * v2;
        }
    }
    rows.store(v_coeffs, i0, min(n - i0, rows.kRows));
}

}  // namespace gstex

using namespace gstex;

extern "C" int gstex_get_aabb_2d(int n, const float* means, const float* scales, float glob_scale,
                                 const float* quats, const float* viewmat, float fx, float fy, float cx, float cy,
                                 float* centers, float* extents, gstex_stream_t stream) {
    GSTEX_REQUIRE(n >= 0);
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(means && scales && quats && viewmat && centers && extents);
    aabb_kernel<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(
        n, (const float3*)means, scales, glob_scale, (const float4*)quats, viewmat, fx, fy, cx, cy,
        (float2*)centers, (float2*)extents);
    return check_launch("get_aabb_2d");
}

extern "C" int gstex_num_tiles_hit(int n, const float* centers, const float* extents, int img_height,
                                   int img_width, int block_width, int32_t* out, gstex_stream_t stream) {
    GSTEX_REQUIRE(n >= 0 && img_height > 0 && img_width > 0 && block_width > 0);
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(centers && extents && out);
    const int tx = ceil_div(img_width, block_width), ty = ceil_div(img_height, block_width);
    tiles_hit_kernel<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(
        n, (const float2*)centers, (const float2*)extents, tx, ty, (float)block_width, out);
    return check_launch("num_tiles_hit");
}

extern "C" int gstex_project_points(int n, const float* points, const float* viewmat, float fx, float fy, float cx,
                                    float cy, float* pix, float* depths, gstex_stream_t stream) {
    GSTEX_REQUIRE(n >= 0);
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(points && viewmat && pix && ((uintptr_t)pix & 7) == 0 && depths);
    project_points_kernel<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(n, (const float3*)points, viewmat, fx, fy,
                                                                            cx, cy, (float2*)pix, depths);
    return check_launch("project_points");
}

// sum of h * w over the charts of dims [n, 3]
namespace gstex {
__global__ void __launch_bounds__(1024) chart_texels_kernel(int n, const int32_t* __restrict__ dims,
                                                            int64_t* __restrict__ total) {
    __shared__ long long part[32];
    long long s = 0;
    for (int i = blockIdx.x * 1024 + threadIdx.x; i < n; i += gridDim.x * 1024)
        s += (long long)dims[3 * (size_t)i] * dims[3 * (size_t)i + 1];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = part[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) atomicAdd((unsigned long long*)total, (unsigned long long)s);
    }
}
}  // namespace gstex

extern "C" int gstex_chart_texels(int n, const int32_t* dims, int64_t* total, gstex_stream_t s) {
    GSTEX_REQUIRE(n >= 0 && total);
    cudaStream_t stream = (cudaStream_t)s;
    cudaError_t e = cudaMemsetAsync(total, 0, sizeof(int64_t), stream);
    if (e != cudaSuccess) { set_cuda_error(e, "chart_texels"); return GSTEX_ERR_CUDA; }
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(dims);
    chart_texels_kernel<<<std::min(ceil_div(n, 1024), 152), 1024, 0, stream>>>(n, dims, total);
    return check_launch("chart_texels");
}

extern "C" size_t gstex_scan_workspace_bytes(int n) {
    return (size_t)(ceil_div(n > 0 ? n : 1, kScanTile) + 1) * sizeof(int64_t);
}

// Up to one block per thread of a block (2M counts) two launches do: with the
// third and one that gathers, 21 instead of 11 us for 32k to 100k counts and 33
// instead of 22 us for 800k.
static int inclusive_scan(int n, const int32_t* counts, const int32_t* order, int32_t* picked, int32_t* cum,
                          int64_t* total, void* ws, size_t ws_bytes, cudaStream_t stream) {
    if (n == 0) {
        cudaError_t e = cudaMemsetAsync(total, 0, sizeof(int64_t), stream);
        if (e != cudaSuccess) { set_cuda_error(e, "scan"); return GSTEX_ERR_CUDA; }
        return GSTEX_OK;
    }
    GSTEX_REQUIRE(counts && cum && ws);
    if (ws_bytes < gstex_scan_workspace_bytes(n)) return GSTEX_ERR_CAPACITY;
    const int nb = ceil_div(n, kScanTile);
    const bool two = nb <= kScanThreads;
    int64_t* sums = (int64_t*)ws;
    launch_chained(scan_block_sums, nb, kScanThreads, 0, stream, n, counts, order, picked, sums);
    if (!two) launch_chained(scan_sums, 1, 1024, 0, stream, nb, sums, total);
    launch_chained(scan_apply, nb, kScanThreads, 0, stream,
                   n, order ? picked : counts, sums, two ? total : nullptr, cum);
    return check_launch("inclusive_scan", two ? 2 : 3);
}

extern "C" int gstex_inclusive_scan_i32(int n, const int32_t* counts, int32_t* cum, int64_t* total, void* ws,
                                        size_t ws_bytes, gstex_stream_t s) {
    GSTEX_REQUIRE(n >= 0 && total);
    return inclusive_scan(n, counts, nullptr, nullptr, cum, total, ws, ws_bytes, (cudaStream_t)s);
}

extern "C" int gstex_inclusive_scan_picked_i32(int n, const int32_t* counts, const int32_t* order, int32_t* picked,
                                               int32_t* cum, int64_t* total, void* ws, size_t ws_bytes,
                                               gstex_stream_t s) {
    GSTEX_REQUIRE(n >= 0 && total);
    if (n > 0) GSTEX_REQUIRE(order && picked);
    return inclusive_scan(n, counts, order, picked, cum, total, ws, ws_bytes, (cudaStream_t)s);
}

// Degrees above 4 are not supported (sh.cuh:46-253 stops at 4); the degree in
// use must not exceed the stored one (the reference's wrapper asserts it,
// sh.py:54, and its kernel would read the next Gaussian's coefficients).
static int sh_degrees_ok(int degree, int degrees_to_use) {
    if (degree < 0 || degrees_to_use < 0 || degrees_to_use > degree) return GSTEX_ERR_INVALID_ARGUMENT;
    if (degree > 4) return GSTEX_ERR_UNSUPPORTED;
    return GSTEX_OK;
}

extern "C" int gstex_compute_sh_forward(int n, int degree, int degrees_to_use, const float* viewdirs,
                                        const float* coeffs, float* colors, gstex_stream_t stream) {
    GSTEX_REQUIRE(n >= 0);
    int rc = sh_degrees_ok(degree, degrees_to_use);
    if (rc) return rc;
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(viewdirs && coeffs && colors);
    const dim3 grid(ceil_div(n, 256)), block(256);
    cudaStream_t st = (cudaStream_t)stream;
    const float3* d = (const float3*)viewdirs;
    if (degrees_to_use == degree && degree >= 1) {
        const dim3 rgrid(ceil_div(n, RowStage<1>::kRows)), rblock(RowStage<1>::kRows);
        switch (degree) {
            case 1: sh_forward_rows_kernel<1><<<rgrid, rblock, 0, st>>>(n, d, coeffs, colors); break;
            case 2: sh_forward_rows_kernel<2><<<rgrid, rblock, 0, st>>>(n, d, coeffs, colors); break;
            case 3: sh_forward_rows_kernel<3><<<rgrid, rblock, 0, st>>>(n, d, coeffs, colors); break;
            default: sh_forward_rows_kernel<4><<<rgrid, rblock, 0, st>>>(n, d, coeffs, colors); break;
        }
        return check_launch("compute_sh_forward");
    }
    switch (degrees_to_use) {
        case 0: sh_forward_kernel<0><<<grid, block, 0, st>>>(n, degree, d, coeffs, colors); break;
        case 1: sh_forward_kernel<1><<<grid, block, 0, st>>>(n, degree, d, coeffs, colors); break;
        case 2: sh_forward_kernel<2><<<grid, block, 0, st>>>(n, degree, d, coeffs, colors); break;
        case 3: sh_forward_kernel<3><<<grid, block, 0, st>>>(n, degree, d, coeffs, colors); break;
        default: sh_forward_kernel<4><<<grid, block, 0, st>>>(n, degree, d, coeffs, colors); break;
    }
    return check_launch("compute_sh_forward");
}

extern "C" int gstex_compute_sh_backward(int n, int degree, int degrees_to_use, const float* viewdirs,
                                         const float* v_colors, float* v_coeffs, gstex_stream_t stream) {
    GSTEX_REQUIRE(n >= 0);
    int rc = sh_degrees_ok(degree, degrees_to_use);
    if (rc) return rc;
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(viewdirs && v_colors && v_coeffs);
    const dim3 grid(ceil_div(n, 256)), block(256);
    cudaStream_t st = (cudaStream_t)stream;
    const float3* d = (const float3*)viewdirs;
    if (degrees_to_use == degree && degree >= 1) {
        const dim3 rgrid(ceil_div(n, RowStage<1>::kRows)), rblock(RowStage<1>::kRows);
        switch (degree) {
            case 1: sh_backward_rows_kernel<1><<<rgrid, rblock, 0, st>>>(n, d, v_colors, v_coeffs); break;
            case 2: sh_backward_rows_kernel<2><<<rgrid, rblock, 0, st>>>(n, d, v_colors, v_coeffs); break;
            case 3: sh_backward_rows_kernel<3><<<rgrid, rblock, 0, st>>>(n, d, v_colors, v_coeffs); break;
            default: sh_backward_rows_kernel<4><<<rgrid, rblock, 0, st>>>(n, d, v_colors, v_coeffs); break;
        }
        return check_launch("compute_sh_backward");
    }
    switch (degrees_to_use) {
        case 0: sh_backward_kernel<0><<<grid, block, 0, st>>>(n, degree, d, v_colors, v_coeffs); break;
        case 1: sh_backward_kernel<1><<<grid, block, 0, st>>>(n, degree, d, v_colors, v_coeffs); break;
        case 2: sh_backward_kernel<2><<<grid, block, 0, st>>>(n, degree, d, v_colors, v_coeffs); break;
        case 3: sh_backward_kernel<3><<<grid, block, 0, st>>>(n, degree, d, v_colors, v_coeffs); break;
        default: sh_backward_kernel<4><<<grid, block, 0, st>>>(n, degree, d, v_colors, v_coeffs); break;
    }
    return check_launch("compute_sh_backward");
}
