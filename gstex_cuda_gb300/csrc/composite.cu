// Block compositor: the textured 2D-Gaussian forward with one warp per 8x4
// block of pixels.
//
// Reference: csrc/texture.cu:11-329.  A splat reaches about a tenth of
// the pixels of a tile that lists it, so a warp that walks its tile's list
// splat by splat has few of its lanes at work.  Here a warp first turns the
// list into one list per pixel and then every lane walks its own:
//
//   1. cull: 32 listed splats at a time, one per lane, are tested against the
//      block's four pixel rows (RecCull); a splat's answer is the 32-bit mask
//      of the pixels it can reach.  Those that reach none are dropped, the
//      others queue up until 32 are there;
//   2. stage: the records of these 32 are copied to shared memory
//      (cp.async) while the 32 masks are transposed with five shuffles, which
//      gives each lane the 32-bit set of the splats that can reach its pixel;
//   3. walk: every lane goes through its own set in order.  The lanes of one
//      step are usually at different splats.
//
// What bounds it: the L1 data path (77% of its cycles at 24 warps per SM; half
// of it staged records, half texel gathers), then the ALUs (47%).  Measured
// against the list walk with one CTA per tile (forward kernel alone): 32 views
// with 81M intersections, bf16 texels, 8x8 tiles 17.4 -> 8.9 ms; 8 clustered
// full-HD views 9.2 -> 5.3 ms; one 800x800 view, 16x16 tiles 232 -> 62 us; one
// full-HD view of large splats 5.1 -> 2.2 ms.  About 16 of 32 lanes blend in a
// step, against 3 to 7 before.
//
// A warp needs no barrier with any other.  Results are those of the list
// walk: a dropped (splat, pixel) pair has alpha < 1/255, which the reference
// skips; that a skipped splat can end a pixel whose T is already within
// 1 / (1 - 1/255) of 1e-4 (texture.cu:213-221) is kept by finish_close().
#include "common.cuh"
#include "pixel.cuh"
#include "raster.cuh"

namespace gstex {

// CTAs per SM asked of the register allocator: 12 (80 registers).  10 (96) is
// a few per cent better on one small view and 8% worse on 32 views; 14 (72)
// spills 220 bytes for 2% there and loses 10% on small views; 16 loses 25%.
constexpr int kFwdCtas = 12;
constexpr int kBlockWarps = 2;       // warps per CTA (blocks of one 8x8 tile, or a quarter of a 16x16 one)
constexpr unsigned kFull = 0xffffffffu;

// One block of 8x4 pixels.
struct Block {
    int W, H, x0, y0;   // image size, first pixel
    int2 range;         // the tile's list
    size_t pix;         // first pixel of the view in the per-pixel arrays
    const RecAll* recs;
    float* vcolors;
    int view;
    float fx, fy, cx, cy;
};

__device__ __forceinline__ View block_view(const BlockArgs& ba, int v) {
    return ba.views ? ba.views[v].V : load_view(ba.viewmat, ba.fx, ba.fy, ba.cx, ba.cy);
}

// Pixel of a lane in its block: each quarter of the warp, whose shared-memory
// reads are served together, covers 4x2 pixels, which have more splats in
// common than an 8x1 row.
__device__ __forceinline__ int lane_col(unsigned lane) { return (int)(((lane >> 1) & 4u) | (lane & 3u)); }
__device__ __forceinline__ int lane_row(unsigned lane) { return (int)(((lane >> 3) & 2u) | ((lane >> 2) & 1u)); }

// Block g of the launch (tiles in queue order, the blocks of a tile back to
// back); false when it lies outside the launch or the image.
__device__ __forceinline__ bool load_block(const BlockArgs& ba, int g, Block& J) {
    const int wx = ba.bw >> 3, per_tile = wx * (ba.bw >> 2);
    const int q = g / per_tile, sub = g - q * per_tile;
    if (q >= ba.total_tiles) return false;
    const int t = ba.order ? ba.order[q] : q;
    int tiles_x, local = t;
    if (ba.views) {
        J.view = ba.tile_view[t];
        const BatchView& bv = ba.views[J.view];
        J.W = bv.W; J.H = bv.H;
        J.fx = bv.V.fx; J.fy = bv.V.fy; J.cx = bv.V.cx; J.cy = bv.V.cy;
        tiles_x = bv.tiles_x;
        local = t - bv.tile_offset;
        J.pix = bv.pix_offset;
        J.recs = ba.recs + (size_t)J.view * ba.num_points;
        J.vcolors = ba.vcolors ? ba.vcolors + (size_t)J.view * ba.num_points * ba.vc_stride : nullptr;
    } else {
        J.view = 0;
        J.W = ba.W; J.H = ba.H;
        J.fx = ba.fx; J.fy = ba.fy; J.cx = ba.cx; J.cy = ba.cy;
        tiles_x = ba.tiles_x;
        J.pix = 0;
        J.recs = ba.recs;
        J.vcolors = ba.vcolors;
    }
    const int ty = local / tiles_x, tx = local - ty * tiles_x;
    const int by = sub / wx, bx = sub - by * wx;
    J.x0 = tx * ba.bw + bx * 8;
    J.y0 = ty * ba.bw + by * 4;
    J.range = ba.bins[t];
    return J.x0 < J.W && J.y0 < J.H;
}

// Splats that passed the cull and wait to be staged: up to 31 left over plus
// one round of 32.
struct Queue {
    int gid[64];
    int idx[64];        // position in the sorted list
    unsigned mask[64];  // pixels of the block it can reach
};

// Scans the list from `pos` (towards higher positions for DIR 1, lower for
// DIR -1, up to but not including `end`) until 32 splats that reach a pixel
// of `live` are queued or the list ends.  Returns the number queued.
template <int DIR>
__device__ __forceinline__ int fill_queue(Queue& q, int n, int& pos, int end, const int32_t* __restrict__ gids,
                                          const RecAll* __restrict__ recs, float fx0, float fy0, unsigned live,
                                          unsigned lane) {
    while (n < 32 && (DIR > 0 ? pos < end : pos > end)) {
        const int i = pos + DIR * (int)lane;
        int gid = 0;
        unsigned m = 0;
        if (DIR > 0 ? i < end : i > end) {
            gid = __ldg(gids + i);
            const RecCull c = unpack_cull(__ldg(recs[gid].c + kChunkCull));
#pragma unroll
            for (int r = 0; r < 2; r++) {  // two rows are two quarters of 4x2 pixels
                const unsigned b0 = cull_row(c, fx0, fy0 + (float)(2 * r));
                const unsigned b1 = cull_row(c, fx0, fy0 + (float)(2 * r + 1));
                m |= ((b0 & 0xfu) | ((b0 & 0xf0u) << 4) | ((b1 & 0xfu) << 4) | ((b1 & 0xf0u) << 8)) << (16 * r);
            }
            m &= live;
        }
        const unsigned b = __ballot_sync(kFull, m != 0u);
        if (m) {
            const int s = n + __popc(b & ((1u << lane) - 1u));
            q.gid[s] = gid;
            q.idx[s] = i;
            q.mask[s] = m;
        }
        n += __popc(b);
        pos += DIR * 32;
    }
    __syncwarp();
    return n;
}

// Drops the 32 staged entries of the queue.
__device__ __forceinline__ int pop_queue(Queue& q, int n, unsigned lane) {
    if (n <= 32) return 0;
    const int m = n - 32;
    int g = 0, i = 0;
    unsigned k = 0;
    if ((int)lane < m) {
        g = q.gid[32 + lane];
        i = q.idx[32 + lane];
        k = q.mask[32 + lane];
    }
    __syncwarp();
    if ((int)lane < m) {
        q.gid[lane] = g;
        q.idx[lane] = i;
        q.mask[lane] = k;
    }
    __syncwarp();
    return m;
}

// Bit matrix transpose over the warp: lane p's result has bit k set where lane
// k's x has bit p set.
__device__ __forceinline__ unsigned transpose32(unsigned x, unsigned lane) {
    constexpr unsigned masks[5] = { 0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u };
#pragma unroll
    for (int s = 0; s < 5; s++) {
        const int j = 16 >> s;
        const unsigned m = masks[s], y = __shfl_xor_sync(kFull, x, j);
        x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
    }
    return x;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Staged records: NCH chunks (from kChunkOrg on) of 32 records, chunk-major.
// Rows of 33 keep the eight lanes that write one record's chunks, and lanes
// that read one chunk of neighbouring records, on different banks.
template <int NCH>
struct Staged {
    float4 c[NCH][33];
};

// Starts copying the records of the first n (at most 32) queued splats: eight
// lanes take one record's contiguous chunks.
template <int NCH>
__device__ __forceinline__ void stage_records(Staged<NCH>& S, const Queue& q, int n, const RecAll* __restrict__ recs,
                                              unsigned lane) {
    const int ch = lane & 7, r0 = lane >> 3;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int r = j * 4 + r0;
        if (r < n && ch < NCH) cp_async16(&S.c[ch][r], recs[q.gid[r]].c + kChunkOrg + ch);
    }
}

// Chunk access of one record, staged or in device memory.
template <int NCH>
struct StagedRec {
    const float4* p;
    __device__ __forceinline__ StagedRec(const Staged<NCH>& S, int k) : p(&S.c[0][k]) {}
    __device__ __forceinline__ float4 operator()(int chunk) const { return p[(chunk - kChunkOrg) * 33]; }
};
struct GlobalRec {
    const float4* p;
    __device__ __forceinline__ float4 operator()(int chunk) const { return __ldg(p + chunk); }
};

template <class Rec>
__device__ __forceinline__ Hit block_hit(const SceneArgs& a, const BlockArgs& ba, int view, const Rec& rec, int gid,
                                         const PixelRay& P, float& opac) {
    RecHot Hr;
    Hr.org = rec(kChunkOrg);
    Hr.lc = rec(kChunkLc);
    Hr.nop = rec(kChunkNop);
    opac = Hr.nop.z;
    Hr.nop.w = 0.f;  // (a NaN in org.z selects the direct form)
    Hit H = intersect(Hr, P);
    if (H.direct) {  // (rare)
        const View V = block_view(ba, view);
        const PixelRay Q = make_pixel(V, (int)(P.py - 0.5f), (int)(P.px - 0.5f));
        direct_hit(H, a.quats, a.means, a.scales, a.glob, a.uv0, a.umap, a.vmap, V, gid, Q, Hr.org.w);
    }
    return H;
}

// exp(-sigma), or with blur the larger of it and the screen-space filter's.
template <int FIX>
__device__ __forceinline__ float block_alpha(const Hit& H, float opac, bool use_blur, const RecAll* rec,
                                             const PixelRay& P, float& nbf, float& bf, float& e, float& eb) {
    const float sigma = 0.5f * (H.l1s * H.l1s + H.l2s * H.l2s);
    nbf = 1.f;
    bf = 0.f;
    float sigma_blur = 0.f;
    if (!FIX && use_blur) {
        const float4 c = __ldg(rec->c + kChunkMisc);
        const float dx = c.x - P.px, dy = c.y - P.py;
        sigma_blur = 0.5f * kBlurFsq * (dx * dx + dy * dy);
        if (sigma_blur < sigma) { bf = 1.f; nbf = 0.f; }
    }
    e = __expf(-sigma);
    eb = (!FIX && use_blur) ? __expf(-sigma_blur) : 0.f;
    return fminf(kAlphaMax, opac * (nbf * e + bf * eb));
}

// uv of the hit before clamping (hit_uv on the stored chunks).
__device__ __forceinline__ float2 block_uv(const Hit& H, float4 uvm, float2 uv0) {
    if (H.direct) return make_float2(H.tu, H.tv);
    const float2 t = fma2(make_float2(uvm.y, uvm.w), dup2(H.dv), mul2(make_float2(uvm.x, uvm.z), dup2(H.du)));
    return fma2(t, dup2(H.inv), uv0);
}

// ---------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------
constexpr int kFwdChunks = 7;
struct FwdMem {
    Staged<kFwdChunks> rec;
    Queue q;
};

template <int CT>
struct FwdPix {
    float T, depth, reg;
    int cur, didx;
    float3 out, nrm, ts;
    float tex[CT > 0 ? CT : 1];
};

// Blends one contributing pair into the pixel (texture.cu:222-296).
template <int TM, int CT, int FIX, class Rec>
__device__ __forceinline__ void blend(FwdPix<CT>& S, const SceneArgs& a, const Rec& rec, const Hit& H, float alpha,
                                      float next_T, int idx) {
    const float vis = alpha * S.T;
    const float4 col = rec(kChunkCol), nw = rec(kChunkNrm);
    const float2 o2 = fma2(make_float2(col.x, col.y), dup2(vis), make_float2(S.out.x, S.out.y));
    S.out.x = o2.x;
    S.out.y = o2.y;
    S.out.z = S.out.z + col.z * vis;
    float3 hn = f3(nw);
    if (!FIX && (a.settings & (1 << 15)) && H.nd > 0.f) hn = make_float3(-hn.x, -hn.y, -hn.z);
    const float2 n2 = fma2(dup2(vis), make_float2(hn.x, hn.y), make_float2(S.nrm.x, S.nrm.y));
    S.nrm.x = n2.x;
    S.nrm.y = n2.y;
    S.nrm.z += vis * hn.z;
    if (CT == 3) {
        const float4 uvs = rec(kChunkUvs);
        const float2 uv = block_uv(H, rec(kChunkUvm), make_float2(uvs.x, uvs.y));
        const Bilerp B = bilerp(__float_as_int(uvs.z), __float_as_int(uvs.w), __float_as_int(rec(kChunkNop).w),
                                clamp01(uv.x), clamp01(uv.y), FIX || !(a.settings & (1 << 2)));
        float c[4][3];
        fetch3<TM>(a.tex, B, c);
        float2 v = mul2(dup2(B.w00), make_float2(c[0][0], c[0][1]));
        v = fma2(dup2(B.w01), make_float2(c[1][0], c[1][1]), v);
        v = fma2(dup2(B.w10), make_float2(c[2][0], c[2][1]), v);
        v = fma2(dup2(B.w11), make_float2(c[3][0], c[3][1]), v);
        const float2 t2 = fma2(dup2(vis), v, make_float2(S.tex[0], S.tex[1]));
        S.tex[0] = t2.x;
        S.tex[1] = t2.y;
        S.tex[2] += vis * (B.w00 * c[0][2] + B.w01 * c[1][2] + B.w10 * c[2][2] + B.w11 * c[3][2]);
    }
    const float t_view = H.tcam;
    if (S.T > 0.5f) { S.depth = t_view; S.didx = idx; }
    const float dv = (!FIX && (a.settings & (1 << 10)))
                         ? (kTFar * t_view - kTFar * kTNear) / ((kTFar - kTNear) * t_view) : H.t;
    S.reg += vis * (dv * dv * S.ts.x + S.ts.z - 2.f * dv * S.ts.y);
    S.ts.x += vis;
    const float2 s2 = fma2(dup2(vis), make_float2(dv, dv * dv), make_float2(S.ts.y, S.ts.z));
    S.ts.y = s2.x;
    S.ts.z = s2.y;
    S.T = next_T;
    S.cur = idx;
}

// T at or below this: a splat that the cull dropped (alpha < 1/255) could
// still end the pixel, since T (1 - alpha) <= 1e-4 is tested before alpha.
constexpr float kTClose = 1.01e-4f;

// Walks the rest of the list, every splat of it, for the one pixel of lane
// `src` whose T has come that close to the end; its lane's state S is brought
// to the end of the pixel.  The warp evaluates 32 splats at a time and acts on
// the first that ends the pixel or still contributes.
template <int TM, int CT, int FIX>
__device__ __forceinline__ void finish_close(FwdPix<CT>& S, const SceneArgs& a, const BlockArgs& ba, const Block& J,
                                             int src, int from, unsigned lane) {
    PixelRay P;
    {
        View V;
        V.fx = J.fx; V.fy = J.fy; V.cx = J.cx; V.cy = J.cy;
        P = make_pixel(V, J.y0 + lane_row(src), J.x0 + lane_col(src));
    }
    const bool use_blur = !FIX && (a.settings & (1 << 9)) != 0;
    float T = __shfl_sync(kFull, S.T, src);
    for (int base = from; base < J.range.y; base += 32) {
        const int i = base + (int)lane;
        const bool in = i < J.range.y;
        float alpha = 0.f;
        bool skip = true;
        Hit H;
        const int gid = in ? a.gids[i] : 0;
        if (in) {
            const GlobalRec rec{ J.recs[gid].c };
            float opac, nbf, bf, e, eb;
            H = block_hit(a, ba, J.view, rec, gid, P, opac);
            alpha = block_alpha<FIX>(H, opac, use_blur, J.recs + gid, P, nbf, bf, e, eb);
            skip = H.t < kTNear || H.t > kTFar || alpha < kAlphaMin;
        }
        unsigned todo = __ballot_sync(kFull, in);
        while (todo) {
            const bool ends = in && T * (1.f - alpha) <= kTDone;
            const unsigned me = __ballot_sync(kFull, ends) & todo, mc = __ballot_sync(kFull, in && !skip) & todo;
            if (!(me | mc)) break;
            const int f = __ffs(me | mc) - 1;
            if ((me >> f) & 1u) return;
            // the splat of lane f contributes
            const int g = __shfl_sync(kFull, gid, f);
            if ((int)lane == src) {
                const GlobalRec rec{ J.recs[g].c };
                float opac, nbf, bf, e, eb;
                const Hit Hs = block_hit(a, ba, J.view, rec, g, P, opac);
                const float as = block_alpha<FIX>(Hs, opac, use_blur, J.recs + g, P, nbf, bf, e, eb);
                blend<TM, CT, FIX>(S, a, rec, Hs, as, S.T * (1.f - as), base + f);
            }
            T = __shfl_sync(kFull, S.T, src);
            todo &= f == 31 ? 0u : ~0u << (f + 1);
        }
    }
}

template <int TM, int CT, int FIX>
__global__ void __launch_bounds__(32 * kBlockWarps, kFwdCtas) 
    fwd_block_kernel(const __grid_constant__ SceneArgs a, const __grid_constant__ BlockArgs ba, FwdOut o) {
    __shared__ FwdMem mem[kBlockWarps];
    const unsigned lane = threadIdx.x & 31;
    FwdMem& M = mem[threadIdx.x >> 5];
    Block J;
    if (!load_block(ba, (int)blockIdx.x * kBlockWarps + (int)(threadIdx.x >> 5), J)) return;
    const bool use_blur = !FIX && (a.settings & (1 << 9)) != 0;
    const int pi = J.y0 + lane_row(lane), pj = J.x0 + lane_col(lane);
    const bool inside = pi < J.H && pj < J.W;
    PixelRay P;
    {
        View V;
        V.fx = J.fx; V.fy = J.fy; V.cx = J.cx; V.cy = J.cy;
        P = make_pixel(V, pi, pj);
    }
    FwdPix<CT> S;
    S.T = 1.f;
    S.depth = S.reg = 0.f;
    S.cur = 0;
    S.didx = -1;
    S.out = S.nrm = S.ts = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < (CT > 0 ? CT : 1); c++) S.tex[c] = 0.f;
    bool done = !inside;
    int close = -1;  // list position at which T came close to the end
    const float fx0 = (float)J.x0 + 0.5f, fy0 = (float)J.y0 + 0.5f;
    int pos = J.range.x, n = 0;
    for (;;) {
        const unsigned live = __ballot_sync(kFull, !done);
        if (!live) break;
        n = fill_queue<1>(M.q, n, pos, J.range.y, a.gids, J.recs, fx0, fy0, live, lane);
        if (n == 0) break;
        const int ns = min(n, 32);
        stage_records(M.rec, M.q, ns, J.recs, lane);
        unsigned bits = transpose32((int)lane < ns ? M.q.mask[lane] : 0u, lane);
        if (done) bits = 0;
        cp_async_wait();
        __syncwarp();
        while (bits) {
            const int k = __ffs(bits) - 1;
            bits &= bits - 1;
            const StagedRec<kFwdChunks> rec(M.rec, k);
            float opac, nbf, bf, e, eb;
            const Hit H = block_hit(a, ba, J.view, rec, M.q.gid[k], P, opac);
            const float alpha = block_alpha<FIX>(H, opac, use_blur, FIX ? nullptr : J.recs + M.q.gid[k], P, nbf, bf, e, eb);
            const bool skip = H.t < kTNear || H.t > kTFar || alpha < kAlphaMin;
            const float next_T = S.T * (1.f - alpha);
            if (next_T <= kTDone) {
                done = true;
                bits = 0;
            } else if (!skip) {
                const int idx = M.q.idx[k];
                blend<TM, CT, FIX>(S, a, rec, H, alpha, next_T, idx);
                if (next_T <= kTClose) {
                    close = idx;
                    done = true;
                    bits = 0;
                }
            }
        }
        __syncwarp();
        n = pop_queue(M.q, n, lane);
    }
    for (unsigned cm = __ballot_sync(kFull, close >= 0); cm; cm &= cm - 1) {
        const int src = __ffs(cm) - 1;
        finish_close<TM, CT, FIX>(S, a, ba, J, src, __shfl_sync(kFull, close, src) + 1, lane);
    }
    if (!inside) return;
    const size_t pix = J.pix + (size_t)pi * J.W + pj;
    o.final_T[pix] = S.T;
    o.final_idx[pix] = S.cur;
    o.depth_idx[pix] = S.didx;
    o.img[pix] = make_float3(S.out.x + S.T * a.bg[0], S.out.y + S.T * a.bg[1], S.out.z + S.T * a.bg[2]);
    o.normal[pix] = S.nrm;
    o.depth[pix] = S.depth;
    o.reg[pix] = S.reg;
    o.reg_s[pix] = S.ts;
#pragma unroll
    for (int c = 0; c < CT; c++) o.tex[pix * CT + c] = S.tex[c];
}

// ---------------------------------------------------------------------------
// Launches
// ---------------------------------------------------------------------------
// The block kernels take tile widths that are multiples of 8 (8 or 16), no
// texture or three channels, and prebuilt records; the tile kernels of
// raster.cu take the rest, and the alpha-visualisation mode.
bool blocks_apply(int bw, int C, int settings, const RecAll* recs) {
    return (bw & 7) == 0 && (C == 0 || C == 3) && recs && !(settings & (1 << 16));
}

int launch_fwd_blocks(const SceneArgs& a, const BlockArgs& ba, const FwdOut& o, int texmode, cudaStream_t stream) {
    const long long blocks = (long long)ba.total_tiles * ((ba.bw >> 3) * (ba.bw >> 2));
    const long long grid = (blocks + kBlockWarps - 1) / kBlockWarps;
    if (grid > 0x7fffffffLL) return GSTEX_ERR_UNSUPPORTED;
    const bool fix = (a.settings & kFixedFwdMask) == 0;
    void (*k)(const SceneArgs, const BlockArgs, FwdOut);
    if (a.C == 0) k = fix ? fwd_block_kernel<0, 0, 1> : fwd_block_kernel<0, 0, 0>;
    else if (texmode == 1) k = fix ? fwd_block_kernel<1, 3, 1> : fwd_block_kernel<1, 3, 0>;
    else k = fix ? fwd_block_kernel<0, 3, 1> : fwd_block_kernel<0, 3, 0>;
    k<<<(unsigned)grid, 32 * kBlockWarps, 0, stream>>>(a, ba, o);
    return check_launch("forward blocks");
}

}  // namespace gstex
