// Block compositor: the textured 2D-Gaussian forward and backward with one
// warp per 8x4 block of pixels.
//
// Reference: csrc/texture.cu:11-329 and 331-760.  A splat reaches about a tenth of
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
// What bounds it: the L1 data path (73% of its cycles at 24 warps per SM, 78% with
// float32 texels; half of it staged records, a third to a half texel gathers),
// then the ALUs (49%).  Measured
// against the list walk with one CTA per tile (forward kernel alone): 32 views
// with 81M intersections, bf16 texels, 8x8 tiles 17.4 -> 8.7 ms; 8 clustered
// full-HD views 9.2 -> 5.2 ms; one 800x800 view, 16x16 tiles 232 -> 59 us; one
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

__device__ __forceinline__ PixelRay block_pixel(const Block& J, int pi, int pj) {
    View V;
    V.fx = J.fx; V.fy = J.fy; V.cx = J.cx; V.cy = J.cy;
    return make_pixel(V, pi, pj);
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
// (Upwards, positions are compared as unsigned numbers: 32 beyond the end may
// pass 31 bits.  Downwards, `end` may be -1.)
template <int DIR>
__device__ __forceinline__ int fill_queue(Queue& q, int n, int& pos, int end, const int32_t* __restrict__ gids,
                                          const RecAll* __restrict__ recs, float fx0, float fy0, unsigned live,
                                          unsigned lane) {
    while (n < 32 && (DIR > 0 ? (unsigned)pos < (unsigned)end : pos > end)) {
        const int i = DIR > 0 ? (int)((unsigned)pos + lane) : pos - (int)lane;
        int gid = 0;
        unsigned m = 0;
        if (DIR > 0 ? (unsigned)i < (unsigned)end : i > end) {
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
        pos = DIR > 0 ? (int)((unsigned)pos + 32u) : pos - 32;
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

// Staged records: NCH chunks (from kChunkOrg on) of 32 records.  An odd number
// of 16-byte words a record keeps lanes that read one chunk of neighbouring
// records on different banks, and a record is written as one run (chunk-major
// rows of 33: forward 8.94 instead of 8.70 ms, backward 22.6 instead of 22.3 on
// 32 views; copied by cp.async.bulk, one instruction a record: 9.17 and 24.3).
template <int NCH>
struct Staged {
    float4 c[32][NCH | 1];
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
        if (r < n && ch < NCH) cp_async16(&S.c[r][ch], recs[q.gid[r]].c + kChunkOrg + ch);
    }
}

// Chunk access of one record, staged or in device memory.
template <int NCH>
struct StagedRec {
    const float4* p;
    __device__ __forceinline__ StagedRec(const Staged<NCH>& S, int k) : p(S.c[k]) {}
    __device__ __forceinline__ float4 operator()(int chunk) const { return p[chunk - kChunkOrg]; }
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

// Weights of the four corners; beyond a chart's last row or column two texels
// are one, and its weights are added up.
__device__ __forceinline__ void corner_weights(const Bilerp& B, float (&wts)[4]) {
    wts[0] = B.w00; wts[1] = B.w01; wts[2] = B.w10; wts[3] = B.w11;
    if (B.i10 == B.i00) {
        wts[0] += wts[2]; wts[1] += wts[3];
        wts[2] = wts[3] = 0.f;
    }
    if (B.i01 == B.i00) {
        wts[0] += wts[1]; wts[2] += wts[3];
        wts[1] = wts[3] = 0.f;
    }
}

__device__ __forceinline__ int chart_start(float4 nop) { return (int)(__float_as_uint(nop.w) & ~kCoarseChart); }
__device__ __forceinline__ bool is_coarse(float4 nop) { return (__float_as_uint(nop.w) & kCoarseChart) != 0u; }

// uv of the hit before clamping (hit_uv on the stored chunks).
__device__ __forceinline__ float2 block_uv(const Hit& H, float4 uvm, float2 uv0) {
    if (H.direct) return make_float2(H.tu, H.tv);
    const float2 t = fma2(make_float2(uvm.y, uvm.w), dup2(H.dv), mul2(make_float2(uvm.x, uvm.z), dup2(H.du)));
    return fma2(t, dup2(H.inv), uv0);
}

// ---------------------------------------------------------------------------
// The walk, front to back, shared by the forward and by texture editing: Pix
// is a pixel's state, with its transmittance T and take(), which applies one
// contributing pair.
// ---------------------------------------------------------------------------
constexpr int kFwdChunks = 7;
template <int NCH>
struct WalkMem {
    Staged<NCH> rec;
    Queue q;
};

template <int TM, int CT, int FIX>
struct FwdPix {
    float T, depth, reg;
    int cur, didx;
    float3 out, nrm, ts;
    float tex[CT > 0 ? CT : 1];

    // Blends the pair into the pixel (texture.cu:222-296).
    template <class Rec>
    __device__ __forceinline__ void take(const SceneArgs& a, const Rec& rec, const Hit& H, float alpha, float next_T,
                                         int idx) {
        const float vis = alpha * T;
        const float4 col = rec(kChunkCol), nw = rec(kChunkNrm);
        const float2 o2 = fma2(make_float2(col.x, col.y), dup2(vis), make_float2(out.x, out.y));
        out.x = o2.x;
        out.y = o2.y;
        out.z = out.z + col.z * vis;
        float3 hn = f3(nw);
        if (!FIX && (a.settings & (1 << 15)) && H.nd > 0.f) hn = make_float3(-hn.x, -hn.y, -hn.z);
        const float2 n2 = fma2(dup2(vis), make_float2(hn.x, hn.y), make_float2(nrm.x, nrm.y));
        nrm.x = n2.x;
        nrm.y = n2.y;
        nrm.z += vis * hn.z;
        if (CT == 3) {
            const float4 uvs = rec(kChunkUvs);
            const float2 uv = block_uv(H, rec(kChunkUvm), make_float2(uvs.x, uvs.y));
            const Bilerp B = bilerp(__float_as_int(uvs.z), __float_as_int(uvs.w), chart_start(rec(kChunkNop)),
                                    clamp01(uv.x), clamp01(uv.y), FIX || !(a.settings & (1 << 2)));
            float c[4][3];
            fetch3<TM>(a.tex, B, c);
            float2 v = mul2(dup2(B.w00), make_float2(c[0][0], c[0][1]));
            v = fma2(dup2(B.w01), make_float2(c[1][0], c[1][1]), v);
            v = fma2(dup2(B.w10), make_float2(c[2][0], c[2][1]), v);
            v = fma2(dup2(B.w11), make_float2(c[3][0], c[3][1]), v);
            const float2 t2 = fma2(dup2(vis), v, make_float2(tex[0], tex[1]));
            tex[0] = t2.x;
            tex[1] = t2.y;
            tex[2] += vis * (B.w00 * c[0][2] + B.w01 * c[1][2] + B.w10 * c[2][2] + B.w11 * c[3][2]);
        }
        const float t_view = H.tcam;
        if (T > 0.5f) { depth = t_view; didx = idx; }
        const float dv = (!FIX && (a.settings & (1 << 10)))
                             ? (kTFar * t_view - kTFar * kTNear) / ((kTFar - kTNear) * t_view) : H.t;
        reg += vis * (dv * dv * ts.x + ts.z - 2.f * dv * ts.y);
        ts.x += vis;
        const float2 s2 = fma2(dup2(vis), make_float2(dv, dv * dv), make_float2(ts.y, ts.z));
        ts.y = s2.x;
        ts.z = s2.y;
        T = next_T;
        cur = idx;
    }
};

// T at or below this: a splat that the cull dropped (alpha < 1/255) could
// still end the pixel, since T (1 - alpha) <= 1e-4 is tested before alpha.
constexpr float kTClose = 1.01e-4f;

// Walks the rest of the list, every splat of it, for the one pixel of lane
// `src` whose T has come that close to the end; its lane's state S is brought
// to the end of the pixel.  The warp evaluates 32 splats at a time and acts on
// the first that ends the pixel or still contributes.
template <int FIX, class Pix>
__device__ __forceinline__ void finish_close(Pix& S, const SceneArgs& a, const BlockArgs& ba, const Block& J, int src,
                                             int from, unsigned lane) {
    const PixelRay P = block_pixel(J, J.y0 + lane_row(src), J.x0 + lane_col(src));
    const bool use_blur = !FIX && (a.settings & (1 << 9)) != 0;
    float T = __shfl_sync(kFull, S.T, src);
    for (unsigned base = from; base < (unsigned)J.range.y; base += 32) {
        const unsigned i = base + lane;
        const bool in = i < (unsigned)J.range.y;
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
                S.take(a, rec, Hs, as, S.T * (1.f - as), (int)base + f);
            }
            T = __shfl_sync(kFull, S.T, src);
            todo &= f == 31 ? 0u : ~0u << (f + 1);
        }
    }
}

// Walks the block's list; `done`: the lane has no pixel.
template <int FIX, int NCH, class Pix>
__device__ __forceinline__ void walk_list(WalkMem<NCH>& M, const SceneArgs& a, const BlockArgs& ba, const Block& J,
                                          const PixelRay& P, Pix& S, bool done, unsigned lane) {
    const bool use_blur = !FIX && (a.settings & (1 << 9)) != 0;
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
            const StagedRec<NCH> rec(M.rec, k);
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
                S.take(a, rec, H, alpha, next_T, idx);
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
        finish_close<FIX>(S, a, ba, J, src, __shfl_sync(kFull, close, src) + 1, lane);
    }
}

template <int TM, int CT, int FIX>
__global__ void __launch_bounds__(32 * kBlockWarps, kFwdCtas)
    fwd_block_kernel(const __grid_constant__ SceneArgs a, const __grid_constant__ BlockArgs ba, FwdOut o) {
    __shared__ WalkMem<kFwdChunks> mem[kBlockWarps];
    const unsigned lane = threadIdx.x & 31;
    Block J;
    if (!load_block(ba, (int)blockIdx.x * kBlockWarps + (int)(threadIdx.x >> 5), J)) return;
    const int pi = J.y0 + lane_row(lane), pj = J.x0 + lane_col(lane);
    const bool inside = pi < J.H && pj < J.W;
    FwdPix<TM, CT, FIX> S;
    S.T = 1.f;
    S.depth = S.reg = 0.f;
    S.cur = 0;
    S.didx = -1;
    S.out = S.nrm = S.ts = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < (CT > 0 ? CT : 1); c++) S.tex[c] = 0.f;
    walk_list<FIX>(mem[threadIdx.x >> 5], a, ba, J, block_pixel(J, pi, pj), S, !inside, lane);
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
// Texture editing (csrc/texture_edit.cu:11-236): the forward walk, and for every
// contributing pair whose camera depth lies in the pixel's [lower, upper] range
// a bilinear splat of (r a, g a, b a, a, 1) of the edited pixel into the chart's
// [T, 5] texels.  800x800, 100k Gaussians: 190 us with one CTA per tile that
// derives its records -> 74 us.
// ---------------------------------------------------------------------------
constexpr int kEditChunks = 5;  // up to kChunkUvs
struct EditPix {
    float T;
    float vals[4], lo, hi;
    float* texels;

    template <class Rec>
    __device__ __forceinline__ void take(const SceneArgs&, const Rec& rec, const Hit& H, float, float next_T, int) {
        T = next_T;
        if (!(H.tcam >= lo && H.tcam <= hi)) return;
        const float4 uvs = rec(kChunkUvs);
        const float2 uv = block_uv(H, rec(kChunkUvm), make_float2(uvs.x, uvs.y));
        const Bilerp B = bilerp(__float_as_int(uvs.z), __float_as_int(uvs.w), chart_start(rec(kChunkNop)),
                                clamp01(uv.x), clamp01(uv.y), true);
        const int rows[4] = { B.i00, B.i01, B.i10, B.i11 };
        float wts[4] = { B.w00, B.w01, B.w10, B.w11 };
        // (an infinite value times a weight of 0 is added as the NaN it is)
        const bool finite = fabsf(vals[0]) + fabsf(vals[1]) + fabsf(vals[2]) + fabsf(vals[3]) < INFINITY;
        if (finite) corner_weights(B, wts);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (finite && wts[q] == 0.f) continue;
            float* dst = texels + 5 * (size_t)rows[q];
#pragma unroll
            for (int c = 0; c < 4; c++) atomicAdd(dst + c, wts[q] * vals[c]);
            atomicAdd(dst + 4, wts[q]);
        }
    }
};

template <int FIX>
__global__ void __launch_bounds__(32 * kBlockWarps, kFwdCtas)
    edit_block_kernel(const __grid_constant__ SceneArgs a, const __grid_constant__ BlockArgs ba, EditIO E) {
    __shared__ WalkMem<kEditChunks> mem[kBlockWarps];
    const unsigned lane = threadIdx.x & 31;
    Block J;
    if (!load_block(ba, (int)blockIdx.x * kBlockWarps + (int)(threadIdx.x >> 5), J)) return;
    const int pi = J.y0 + lane_row(lane), pj = J.x0 + lane_col(lane);
    const bool inside = pi < J.H && pj < J.W;
    EditPix S;
    S.T = 1.f;
    S.vals[0] = S.vals[1] = S.vals[2] = S.vals[3] = S.lo = S.hi = 0.f;
    S.texels = E.out;
    if (inside) {
        const size_t pix = J.pix + (size_t)pi * J.W + pj;
        const float3 c = E.img[pix];
        const float m = E.alpha[pix];
        S.vals[0] = c.x * m; S.vals[1] = c.y * m; S.vals[2] = c.z * m; S.vals[3] = m;
        S.lo = E.lower[pix];
        S.hi = E.upper[pix];
    }
    walk_list<FIX>(mem[threadIdx.x >> 5], a, ba, J, block_pixel(J, pi, pj), S, !inside, lane);
}

// ---------------------------------------------------------------------------
// Backward.  The walk is the forward's, back to front; a splat's gradients are
// sums over pixels (finalize_kernel turns 21 of them into the parameters'
// gradients), and the pixels of a step are at different splats.  So every lane
// first steps back over its pixel's pairs with as many staged splats as there
// is room for (kPairs) and leaves eight numbers per pair in shared memory; then the roles turn (one more transpose):
// every lane takes a splat and sums the pairs of its pixels in registers,
// without the shuffles and shared-memory atomics of a reduction over the warp,
// and adds the sums to the splat's row with 16-byte atomics.
//
// What bounds it: the L1 data path (75% of its cycles; a 16-byte reduction
// takes about a cycle per lane there) and the latency of its chains at 16 warps
// per SM.  Of 22.1 ms on 32 views (36.6 ms with the list walk, its moment
// reduction by shuffles and 8-lane groups) the scan, staging and ray-plane
// solves take 6 ms, the adjoint 4, texel reads 3.5, texel atomics 4 and the
// sums 5.  8 clustered full-HD views: 22.3 -> 13.2 ms; one 800x800 view of 1x1
// charts 254 -> 108 us; one full-HD view of large splats 36.0 -> 7.0 ms (where
// the list walk also staged every splat behind the last contributor).  The
// pixels' upstream gradients by shuffles instead of from shared memory in the
// sums: 23.7 ms.
// ---------------------------------------------------------------------------
constexpr int kBwdChunks = 8;
// Pairs between two summations, and CTAs per SM (at most 128 registers): what
// fits 8 CTAs' shared memory (32 staged splats have 230 pairs on average; with
// 192, 1% slower; with 224, which fit 7 CTAs, 23.5 instead of 22.1 ms).  Pairs
// are placed splat by splat, so the room is used up and a splat is summed once:
// 7 rounds of one pair per pixel in the same room took 23.6 instead of 22.8 ms
// on 32 views, 14.4 instead of 13.7 ms on 8 clustered ones.
constexpr int kPairs = 220;
constexpr int kBwdCtas = 8;
struct BwdMem {
    Staged<kBwdChunks> rec;
    float4 pair[2][kPairs];       // (vis, e v_alpha, v_sigma, v_t / (n . r)), (v_u, v_v, l1s, l2s), splat by splat
    float4 pix[2][32];            // the pixels' upstream colour and normal x; texture gradients
    float2 pix_n[32];             // normal y, z
    uint2 place[32];              // first pair of a staged splat; its pixels that may have one
    uint8_t slot[32];             // splats with pairs
    Queue q;
};

template <int CT>
struct BwdState {
    float T, vT_run;
    float3 sfin, vout, vnorm;
    int dfin, bfin;
    float vdepth, vreg;
    float vtex[CT > 0 ? CT : 1];
};

// Adds three values to three neighbouring floats: the two that share an 8-byte
// word at once.
__device__ __forceinline__ void add3(float* dst, float x, float y, float z) {
    const bool odd = ((uintptr_t)dst & 4) != 0;
    atomicAdd(reinterpret_cast<float2*>(dst + (odd ? 1 : 0)), odd ? make_float2(y, z) : make_float2(x, y));
    atomicAdd(dst + (odd ? 0 : 2), odd ? x : z);
}

// Adds two neighbouring texels' three values each, as the two or three 16-byte
// words they lie in; the rest of these gets + 0, so 12 bytes before and after
// the texels have to belong to the buffer.
__device__ __forceinline__ void add6(float* dst, float2 a01, float a2, float2 b01, float b2) {
    const bool s1 = ((uintptr_t)dst & 4) != 0, s2 = ((uintptr_t)dst & 8) != 0;
    const float g0 = s1 ? 0.f : a01.x, g1 = s1 ? a01.x : a01.y, g2 = s1 ? a01.y : a2, g3 = s1 ? a2 : b01.x;
    const float g4 = s1 ? b01.x : b01.y, g5 = s1 ? b01.y : b2, g6 = s1 ? b2 : 0.f;
    // (an offset from dst: an address made from an integer is no longer known to
    // be global memory, and such atomics are far slower)
    float4* w = reinterpret_cast<float4*>(dst - (s1 ? 1 : 0) - (s2 ? 2 : 0));
    atomicAdd(w, make_float4(s2 ? 0.f : g0, s2 ? 0.f : g1, s2 ? g0 : g2, s2 ? g1 : g3));
    if (s2 || b01.x != 0.f || b01.y != 0.f || b2 != 0.f)
        atomicAdd(w + 1, make_float4(s2 ? g2 : g4, s2 ? g3 : g5, s2 ? g4 : g6, s2 ? g5 : 0.f));
    if (s1 && s2) atomicAdd(&w[2].x, b2);
}

// Texel gradients of one pair: gv = vis * upstream texture gradient.  The cost
// is the number of atomics, which 32 lanes on few texels queue up for: float32
// texels (12 bytes, T of them) take 4 to 6 instead of 12 (with 8, three values
// as 8 + 4 bytes: second figure): full HD with 48 pixels a texel 8.5 -> 7.3 ->
// 7.0 ms of backward, a 253x187 view 182 -> 150 -> 132 us, four views with less
// than two pixels a texel 213 -> 209 -> 211 us.
template <int TM, int FIX>
__device__ __forceinline__ void add_texel_grads(float* __restrict__ v_texgrad, int T, const Bilerp& B, float2 gv01,
                                                float gv2) {
    if (gv01.x == 0.f && gv01.y == 0.f && gv2 == 0.f) return;
    const int rows[4] = { B.i00, B.i01, B.i10, B.i11 };
    float wts[4];
    corner_weights(B, wts);
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
        const float w0 = wts[q], w1 = wts[q + 1];
        float2 a01 = mul2(dup2(w0), gv01), b01 = mul2(dup2(w1), gv01);
        float a2 = w0 * gv2, b2 = w1 * gv2;
        if (TM == 0) {
            // a corner without weight adds 0 whatever the gradient: the word it shares may
            // be another chart's texel, and 0 times infinity is not 0 (of two bilinear
            // weights the first is never the only 0)
            if (!FIX && w0 == 0.f) { a01 = make_float2(0.f, 0.f); a2 = 0.f; }
            if (w1 == 0.f) { b01 = make_float2(0.f, 0.f); b2 = 0.f; }
        }
        if (TM == 1) {
            if (w0 != 0.f) atomicAdd(reinterpret_cast<float4*>(v_texgrad) + rows[q], make_float4(a01.x, a01.y, a2, 0.f));
            if (w1 != 0.f)
                atomicAdd(reinterpret_cast<float4*>(v_texgrad) + rows[q + 1], make_float4(b01.x, b01.y, b2, 0.f));
        } else if (w0 != 0.f || w1 != 0.f) {
            float* dst = v_texgrad + 3 * (size_t)rows[q];
            if (rows[q] > 0 && rows[q] + 3 <= T) {  // (texel rows[q + 1] is the next one, or w1 is 0)
                add6(dst, a01, a2, b01, b2);
            } else {
                add3(dst, a01.x, a01.y, a2);
                if (w1 != 0.f) add3(v_texgrad + 3 * (size_t)rows[q + 1], b01.x, b01.y, b2);
            }
        }
    }
}

// Adjoint of one contributing pair (csrc/texture.cu:577-708): steps the pixel's
// recurrences back over it, adds its texel gradients and returns what the
// per-splat sums need of it.
template <int TM, int CT, int FIX>
__device__ __forceinline__ void pair_adjoint(BwdState<CT>& S, const SceneArgs& a, const BwdArgs& g,
                                             const StagedRec<kBwdChunks>& rec, const Hit& H, const PixelRay& P, int idx,
                                             float opac, float alpha, float nbf, float bf, float e, float eb, float4& q0,
                                             float4& q1) {
    const bool use_ndc = !FIX && (a.settings & (1 << 10)), prop_uv = FIX || (a.settings & (1 << 8));
    const bool bilinear = FIX || !(a.settings & (1 << 2));
    const float4 col = rec(kChunkCol), nw = rec(kChunkNrm), ray = rec(kChunkRay);
    S.T = __fdividef(S.T, 1.f - alpha);
    const float T = S.T;
    const float vis = alpha * T;
    float v_vis = col.x * S.vout.x + col.y * S.vout.y + col.z * S.vout.z + nw.x * S.vnorm.x + nw.y * S.vnorm.y +
                  nw.z * S.vnorm.z;
    float v_u = 0.f, v_v = 0.f;
    float2 duv = make_float2(0.f, 0.f);  // uv of the hit, relative to uv0
    if (CT == 3) {
        const float4 uvs = rec(kChunkUvs);
        const float2 uv = block_uv(H, rec(kChunkUvm), make_float2(uvs.x, uvs.y));
        duv = sub2(uv, make_float2(uvs.x, uvs.y));
        const int h = __float_as_int(uvs.z), w = __float_as_int(uvs.w);
        const float4 nop = rec(kChunkNop);
        const Bilerp B = bilerp(h, w, chart_start(nop), clamp01(uv.x), clamp01(uv.y), bilinear);
        float c[4][3];
        fetch3<TM>(a.tex, B, c);
        // channels 0 and 1 as f32x2 pairs, channel 2 alone
        const float2 c0 = make_float2(c[0][0], c[0][1]), c1 = make_float2(c[1][0], c[1][1]);
        const float2 c2 = make_float2(c[2][0], c[2][1]), c3 = make_float2(c[3][0], c[3][1]);
        const float2 vt = make_float2(S.vtex[0], S.vtex[1]);
        float2 val = mul2(dup2(B.w00), c0);
        val = fma2(dup2(B.w01), c1, val);
        val = fma2(dup2(B.w10), c2, val);
        val = fma2(dup2(B.w11), c3, val);
        const float val2 = B.w00 * c[0][2] + B.w01 * c[1][2] + B.w10 * c[2][2] + B.w11 * c[3][2];
        const float2 gv01 = mul2(dup2(vis), vt);
        const float gv2 = vis * S.vtex[2];
        if (bilinear && prop_uv) {
            // d(val)/d(tcx) = (1 - fy)(c10 - c00) + fy (c11 - c01),
            // d(val)/d(tcy) = (1 - fx)(c01 - c00) + fx (c11 - c10)
            const float2 du = fma2(dup2(B.fy), sub2(c3, c1), mul2(dup2(1.f - B.fy), sub2(c2, c0)));
            const float2 dv = fma2(dup2(B.fx), sub2(c3, c2), mul2(dup2(1.f - B.fx), sub2(c1, c0)));
            const float du2 = (1.f - B.fy) * (c[2][2] - c[0][2]) + B.fy * (c[3][2] - c[1][2]);
            const float dv2 = (1.f - B.fx) * (c[1][2] - c[0][2]) + B.fx * (c[3][2] - c[2][2]);
            const float2 pu = mul2(gv01, du), pv = mul2(gv01, dv);
            v_u = (float)h * (pu.x + pu.y + gv2 * du2);
            v_v = (float)w * (pv.x + pv.y + gv2 * dv2);
        }
        const float2 vs = mul2(val, vt);
        v_vis += vs.x + vs.y + val2 * S.vtex[2];
        // (a coarse chart's are summed over the pixels first, but for pairs in the direct form)
        if (!is_coarse(nop) || H.direct) add_texel_grads<TM, FIX>(g.v_texgrad, a.T, B, gv01, gv2);
    }
    float v_alpha = T * v_vis - T * S.vT_run;
    float vT_cur = alpha * v_vis + (1.f - alpha) * S.vT_run;
    const float t_view = H.tcam;
    float v_t = 0.f, v_t_ndc = 0.f, v_w = 0.f;
    if (use_ndc) {
        const float t_ndc = (kTFar * t_view - kTFar * kTNear) / ((kTFar - kTNear) * t_view);
        v_t_ndc = 2.f * (vis * t_ndc * S.sfin.x - vis * S.sfin.y) * S.vreg;
        v_w = (t_ndc * t_ndc * S.sfin.x - 2.f * t_ndc * S.sfin.y + S.sfin.z) * S.vreg;
    } else {
        v_t = 2.f * (vis * H.t * S.sfin.x - vis * S.sfin.y) * S.vreg;
        v_w = (H.t * H.t * S.sfin.x - 2.f * H.t * S.sfin.y + S.sfin.z) * S.vreg;
    }
    v_alpha += v_w * T;
    vT_cur += v_w * alpha;
    S.vT_run = vT_cur;
    const float v_sigma = -nbf * opac * e * v_alpha;
    // sigma = (l1s^2 + l2s^2) / 2 with l_ks = l_k / s_k.  A point l of the
    // plane has a . r = (l + a . mu) / t along the ray r, so dsigma/dt = sum_k
    // l_ks (l_ks + a_k . mu / s_k) / t, and likewise for the uv
    float v_ray = H.l1s * v_sigma * (H.l1s + ray.x) + H.l2s * v_sigma * (H.l2s + ray.y);
    if (prop_uv) v_ray += v_u * (duv.x + ray.z) + v_v * (duv.y + ray.w);
    v_t += v_ray * __fdividef(1.f, H.t);
    float v_t_view = 0.f;
    if (idx == S.dfin) v_t_view += S.vdepth;
    if (use_ndc) v_t_view += (kTFar * kTNear) / ((kTFar - kTNear) * t_view * t_view) * v_t_ndc;
    v_t += P.idn * v_t_view;
    q0 = make_float4(vis, (nbf * e + bf * eb) * v_alpha, v_sigma, v_t * (P.dn * H.inv));
    q1 = make_float4(v_u, v_v, H.l1s, H.l2s);
}

// Texel gradients of a coarse chart (kCoarseChart): atomics of 32 lanes on the
// same texel are served one after the other, so the lane sums a staged splat's pairs over
// its pixels (own) as long as they fall between the same four texels.  k: the
// lane's staged splat, whose pairs start at `first` in the order of `may`.  Pairs
// in the direct form are not among them: the fast form, which this takes again,
// has no uv where the ray lies in the splat's plane (pair_adjoint adds theirs).
template <int TM, int FIX>
__device__ __forceinline__ void add_coarse_texel_grads(const BwdMem& M, const SceneArgs& a, float* __restrict__ v_texgrad,
                                                       int k, unsigned own, unsigned may, int first, float fx0,
                                                       float fy0) {
    const StagedRec<kBwdChunks> rec(M.rec, k);
    const float4 nop = rec(kChunkNop), uvs = rec(kChunkUvs), uvm = rec(kChunkUvm);
    RecHot Hr;
    Hr.org = rec(kChunkOrg);
    Hr.lc = make_float4(0.f, 0.f, 0.f, 0.f);
    Hr.nop = make_float4(nop.x, nop.y, nop.z, 0.f);
    Bilerp cell;
    cell.i00 = -1;
    float acc[4][3];
    auto flush = [&]() {
        const int rows[4] = { cell.i00, cell.i01, cell.i10, cell.i11 };
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (acc[q][0] == 0.f && acc[q][1] == 0.f && acc[q][2] == 0.f) continue;
            if (TM == 1) {
                atomicAdd(reinterpret_cast<float4*>(v_texgrad) + rows[q],
                          make_float4(acc[q][0], acc[q][1], acc[q][2], 0.f));
            } else {
                add3(v_texgrad + 3 * (size_t)rows[q], acc[q][0], acc[q][1], acc[q][2]);
            }
        }
    };
    for (; own; own &= own - 1) {
        const int p = __ffs(own) - 1;
        const float vis = M.pair[0][first + __popc(may & ((1u << p) - 1u))].x;
        const float4 vt = M.pix[1][p];
        PixelRay P;
        P.px = fx0 + (float)lane_col(p);
        P.py = fy0 + (float)lane_row(p);
        P.dn = 0.f;
        const Hit H = intersect(Hr, P);
        const float2 t = fma2(make_float2(uvm.y, uvm.w), dup2(H.dv), mul2(make_float2(uvm.x, uvm.z), dup2(H.du)));
        const float2 uv = fma2(t, dup2(H.inv), make_float2(uvs.x, uvs.y));
        const Bilerp B = bilerp(__float_as_int(uvs.z), __float_as_int(uvs.w), chart_start(nop), clamp01(uv.x),
                                clamp01(uv.y), FIX || !(a.settings & (1 << 2)));
        if (B.i00 != cell.i00) {  // (i00 fixes the other three)
            if (cell.i00 >= 0) flush();
            cell = B;
#pragma unroll
            for (int q = 0; q < 4; q++) acc[q][0] = acc[q][1] = acc[q][2] = 0.f;
        }
        const float gv[3] = { vis * vt.x, vis * vt.y, vis * vt.z };
        const float wts[4] = { B.w00, B.w01, B.w10, B.w11 };
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int c = 0; c < 3; c++) acc[q][c] += wts[q] != 0.f ? wts[q] * gv[c] : 0.f;
    }
    if (cell.i00 >= 0) flush();
}

// (The sums as asynchronous bulk additions from shared memory, 80 and 16 bytes a
// splat, took 23.5 instead of 22.5 ms on 32 views.)
// Adds the sums of one splat over the pixels of a block to its gradients (the
// moment rows of finalize_kernel).  m: 0-2 colour, 3 opacity, 4-6 l1^2, l2^2,
// l1 l2 times v_sigma, 7-8 l v_sigma, 9-11 (1, l1, l2) v_t / (n . r), 12-14
// normal, 15-16 v_uv, 17-20 l v_uv, 21-22 blur; l in units of the scales.
template <int FIX>
__device__ __forceinline__ void flush_moments(const float* m, const BlockArgs& ba, const BwdArgs& g, const Block& J,
                                              int gid, bool use_blur) {
    if (ba.vc_stride == 4) {
        atomicAdd(reinterpret_cast<float4*>(J.vcolors) + gid, make_float4(m[0], m[1], m[2], 0.f));
    } else {
        float* vc = J.vcolors + 3 * (size_t)gid;
        atomicAdd(vc + 0, m[0]);
        atomicAdd(vc + 1, m[1]);
        atomicAdd(vc + 2, m[2]);
    }
    float4* dst = reinterpret_cast<float4*>(g.moments + (size_t)gid * kMomStride);
#pragma unroll
    for (int q = 0; q < 4; q++)
        atomicAdd(dst + q, make_float4(m[3 + 4 * q], m[4 + 4 * q], m[5 + 4 * q], m[6 + 4 * q]));
    atomicAdd(reinterpret_cast<float2*>(dst + 4), make_float2(m[19], m[20]));
    if (!FIX && use_blur) {
        const float3 vmb = blur_mean_grad(block_view(ba, J.view), f3(__ldg(J.recs[gid].c + kChunkMu)), m[21], m[22]);
        float* vb = reinterpret_cast<float*>(dst + 5);
        atomicAdd(vb + 0, vmb.x);
        atomicAdd(vb + 1, vmb.y);
        atomicAdd(vb + 2, vmb.z);
    }
}

template <int TM, int CT, int FIX>
__global__ void __launch_bounds__(32 * kBlockWarps, kBwdCtas)
    bwd_block_kernel(const __grid_constant__ SceneArgs a, const __grid_constant__ BlockArgs ba, BwdArgs g) {
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned lane = threadIdx.x & 31;
    BwdMem& M = reinterpret_cast<BwdMem*>(smem)[threadIdx.x >> 5];
    Block J;
    if (!load_block(ba, (int)blockIdx.x * kBlockWarps + (int)(threadIdx.x >> 5), J)) return;
    if (J.range.x >= J.range.y) return;
    const bool use_blur = !FIX && (a.settings & (1 << 9)) != 0;
    const int pi = J.y0 + lane_row(lane), pj = J.x0 + lane_col(lane);
    const bool inside = pi < J.H && pj < J.W;
    const PixelRay P = block_pixel(J, pi, pj);
    const float3 z3 = make_float3(0.f, 0.f, 0.f);
    BwdState<CT> S;
    const size_t pix = inside ? J.pix + (size_t)pi * J.W + pj : 0;
    S.bfin = inside ? g.final_idx[pix] : -1;
    // splats beyond the last contributor of the block's pixels add nothing
    int pos = min(J.range.y - 1, __reduce_max_sync(kFull, S.bfin));
    if (pos < J.range.x) return;
    S.T = inside ? g.final_T[pix] : 1.f;
    S.sfin = inside ? g.reg_s[pix] : z3;
    S.dfin = inside ? g.depth_idx[pix] : -1;
    S.vout = inside ? ld_or(g.v_img, pix, z3) : z3;
    S.vdepth = inside ? ld_or(g.v_depth, pix, 0.f) : 0.f;
    S.vreg = inside ? ld_or(g.v_reg, pix, 0.f) : 0.f;
    S.vnorm = inside ? ld_or(g.v_normal, pix, z3) : z3;
    const float valph = inside ? ld_or(g.v_alpha, pix, 0.f) : 0.f;
#pragma unroll
    for (int c = 0; c < (CT > 0 ? CT : 1); c++) S.vtex[c] = (CT > 0 && inside && g.v_tex) ? g.v_tex[pix * CT + c] : 0.f;
    S.vT_run = a.bg[0] * S.vout.x + a.bg[1] * S.vout.y + a.bg[2] * S.vout.z - valph;
    M.pix[0][lane] = f4(S.vout, S.vnorm.x);
    M.pix_n[lane] = make_float2(S.vnorm.y, S.vnorm.z);
    if (CT == 3) M.pix[1][lane] = make_float4(S.vtex[0], S.vtex[CT > 1 ? 1 : 0], S.vtex[CT > 2 ? 2 : 0], 0.f);
    const float fx0 = (float)J.x0 + 0.5f, fy0 = (float)J.y0 + 0.5f;
    const unsigned live = __ballot_sync(kFull, S.bfin >= J.range.x), below = (1u << lane) - 1u;
    int n = 0;
    for (;;) {
        n = fill_queue<-1>(M.q, n, pos, J.range.x - 1, a.gids, J.recs, fx0, fy0, live, lane);
        if (n == 0) break;
        const int ns = min(n, 32);
        stage_records(M.rec, M.q, ns, J.recs, lane);
        unsigned todo = transpose32((int)lane < ns ? M.q.mask[lane] : 0u, lane);
        if (M.q.idx[0] > S.bfin) {  // skip the splats beyond this pixel's last contributor
            int k = 0;
#pragma unroll
            for (int step = 32; step > 0; step >>= 1)
                if (k + step <= ns && M.q.idx[k + step - 1] > S.bfin) k += step;
            todo = k >= 32 ? 0u : todo & (~0u << k);
        }
        if (!((live >> lane) & 1u)) todo = 0;
        cp_async_wait();
        __syncwarp();
        // room for the pairs: splat by splat, in pixel order; as many splats at
        // a time as there is room for
        const unsigned may = transpose32(todo, lane);
        int last = __popc(may);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, last, o);
            if ((int)lane >= o) last += y;
        }
        const int total = __shfl_sync(kFull, last, 31);
        const int first = last - __popc(may);
        M.place[lane] = make_uint2((unsigned)first, may);
        for (int base = 0; base < total;) {
            const unsigned fits = __ballot_sync(kFull, first >= base && last - base <= kPairs);
            const int stop = __shfl_sync(kFull, last, 31 - __clz(fits));
            __syncwarp();
            // every lane steps back over its pixel's pairs
            unsigned valid = 0, direct = 0;
            for (unsigned bits = todo & fits; bits; bits &= bits - 1) {
                const int k = __ffs(bits) - 1;
                const StagedRec<kBwdChunks> rec(M.rec, k);
                float opac, nbf, bf, e, eb;
                const int gid = M.q.gid[k];
                const Hit H = block_hit(a, ba, J.view, rec, gid, P, opac);
                const float alpha = block_alpha<FIX>(H, opac, use_blur, J.recs + gid, P, nbf, bf, e, eb);
                if (H.t < kTNear || H.t > kTFar || alpha < kAlphaMin) continue;
                float4 q0, q1;
                pair_adjoint<TM, CT, FIX>(S, a, g, rec, H, P, M.q.idx[k], opac, alpha, nbf, bf, e, eb, q0, q1);
                const uint2 pl = M.place[k];
                const int at = (int)pl.x - base + __popc(pl.y & below);
                M.pair[0][at] = q0;
                M.pair[1][at] = q1;
                valid |= 1u << k;
                if (CT == 3 && H.direct) direct |= 1u << k;
            }
            __syncwarp();
            // sum every splat's pairs over the pixels: one lane per splat, or
            // two or four where few splats have pairs (splats that cover the
            // block fill the room with few of them)
            unsigned mine = transpose32(valid, lane);
            const unsigned act = __ballot_sync(kFull, mine != 0u);
            const int na = __popc(act), shift = na <= 8 ? 2 : na <= 16 ? 1 : 0, sub = (int)lane & ((1 << shift) - 1);
            int k = (int)lane;
            if (shift) {
                if (mine) M.slot[__popc(act & below)] = (uint8_t)lane;
                __syncwarp();
                const int j = (int)lane >> shift;
                k = j < na ? M.slot[j] : 0;
                mine = __shfl_sync(kFull, mine, k);
                if (j >= na) mine = 0;
            }
            const unsigned own = mine & ((shift == 2 ? 0x11111111u : shift == 1 ? 0x55555555u : kFull) << sub);
            const uint2 pl = M.place[k];
            float m[FIX ? 21 : 23];
#pragma unroll
            for (int q = 0; q < (FIX ? 21 : 23); q++) m[q] = 0.f;
            const float4 nop = M.rec.c[k][kChunkNop - kChunkOrg];
            for (unsigned todo_p = own; todo_p; todo_p &= todo_p - 1) {
                const int p = __ffs(todo_p) - 1;
                const int at = (int)pl.x - base + __popc(pl.y & ((1u << p) - 1u));
                const float4 q0 = M.pair[0][at], q1 = M.pair[1][at];
                const float4 vo = M.pix[0][p];
                const float2 vn = M.pix_n[p];
                const float vis = q0.x, vtd = q0.w;
                const float vsig = FIX ? q0.y : q0.z;  // (FIX: v_sigma = -opacity times this, applied below)
                const float2 ls = make_float2(q1.z, q1.w);
                float2 t2 = fma2(dup2(vis), make_float2(vo.x, vo.y), make_float2(m[0], m[1]));
                m[0] = t2.x; m[1] = t2.y;
                m[2] += vis * vo.z;
                m[3] += q0.y;
                const float2 pk = mul2(ls, dup2(vsig));
                t2 = fma2(ls, pk, make_float2(m[4], m[5]));
                m[4] = t2.x; m[5] = t2.y;
                m[6] += ls.x * pk.y;
                t2 = add2(make_float2(m[7], m[8]), pk);
                m[7] = t2.x; m[8] = t2.y;
                m[9] += vtd;
                t2 = fma2(ls, dup2(vtd), make_float2(m[10], m[11]));
                m[10] = t2.x; m[11] = t2.y;
                m[12] += vis * vo.w;
                t2 = fma2(dup2(vis), vn, make_float2(m[13], m[14]));
                m[13] = t2.x; m[14] = t2.y;
                if (CT > 0) {
                    t2 = add2(make_float2(m[15], m[16]), make_float2(q1.x, q1.y));
                    m[15] = t2.x; m[16] = t2.y;
                    t2 = fma2(ls, dup2(q1.x), make_float2(m[17], m[18]));
                    m[17] = t2.x; m[18] = t2.y;
                    t2 = fma2(ls, dup2(q1.y), make_float2(m[19], m[20]));
                    m[19] = t2.x; m[20] = t2.y;
                }
                if constexpr (!FIX) {
                    // one of the two alphas is the pair's.  The filter's has no v_sigma, and the
                    // splat's no v_sigma_blur: as -opacity e v_alpha - v_sigma it would be the two
                    // products' rounding, which a large splat's small gradients do not bear
                    if (use_blur) {
                        const float4 c = __ldg(J.recs[M.q.gid[k]].c + kChunkMisc);
                        const float vsb = q0.z == 0.f ? -nop.z * q0.y : 0.f;
                        m[21] += kBlurFsq * vsb * (c.x - (fx0 + (float)lane_col(p)));
                        m[22] += kBlurFsq * vsb * (c.y - (fy0 + (float)lane_row(p)));
                    }
                }
            }
            __syncwarp();
            for (int o = 1; o < 1 << shift; o <<= 1) {
#pragma unroll
                for (int q = 0; q < (FIX ? 21 : 23); q++) m[q] += __shfl_xor_sync(kFull, m[q], o);
            }
            if (mine && sub == 0) {
                if (FIX) {
#pragma unroll
                    for (int q = 4; q < 9; q++) m[q] *= -nop.z;
                }
                flush_moments<FIX>(m, ba, g, J, M.q.gid[k], use_blur);
            }
            if (CT == 3) {
                unsigned coarse = is_coarse(nop) ? own : 0u;
                if (__any_sync(kFull, direct != 0u)) coarse &= ~__shfl_sync(kFull, transpose32(direct, lane), k);
                if (coarse) add_coarse_texel_grads<TM, FIX>(M, a, g.v_texgrad, k, coarse, pl.y, (int)pl.x - base, fx0, fy0);
            }
            __syncwarp();
            base = stop;
        }
        n = pop_queue(M.q, n, lane);
    }
}

// ---------------------------------------------------------------------------
// Launches
// ---------------------------------------------------------------------------
// The block kernels take tile widths that are multiples of 8 (8 or 16), no
// texture or three channels, and prebuilt records; the tile kernels of
// raster.cu take the rest, and the alpha-visualisation mode.
bool blocks_apply(int bw, int C, int settings, const RecAll* recs) {
    return gstex_block_kernels(bw, C, settings, recs != nullptr);
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

int launch_edit_blocks(const SceneArgs& a, const BlockArgs& ba, const EditIO& E, cudaStream_t stream) {
    const long long blocks = (long long)ba.total_tiles * ((ba.bw >> 3) * (ba.bw >> 2));
    const long long grid = (blocks + kBlockWarps - 1) / kBlockWarps;
    if (grid > 0x7fffffffLL) return GSTEX_ERR_UNSUPPORTED;
    auto k = (a.settings & (1 << 9)) ? edit_block_kernel<0> : edit_block_kernel<1>;
    k<<<(unsigned)grid, 32 * kBlockWarps, 0, stream>>>(a, ba, E);
    return check_launch("texture_edit");
}

int launch_bwd_blocks(const SceneArgs& a, const BlockArgs& ba, const BwdArgs& g, int texmode, cudaStream_t stream) {
    const long long blocks = (long long)ba.total_tiles * ((ba.bw >> 3) * (ba.bw >> 2));
    const long long grid = (blocks + kBlockWarps - 1) / kBlockWarps;
    if (grid > 0x7fffffffLL) return GSTEX_ERR_UNSUPPORTED;
    const bool fix = (a.settings & kFixedBwdMask) == kFixedBwdSettings;
    void (*k)(const SceneArgs, const BlockArgs, BwdArgs);
    if (a.C == 0) k = fix ? bwd_block_kernel<0, 0, 1> : bwd_block_kernel<0, 0, 0>;
    else if (texmode == 1) k = fix ? bwd_block_kernel<1, 3, 1> : bwd_block_kernel<1, 3, 0>;
    else k = fix ? bwd_block_kernel<0, 3, 1> : bwd_block_kernel<0, 3, 0>;
    const size_t smem = sizeof(BwdMem) * kBlockWarps;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) { set_cuda_error(e, "backward blocks"); return GSTEX_ERR_CUDA; }
    k<<<(unsigned)grid, 32 * kBlockWarps, smem, stream>>>(a, ba, g);
    return check_launch("backward blocks");
}

}  // namespace gstex

extern "C" int gstex_block_kernels(int bw, int C, int settings, int with_records) {
    return (bw & 7) == 0 && (C == 0 || C == 3) && with_records && !(settings & (1 << 16));
}
