// Tile binning: intersection emission, stable LSD radix sort, tile ranges.
#include <algorithm>

#include "common.cuh"
#include "project.cuh"

namespace gstex {

// ---------------------------------------------------------------------------
// Emission (reference csrc/forward.cu:13-71, helpers.cuh:37-111)
// ---------------------------------------------------------------------------
__global__ void emit_kernel(int n, int num_isect, const float2* __restrict__ centers,
                            const float2* __restrict__ extents, const float* __restrict__ depths,
                            const int32_t* __restrict__ cum, int tiles_x, int tiles_y, int bw, int wrapped,
                            int64_t* __restrict__ keys, int32_t* __restrict__ gids) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int lo = i == 0 ? 0 : max(cum[i - 1], 0);  // (sums of counts below 0 are, too)
    const int hi = min(cum[i], num_isect);
    int cur = lo;
    const float2 e = extents[i];
    if (!((double)e.x <= 1e-4 && (double)e.y <= 1e-4)) {
        const float2 c = centers[i];
        const float fbw = (float)bw;
        const float tcx = __fdiv_rn(c.x, fbw), tcy = __fdiv_rn(c.y, fbw);
        const float tex = __fdiv_rn(e.x, fbw), tey = __fdiv_rn(e.y, fbw);
        int x0 = __float2int_rz(__fsub_rn(tcx, tex));
        int x1 = __float2int_rz(__fadd_rn(__fadd_rn(tcx, tex), 1.0f));
        int y0 = __float2int_rz(__fsub_rn(tcy, tey));
        int y1 = __float2int_rz(__fadd_rn(__fadd_rn(tcy, tey), 1.0f));
        if (wrapped) {
            if (x0 <= 0) x0 -= 1;
            if (y0 <= 0) y0 -= 1;
        } else {
            x0 = min(max(0, x0), tiles_x);
            x1 = min(max(0, x1), tiles_x);
            y0 = min(max(0, y0), tiles_y);
            y1 = min(max(0, y1), tiles_y);
        }
        const int64_t depth_id = (int64_t)__float_as_int(depths[i]);  // sign-extended (forward.cu:47)
        for (int ty = y0; ty < y1 && cur < hi; ++ty) {
            for (int tx = x0; tx < x1 && cur < hi; ++tx) {
                int ti = ty, tj = tx;
                if (wrapped) {
                    ti %= tiles_y; if (ti < 0) ti += tiles_y;
                    tj %= tiles_x; if (tj < 0) tj += tiles_x;
                }
                const int64_t tile = (int64_t)(ti * tiles_x + tj);
                keys[cur] = (int64_t)(((uint64_t)tile << 32) | (uint64_t)depth_id);
                gids[cur] = i;
                ++cur;
            }
        }
    }
    // slots this Gaussian did not write keep the zero value of the reference's
    // torch::zeros buffers (bindings.cu:99-102)
    for (; cur < hi; ++cur) {
        keys[cur] = 0;
        gids[cur] = 0;
    }
}

// ---------------------------------------------------------------------------
// Tile ranges (reference csrc/forward.cu:76-98); tiles outside [0, num_tiles)
// are ignored.
// ---------------------------------------------------------------------------
constexpr int kEdgeItems = 4;

// Tile of a sorted key: bits [shift, ...) of a 64-bit (tile | depth) key or of
// a 32-bit (tile | filler bit) key.  ids: receives the bits id_mask of the keys.
template <typename K>
__global__ void bin_edges_kernel(int n, const int64_t* __restrict__ n_dev, const K* __restrict__ sorted, int shift,
                                 int num_tiles, int2* __restrict__ bins, int32_t* __restrict__ ids, uint32_t id_mask) {
    chain_wait();
    if (n_dev) {
        const int64_t m = *n_dev;
        n = (int)(m < (int64_t)n ? (m > 0 ? m : 0) : n);
    }
    // kEdgeItems consecutive items per thread, their keys loaded up front
    const long long i0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * kEdgeItems;
    if (i0 >= n) return;
    int tile[kEdgeItems + 1];
    tile[0] = i0 > 0 ? (int)(sorted[i0 - 1] >> shift) : -1;
    K key[kEdgeItems];
#pragma unroll
    for (int q = 0; q < kEdgeItems; q++) key[q] = i0 + q < n ? sorted[i0 + q] : K(0);
#pragma unroll
    for (int q = 0; q < kEdgeItems; q++) {
        tile[q + 1] = i0 + q < n ? (int)(key[q] >> shift) : -1;
        if (ids && i0 + q < n) ids[i0 + q] = (int32_t)((uint32_t)key[q] & id_mask);
    }
#pragma unroll
    for (int q = 0; q < kEdgeItems; q++) {
        if (i0 + q >= n) break;
        const int i = (int)i0 + q;
        const int prev = tile[q], cur = tile[q + 1];
        const bool ok = cur >= 0 && cur < num_tiles;
        if (i == 0 && ok) bins[cur].x = 0;
        if (i == n - 1 && ok) bins[cur].y = n;
        if (i > 0 && prev != cur) {
            if (prev >= 0 && prev < num_tiles) bins[prev].y = i;
            if (ok) bins[cur].x = i;
        }
    }
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (u64 or u32 key, u32 value), digits of at most 8
// bits, of equal width in all passes.
//
// Each pass: per-block digit histograms -> one exclusive scan in
// (digit, block) order -> stable scatter.  Blocks own contiguous chunks; a
// block ranks each 3072-item tile with ballots + per-warp counters, so the
// order of equal digits is the input order.
//
// What bounds the scatter: instruction issue (62% of cycles) and the runs of a
// digit in a tile, whose partial sectors cost writes: 14 bits as 7 + 7 and 20 as
// 7 + 7 + 6 beat 8 + 6 and 8 + 8 + 4 (158M items 2.56 -> 2.14 ms, 80M 2.13 ->
// 1.68 ms), tiles of 3072 beat 2048 by 3 to 8%.  Ranks by __match_any_sync with
// a counter read and written in every round kept the warps waiting on shared
// memory (14 of 25 stall cycles).  Altogether 158M items of 14 bits 2.71 -> 1.99
// ms, 80M of 20 bits 2.15 -> 1.57 ms, 16M of 32 bits 0.67 -> 0.56 ms.
// ---------------------------------------------------------------------------
constexpr int kRadix = 256;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 12;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortMaxBlocks = 1216;
static_assert(kSortThreads == kRadix, "a thread per digit");

struct SortPlan {
    int blocks, chunk;
};

static SortPlan sort_plan(int n) {
    SortPlan p;
    int tiles = ceil_div(n, kSortTile);
    int tiles_per_block = ceil_div(tiles, kSortMaxBlocks);
    p.chunk = tiles_per_block * kSortTile;
    p.blocks = ceil_div(n, p.chunk);
    if (p.blocks < 1) p.blocks = 1;
    return p;
}

// With n_dev set, the item count is read on the device (clamped to n) and the
// chunk of each block is derived from it, so the launch shape does not depend
// on the count.
__device__ __forceinline__ void resolve_count(const int64_t* n_dev, int& n, int& chunk) {
    if (n_dev) {
        const int64_t m = *n_dev;
        n = (int)(m < (int64_t)n ? (m > 0 ? m : 0) : n);
        chunk = ceil_div(ceil_div(n, kSortTile), (int)gridDim.x) * kSortTile;
        if (chunk < kSortTile) chunk = kSortTile;
    }
}

// Per-block digit counts: each warp loads its kSortItems keys per thread of a
// tile of items up front (so the loads overlap) and counts them in its own
// shared-memory histogram with plain atomics; the warps' histograms are summed
// at the end.  by_block: as [block][digit], followed by zeros for that many
// passes less one.
template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const K* __restrict__ keys, int n, int chunk,
                                                                  const int64_t* __restrict__ n_dev, int shift,
                                                                  uint32_t dmask, uint32_t* __restrict__ hist,
                                                                  int by_block = 0) {
    __shared__ uint32_t h[kSortWarps][kRadix];
    for (int i = threadIdx.x; i < kSortWarps * kRadix; i += blockDim.x) (&h[0][0])[i] = 0;
    chain_wait();
    resolve_count(n_dev, n, chunk);
    __syncthreads();
    // (positions are unsigned and items counted from the tile's first: those behind
    // the last item may pass 31 bits)
    const uint32_t start = blockIdx.x * (uint32_t)chunk;
    const uint32_t end = min(start + (uint32_t)chunk, (uint32_t)n);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    uint32_t* hw = h[warp];
    for (uint32_t tbase = start; tbase < end; tbase += kSortThreads * kSortItems) {
        K key[kSortItems];
        const int l0 = warp * (32 * kSortItems) + lane, left = (int)(end - tbase);
        const K* __restrict__ src = keys + tbase;
#pragma unroll
        for (int k = 0; k < kSortItems; k++) key[k] = l0 + k * 32 < left ? src[l0 + k * 32] : K(0);
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
            if (l0 + k * 32 < left) atomicAdd(&hw[(uint32_t)(key[k] >> shift) & dmask], 1u);
        }
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kRadix; d += blockDim.x) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) c += h[w][d];
        if (by_block) {
            for (int p = 0; p < by_block; p++) hist[((size_t)p * gridDim.x + blockIdx.x) * kRadix + d] = p ? 0u : c;
        } else {
            hist[(size_t)d * gridDim.x + blockIdx.x] = c;
        }
    }
}

// Block-wide exclusive scan of one value per thread (blockDim.x == kSortThreads);
// *total receives the sum.  Ends with a barrier.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* wsum, uint32_t* total) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = lane < (unsigned)kSortWarps ? wsum[lane] : 0u;
#pragma unroll
        for (int o = 1; o < kSortWarps; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= (unsigned)o) t += y;
        }
        if (lane < (unsigned)kSortWarps) wsum[lane] = t;
    }
    __syncthreads();
    const uint32_t before = (warp ? wsum[warp - 1] : 0u) + x - v;
    if (total) *total = wsum[kSortWarps - 1];
    __syncthreads();
    return before;
}

// Exclusive scan of each digit's row of per-block counts, one block per
// digit; the row total goes to totals[digit].
__global__ void __launch_bounds__(kSortThreads) radix_scan_rows_kernel(uint32_t* __restrict__ hist, int blocks,
                                                                       uint32_t* __restrict__ totals) {
    chain_wait();
    __shared__ uint32_t wsum[kSortWarps];
    uint32_t* row = hist + (size_t)blockIdx.x * blocks;
    uint32_t carry = 0;
    for (int base = 0; base < blocks; base += kSortThreads) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < blocks ? row[i] : 0u;
        uint32_t sum;
        const uint32_t before = block_exclusive_scan(v, wsum, &sum);
        if (i < blocks) row[i] = carry + before;
        carry += sum;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Of the lanes in `valid` (a ballot of the whole warp), those whose digit
// equals this lane's d.
template <int DB>
__device__ __forceinline__ uint32_t same_digit(uint32_t valid, uint32_t d) {
    uint32_t peers = valid;
#pragma unroll
    for (int b = 0; b < DB; b++) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// Exclusive scan of one value per thread of a scatter block.  Ends with a
// barrier.
__device__ __forceinline__ uint32_t scatter_scan(uint32_t v, uint32_t* wsum) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t before = x - v;
    for (unsigned w = 0; w < warp; w++) before += wsum[w];
    __syncthreads();
    return before;
}

// Stable scatter of one block's chunk, 3072 items at a time: items are ranked
// by digit (ballots + per-warp counters, so equal digits keep their input
// order), regrouped by digit in shared memory, and written out as runs of
// consecutive positions.  K: 64- or 32-bit keys.
//
// DIRECT: one tile per block and few blocks.  A pass is then bound by its
// launches, so there is only this one: `offsets` holds the counts [block][digit]
// themselves, every block sums them up for its own digits, and counts the next
// pass's digits (shift + dbits on, next_mask) of the places it writes to into
// `next`, which is zero before (null in the last pass).
//
// VALS: the keys carry values; else `vin` and `vout` are not touched.
template <typename K, int DB, bool DIRECT = false, bool VALS = true>
__global__ void __launch_bounds__(kSortThreads, 4) radix_scatter_kernel(
    const K* __restrict__ kin, const uint32_t* __restrict__ vin, K* __restrict__ kout,
    uint32_t* __restrict__ vout, int n, int chunk, const int64_t* __restrict__ n_dev, int shift, int dbits,
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ totals, uint32_t* __restrict__ next = nullptr,
    uint32_t next_mask = 0u) {
    chain_wait();
    __shared__ uint32_t run_off[kRadix];
    __shared__ uint32_t tile_base[kRadix];
    __shared__ uint32_t wsum[kSortWarps];
    __shared__ uint32_t wcnt[kSortWarps][kRadix];
    extern __shared__ __align__(16) unsigned char sort_smem[];
    K* skey = reinterpret_cast<K*>(sort_smem);
    uint32_t* sval = reinterpret_cast<uint32_t*>(skey + kSortTile);
    resolve_count(n_dev, n, chunk);
    const uint32_t dmask = (1u << dbits) - 1u;
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = tid & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    // digit d starts at (sum of the totals of smaller digits) + (this block's row prefix)
    if (DIRECT) {
        const int blocks = ceil_div(n, kSortTile);
        if ((int)blockIdx.x >= blocks) return;
        uint32_t before = 0, total = 0;
        for (int b0 = 0; b0 < blocks; b0 += 32) {
            uint32_t c[32];  // (all loads of a round first)
#pragma unroll
            for (int j = 0; j < 32; j++) c[j] = b0 + j < blocks ? offsets[(size_t)(b0 + j) * kRadix + tid] : 0u;
#pragma unroll
            for (int j = 0; j < 32; j++) {
                before += b0 + j < (int)blockIdx.x ? c[j] : 0u;
                total += c[j];
            }
        }
        run_off[tid] = scatter_scan(total, wsum) + before;
    }
    const uint32_t start = blockIdx.x * (uint32_t)chunk;
    const uint32_t end = min(start + (uint32_t)chunk, (uint32_t)n);
    if (!DIRECT) {
        // One digit that all items share leaves their order as it is (the upper bits of
        // tile and depth keys, and of any key that is sorted by more bits than it uses):
        // 50M such items are copied in 270 us a pass; ranking them takes 435.
        const uint32_t count = totals[tid];
        if (__syncthreads_or(count == (uint32_t)n)) {
            for (uint32_t tbase = start; tbase < end; tbase += kSortTile) {
                const int left = (int)(end - tbase);
#pragma unroll
                for (int k = 0; k < kSortItems; k++) {
                    const int l = k * kSortThreads + tid;
                    if (l < left) {
                        (kout + tbase)[l] = (kin + tbase)[l];
                        if (VALS) (vout + tbase)[l] = (vin + tbase)[l];
                    }
                }
            }
            return;
        }
        const uint32_t base = scatter_scan(count, wsum);
        run_off[tid] = base + offsets[(size_t)tid * gridDim.x + blockIdx.x];
    }
    for (uint32_t tbase = start; tbase < end; tbase += kSortTile) {
        for (int k = tid; k < kSortWarps * kRadix; k += blockDim.x) (&wcnt[0][0])[k] = 0;
        __syncthreads();
        K key[kSortItems];
        uint32_t val[kSortItems];
        uint32_t rank[kSortItems];
        const int l0 = warp * (32 * kSortItems) + (int)lane, left = (int)(end - tbase);
        const K* __restrict__ ksrc = kin + tbase;
        const uint32_t* __restrict__ vsrc = VALS ? vin + tbase : nullptr;
        // all loads first, so that they overlap
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
            const int l = l0 + k * 32;
            key[k] = l < left ? ksrc[l] : K(0);
            if (VALS) val[k] = l < left ? vsrc[l] : 0u;
        }
        // Each round's lowest lane of a digit adds its count to the warp's
        // counter; the additions of a warp are in order, so no round waits for
        // the one before.
        uint32_t old[kSortItems];
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
            const bool in = l0 + k * 32 < left;
            const uint32_t d = (uint32_t)(key[k] >> shift) & dmask;
            const uint32_t peers = same_digit<DB>(__ballot_sync(0xffffffffu, in), d);
            const uint32_t first = __ffs(peers) - 1;
            old[k] = 0;
            if (in && first == lane) old[k] = atomicAdd(&wcnt[warp][d], (uint32_t)__popc(peers));
            rank[k] = (first << 8) | (uint32_t)__popc(peers & lt_mask);
            __syncwarp();
        }
#pragma unroll
        for (int k = 0; k < kSortItems; k++)
            rank[k] = __shfl_sync(0xffffffffu, old[k], rank[k] >> 8) + (rank[k] & 255u);
        __syncthreads();
        // per-warp offsets within each digit, then the digit's start in the tile
        uint32_t tot = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) {
            const uint32_t c = wcnt[w][tid];
            wcnt[w][tid] = tot;
            tot += c;
        }
        const uint32_t tb = scatter_scan(tot, wsum);
        tile_base[tid] = tb;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
            if (l0 + k * 32 < left) {
                const uint32_t d = (uint32_t)(key[k] >> shift) & dmask;
                const uint32_t local = tile_base[d] + wcnt[warp][d] + rank[k];
                skey[local] = key[k];
                if (VALS) sval[local] = val[k];
            }
        }
        __syncthreads();
        const int tile_n = min(kSortTile, left);
        for (int l = tid; l < tile_n; l += kSortThreads) {
            const K kk = skey[l];
            const uint32_t d = (uint32_t)(kk >> shift) & dmask;
            const uint32_t pos = run_off[d] + (uint32_t)l - tile_base[d];
            kout[pos] = kk;
            if (VALS) vout[pos] = sval[l];
            if (DIRECT && next)
                atomicAdd(&next[(size_t)(pos / kSortTile) * kRadix + ((uint32_t)(kk >> (shift + dbits)) & next_mask)], 1u);
        }
        __syncthreads();
        // advance each digit's cursor by the tile's count of that digit
        {
            const uint32_t next = (tid + 1 < kRadix) ? tile_base[tid + 1] : (uint32_t)tile_n;
            run_off[tid] += next - tile_base[tid];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Depth-first binning of one view.  Ordering (tile, depth) keys of all
// intersections takes a 64-bit sort whose passes move every intersection's 12
// bytes five or six times; the depth order is the same in every tile, so the
// Gaussians are sorted by depth once, emit their tiles in that order, and a
// stable sort of 32-bit keys by tile alone (one to three passes of 8 bytes)
// finishes the order.  Keys are (tile << 1 | real); slots a Gaussian does not
// write (the reference's zero entries: tile 0, depth 0, Gaussian 0) have real
// bit 0 and come first in tile 0, and Gaussians of negative depth, whose keys
// the reference turns into tile -1, go to the tile behind the last.
//
// 158M intersections of 200k Gaussians (full HD): emission 3.1 -> 0.46 ms, sorts
// and scans 6.6 -> 1.7 ms; a few thousand: one launch each instead of 18 to 25.
// ---------------------------------------------------------------------------
__global__ void depth_keys_kernel(int n, const float* __restrict__ depths, const int32_t* __restrict__ counts,
                                  uint32_t* __restrict__ keys, int32_t* __restrict__ ids, int64_t* __restrict__ info) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = __float_as_uint(depths[i]);
    const int count = counts[i];
    keys[i] = count > 0 ? k : 0xffffffffu;
    ids[i] = i;
    // a depth of +0 ties with the zero entries, whose order is then their slots';
    // behind a count below 0 slots overlap
    if (count < 0 || (count > 0 && k == 0u)) info[1] = 1;
}

// Key and Gaussian of slot u of the Gaussian gi, whose tile rectangle is
// [x0, x0 + w) x [y0, y0 + h).
__device__ __forceinline__ void view_slot(int u, int x0, int y0, int w, int h, bool behind, int gi, int tiles_x,
                                          int num_tiles, uint32_t& key, int32_t& val) {
    key = 0u;
    val = 0;
    if (w > 0 && h > 0 && (long long)u < (long long)w * h) {
        const int q = (int)((unsigned)u / (unsigned)w);
        const int tile = behind ? num_tiles : (y0 + q) * tiles_x + x0 + (u - q * w);
        key = ((uint32_t)tile << 1) | 1u;
        val = gi;
    }
}

// Tile rectangle of Gaussian i (empty where it emits nothing).
__device__ __forceinline__ void view_rect(const float2* __restrict__ centers, const float2* __restrict__ extents, int i,
                                          int tiles_x, int tiles_y, int bw, int& x0, int& y0, int& w, int& h) {
    const float2 e = extents[i];
    x0 = y0 = w = h = 0;
    if (!((double)e.x <= 1e-4 && (double)e.y <= 1e-4)) {
        int x1, y1;
        tile_rect(centers[i], e, tiles_x, tiles_y, bw, x0, y0, x1, y1);
        w = x1 - x0;
        h = y1 - y0;
    }
}

// Emission in depth order.  A warp writes `slots` consecutive slots, however
// many Gaussians they belong to: it finds the first by a 32-way search of the
// slot offsets, then takes 32 Gaussians at a time, one per lane, and 32 slots
// at a time, each lane finding its slot's Gaussian among the 32.  At most 1024
// slots a warp spread a long emission evenly; short ones take fewer, so that
// there are warps for the whole chip (250k slots: 50 us with 1024, under 10 with 64).
constexpr int kEmitSlots = 1024;
constexpr int kEmitWarps = 152 * 32;

__global__ void __launch_bounds__(256) view_emit_kernel(int n, int num_isect, int slots, const float2* __restrict__ centers,
                                                        const float2* __restrict__ extents,
                                                        const float* __restrict__ depths,
                                                        const int32_t* __restrict__ order,
                                                        const int32_t* __restrict__ cum, int tiles_x, int tiles_y,
                                                        int bw, int id_bits, uint32_t* __restrict__ keys,
                                                        int32_t* __restrict__ vals) {
    chain_wait();
    const unsigned lane = threadIdx.x & 31;
    const long long first = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * slots;
    if (first >= num_isect) return;
    const int end = (int)min(first + slots, (long long)num_isect);
    int cur = (int)first;
    // p0: the first Gaussian in depth order whose slots end beyond `cur`
    int lo = 0, hi = n - 1;
    while (hi > lo) {
        const int step = (hi - lo + 31) / 32;
        const int probe = min(lo + ((int)lane + 1) * step - 1, hi);
        const unsigned beyond = __ballot_sync(0xffffffffu, cum[probe] > cur);
        if (!beyond) {  // (cum[n - 1] is the number of slots)
            lo = hi;
            break;
        }
        const int f = __ffs(beyond) - 1;
        hi = min(lo + (f + 1) * step - 1, hi);
        lo = min(lo + f * step, hi);
    }
    for (int p0 = lo; cur < end && p0 < n; p0 += 32) {
        const int p = p0 + (int)lane;
        const int phi = p < n ? cum[p] : num_isect;
        int plo = __shfl_up_sync(0xffffffffu, phi, 1);
        if (lane == 0) plo = p0 > 0 ? cum[p0 - 1] : 0;
        int x0 = 0, y0 = 0, w = 0, h = 0, gi = 0;
        bool behind = false;
        if (p < n && plo < phi && phi > cur && plo < end) {
            gi = order[p];
            view_rect(centers, extents, gi, tiles_x, tiles_y, bw, x0, y0, w, h);
            behind = (__float_as_uint(depths[gi]) >> 31) != 0u;
        }
        const int stop = min(end, __shfl_sync(0xffffffffu, phi, 31));
        // (warp-uniform trip count; unsigned, as the last step may pass 31 bits)
        for (unsigned base = cur; base < (unsigned)stop; base += 32) {
            const unsigned t = base + lane;
            int q = 0;  // the last lane whose first slot is <= t
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                const int l = __shfl_sync(0xffffffffu, plo, q + s);
                if ((unsigned)l <= t) q += s;
            }
            const int ql = __shfl_sync(0xffffffffu, plo, q), qx = __shfl_sync(0xffffffffu, x0, q);
            const int qy = __shfl_sync(0xffffffffu, y0, q), qw = __shfl_sync(0xffffffffu, w, q);
            const int qh = __shfl_sync(0xffffffffu, h, q), qg = __shfl_sync(0xffffffffu, gi, q);
            const bool qb = __shfl_sync(0xffffffffu, (int)behind, q) != 0;
            if (t < (unsigned)stop) {
                uint32_t key;
                int32_t val;
                view_slot((int)t - ql, qx, qy, qw, qh, qb, qg, tiles_x, tiles_x * tiles_y, key, val);
                keys[t] = vals ? key : key << id_bits | (uint32_t)val;
                if (vals) vals[t] = val;
            }
        }
        cur = max(cur, stop);
    }
}

// Small views (a few thousand Gaussians or intersections): the whole of a
// stage in one launch of one CTA, which sorts in shared memory.
constexpr int kSmallItems = 4096;
constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallPer = kSmallItems / kSmallThreads;

struct SmallSort {
    uint32_t key[2][kSmallItems];
    uint32_t val[2][kSmallItems];
    uint32_t cnt[kSmallWarps][kRadix];
    uint32_t base[kRadix];
    uint32_t wsum[kSmallWarps];
};

// Exclusive scan over the CTA of one value per thread; total in *sum.  Ends
// with a barrier.
__device__ __forceinline__ uint32_t small_scan(uint32_t v, uint32_t* wsum, uint32_t* sum) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= (unsigned)o) t += y;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    const uint32_t before = (warp ? wsum[warp - 1] : 0u) + x - v;
    *sum = wsum[kSmallWarps - 1];
    __syncthreads();
    return before;
}

// Stable LSD radix sort of the n pairs in key[0] / val[0] on bits [0,
// end_bit); returns the buffer that holds the result.  Each warp ranks a
// contiguous share, so equal digits keep their order.
__device__ __forceinline__ int small_sort(SmallSort& S, int n, int end_bit) {
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
    int src = 0;
    for (int shift = 0; shift < end_bit; shift += 8, src ^= 1) {
        for (int k = tid; k < kSmallWarps * kRadix; k += kSmallThreads) (&S.cnt[0][0])[k] = 0;
        __syncthreads();
        uint32_t rank[kSmallPer];
#pragma unroll
        for (int r = 0; r < kSmallPer; r++) {
            const int i = (int)(warp * (32 * kSmallPer) + r * 32 + lane);
            const bool valid = i < n;
            const unsigned mask = __ballot_sync(0xffffffffu, valid);
            uint32_t d = 0, before = 0, peers = 0;
            if (valid) {
                d = (S.key[src][i] >> shift) & (kRadix - 1);
                peers = __match_any_sync(mask, d);
                before = S.cnt[warp][d];
                rank[r] = before + __popc(peers & lt);
            }
            __syncwarp();
            if (valid && lane == (unsigned)(31 - __clz(peers))) S.cnt[warp][d] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        uint32_t tot = 0;
        if (tid < kRadix) {
#pragma unroll 8
            for (int w = 0; w < kSmallWarps; w++) {
                const uint32_t c = S.cnt[w][tid];
                S.cnt[w][tid] = tot;
                tot += c;
            }
        }
        uint32_t all;
        const uint32_t b = small_scan(tot, S.wsum, &all);
        if (tid < kRadix) S.base[tid] = b;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallPer; r++) {
            const int i = (int)(warp * (32 * kSmallPer) + r * 32 + lane);
            if (i < n) {
                const uint32_t key = S.key[src][i], d = (key >> shift) & (kRadix - 1);
                const uint32_t to = S.base[d] + S.cnt[warp][d] + rank[r];
                S.key[src ^ 1][to] = key;
                S.val[src ^ 1][to] = S.val[src][i];
            }
        }
        __syncthreads();
    }
    return src;
}

__global__ void __launch_bounds__(kSmallThreads) view_order_small_kernel(int n, const float* __restrict__ depths,
                                                                         const int32_t* __restrict__ counts,
                                                                         int32_t* __restrict__ order,
                                                                         int32_t* __restrict__ cum,
                                                                         int64_t* __restrict__ info) {
    extern __shared__ __align__(16) unsigned char smem[];
    SmallSort& S = *reinterpret_cast<SmallSort*>(smem);
    bool zero = false;
    for (int i = threadIdx.x; i < n; i += kSmallThreads) {
        const uint32_t k = __float_as_uint(depths[i]);
        const int count = counts[i];
        S.key[0][i] = count > 0 ? k : 0xffffffffu;
        S.val[0][i] = (uint32_t)i;
        zero = zero || count < 0 || (count > 0 && k == 0u);
    }
    const int any_zero = __syncthreads_or(zero);
    const int at = small_sort(S, n, 32);
    // inclusive sums of the counts in depth order, kSmallPer per thread; the
    // total in 64 bits, as the caller refuses one beyond 31
    int c[kSmallPer];
    long long sum = 0;
#pragma unroll
    for (int r = 0; r < kSmallPer; r++) {
        const int i = (int)threadIdx.x * kSmallPer + r;
        c[r] = i < n ? counts[S.val[at][i]] : 0;
        sum += c[r];
    }
    __syncthreads();
    long long* part = reinterpret_cast<long long*>(S.cnt);
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < kSmallThreads; o <<= 1) {
        const long long y = (int)threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += y;
        __syncthreads();
    }
    long long run = part[threadIdx.x] - sum;
#pragma unroll
    for (int r = 0; r < kSmallPer; r++) {
        const int i = (int)threadIdx.x * kSmallPer + r;
        run += c[r];
        if (i < n) {
            order[i] = (int32_t)S.val[at][i];
            cum[i] = (int32_t)run;
        }
    }
    if (threadIdx.x == 0) {
        info[0] = part[kSmallThreads - 1];
        info[1] = any_zero;
    }
}

__global__ void __launch_bounds__(kSmallThreads) view_bins_small_kernel(
    int n, int num_isect, const float2* __restrict__ centers, const float2* __restrict__ extents,
    const float* __restrict__ depths, const int32_t* __restrict__ order, const int32_t* __restrict__ cum, int tiles_x,
    int tiles_y, int bw, int end_bit, int32_t* __restrict__ gids, int2* __restrict__ bins) {
    extern __shared__ __align__(16) unsigned char smem[];
    SmallSort& S = *reinterpret_cast<SmallSort*>(smem);
    const int num_tiles = tiles_x * tiles_y;
    for (int i = threadIdx.x; i < num_tiles; i += kSmallThreads) bins[i] = make_int2(0, 0);
    for (int t = threadIdx.x; t < num_isect; t += kSmallThreads) {
        int lo = 0, hi = n - 1;  // the first Gaussian in depth order whose slots end beyond t
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (cum[mid] > t) hi = mid; else lo = mid + 1;
        }
        const int gi = order[lo];
        int x0, y0, w, h;
        view_rect(centers, extents, gi, tiles_x, tiles_y, bw, x0, y0, w, h);
        uint32_t key;
        int32_t val;
        view_slot(t - (lo > 0 ? cum[lo - 1] : 0), x0, y0, w, h, (__float_as_uint(depths[gi]) >> 31) != 0u, gi, tiles_x,
                  num_tiles, key, val);
        S.key[0][t] = key;
        S.val[0][t] = (uint32_t)val;
    }
    __syncthreads();
    const int at = small_sort(S, num_isect, end_bit);
    for (int t = threadIdx.x; t < num_isect; t += kSmallThreads) {
        gids[t] = (int32_t)S.val[at][t];
        const int tile = (int)(S.key[at][t] >> 1);
        if (tile >= num_tiles) continue;
        if (t == 0 || (int)(S.key[at][t - 1] >> 1) != tile) bins[tile].x = t;
        if (t == num_isect - 1 || (int)(S.key[at][t + 1] >> 1) != tile) bins[tile].y = t + 1;
    }
}

// The forward's queue order (tile_group_keys_kernel) of up to kSmallItems
// groups of tiles in one launch.  groups[i]: first tile, tiles per row of its
// view, width and height in tiles, in tile order.  (Sorting the tiles takes two
// sorts, six passes or more of three launches: 96 us for 3 to 18 thousand
// tiles, 17 to 20 here.)
__global__ void __launch_bounds__(kSmallThreads) tile_order_small_kernel(int n, const int4* __restrict__ groups,
                                                                         const int2* __restrict__ bins,
                                                                         int32_t* __restrict__ order) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    SmallSort& S = *reinterpret_cast<SmallSort*>(smem);
    for (int i = threadIdx.x; i < n; i += kSmallThreads) {
        const int4 g = groups[i];
        uint32_t cost = 0;
        for (int y = 0; y < g.w; y++)
            for (int x = 0; x < g.z; x++) {
                const int2 b = bins[g.x + y * g.y + x];
                cost += (uint32_t)max(b.y - b.x, 0);
            }
        S.key[0][i] = ~cost;
        S.val[0][i] = (uint32_t)i;
    }
    __syncthreads();
    const int at = small_sort(S, n, 32);
    // positions of the groups' tiles: exclusive sums of their sizes in order
    int4 g[kSmallPer];
    uint32_t sum = 0, all;
#pragma unroll
    for (int r = 0; r < kSmallPer; r++) {
        const int i = (int)threadIdx.x * kSmallPer + r;
        g[r] = i < n ? groups[S.val[at][i]] : make_int4(0, 0, 0, 0);
        sum += (uint32_t)(g[r].z * g[r].w);
    }
    uint32_t to = small_scan(sum, S.wsum, &all);
#pragma unroll
    for (int r = 0; r < kSmallPer; r++)
        for (int y = 0; y < g[r].w; y++)
            for (int x = 0; x < g[r].z; x++) order[to++] = g[r].x + y * g[r].y + x;
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace gstex

using namespace gstex;

extern "C" int gstex_map_gaussian_to_intersects(int n, int num_isect, const float* centers, const float* extents,
                                                const float* depths, const int32_t* cum, int tiles_x, int tiles_y,
                                                int bw, int wrapped, int64_t* keys, int32_t* gids,
                                                gstex_stream_t stream) {
    GSTEX_REQUIRE(n >= 0 && num_isect >= 0 && tiles_x > 0 && tiles_y > 0 && bw > 0);
    if (n == 0 || num_isect == 0) return GSTEX_OK;
    GSTEX_REQUIRE(centers && extents && depths && cum && keys && gids);
    emit_kernel<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(n, num_isect, (const float2*)centers,
                                                                     (const float2*)extents, depths, cum, tiles_x,
                                                                     tiles_y, bw, wrapped, keys, gids);
    return check_launch("map_gaussian_to_intersects");
}

// 32-bit sorts of at most one tile per multiprocessor take one launch a pass
// (DIRECT) instead of three.  Every block reads the counts of all blocks, so the
// gain shrinks with their number: 32 bits of 100k items 64 -> 32 us, 240k 65 ->
// 37, 390k (127 tiles) 66 -> 42, but 500k (163) 49 -> 57.
constexpr int kDirectBlocks = 152;

static bool sort_direct(const SortPlan& p, size_t key_bytes) {
    return key_bytes == 4 && p.chunk == kSortTile && p.blocks <= kDirectBlocks;
}

// Never less than for a smaller n, so that one workspace serves all counts up to
// its own: of the rows of block counts it has what the largest launch up to n
// takes (four of each block with one launch a pass, else one).
static size_t sort_workspace_bytes(int n, size_t key_bytes) {
    if (n < 1) n = 1;
    const int tiles = ceil_div(n, kSortTile);
    const size_t rows = std::max(std::min(tiles, kSortMaxBlocks), key_bytes == 4 ? 4 * std::min(tiles, kDirectBlocks) : 0);
    return align_up((size_t)n * key_bytes, 256) + align_up((size_t)n * 4, 256) + rows * kRadix * 4 + (size_t)kRadix * 4;
}

extern "C" size_t gstex_sort_workspace_bytes(int n) { return sort_workspace_bytes(n, 8); }
extern "C" size_t gstex_sort32_workspace_bytes(int n) { return sort_workspace_bytes(n, 4); }

// By the end_bit bits from first_bit on; without VALS there are keys alone.
template <typename K, bool VALS = true>
static int sort_impl(int n, const int64_t* n_dev, int end_bit, const K* keys_in, const int32_t* vals_in,
                     K* keys_out, int32_t* vals_out, void* ws, size_t ws_bytes, cudaStream_t stream, int first_bit = 0) {
    GSTEX_REQUIRE(n >= 0 && end_bit >= 0 && first_bit + end_bit <= (int)(8 * sizeof(K)));
    if (n == 0) return GSTEX_OK;
    GSTEX_REQUIRE(keys_in && keys_out && (!VALS || (vals_in && vals_out)));
    const int passes = ceil_div(end_bit, 8);
    if (passes == 0 || (n == 1 && !n_dev)) {
        cudaError_t e = cudaMemcpyAsync(keys_out, keys_in, (size_t)n * sizeof(K), cudaMemcpyDeviceToDevice, stream);
        if (VALS && e == cudaSuccess)
            e = cudaMemcpyAsync(vals_out, vals_in, (size_t)n * 4, cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) { set_cuda_error(e, "sort_pairs copy"); return GSTEX_ERR_CUDA; }
        return GSTEX_OK;
    }
    GSTEX_REQUIRE(ws);
    if (ws_bytes < sort_workspace_bytes(n, sizeof(K))) return GSTEX_ERR_CAPACITY;
    const SortPlan p = sort_plan(n);
    char* w = (char*)ws;
    K* kalt = (K*)w;
    w += align_up((size_t)n * sizeof(K), 256);
    uint32_t* valt = (uint32_t*)w;
    w += align_up((size_t)n * 4, 256);
    uint32_t* hist = (uint32_t*)w;
    uint32_t* totals = hist + (size_t)kRadix * p.blocks;
    const int digit = ceil_div(end_bit, passes);
    // Ping-pong so that the last pass lands in the output buffers.
    const K* ksrc = keys_in;
    const uint32_t* vsrc = (const uint32_t*)vals_in;
    const bool direct = sort_direct(p, sizeof(K));
    const size_t row = (size_t)kRadix * p.blocks;  // counts of one pass
    if (direct) {
        launch_chained(radix_hist_kernel<K>, p.blocks, kSortThreads, 0, stream, ksrc, n, p.chunk, n_dev, first_bit,
                       (1u << std::min(digit, end_bit)) - 1u, hist, passes);
    }
    for (int pass = 0; pass < passes; pass++) {
        const bool to_out = ((passes - 1 - pass) % 2) == 0;
        K* kdst = to_out ? keys_out : kalt;
        uint32_t* vdst = to_out ? (uint32_t*)vals_out : valt;
        const int done = pass * digit, dbits = std::min(digit, end_bit - done), shift = first_bit + done;
        const size_t smem = (size_t)kSortTile * (sizeof(K) + (VALS ? 4 : 0));
        if (direct) {
            if constexpr (sizeof(K) == 4) {
                const int left = end_bit - done - dbits;
                const uint32_t next_mask = left > 0 ? (1u << std::min(digit, left)) - 1u : 0u;
                auto scatter = dbits <= 5 ? radix_scatter_kernel<K, 5, true, VALS> : dbits == 6 ? radix_scatter_kernel<K, 6, true, VALS>
                             : dbits == 7 ? radix_scatter_kernel<K, 7, true, VALS> : radix_scatter_kernel<K, 8, true, VALS>;
                cudaError_t e = cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                if (e != cudaSuccess) { set_cuda_error(e, "sort_pairs"); return GSTEX_ERR_CUDA; }
                launch_chained(scatter, p.blocks, kSortThreads, smem, stream, ksrc, vsrc, kdst, vdst, n, p.chunk,
                               n_dev, shift, dbits, hist + pass * row, nullptr,
                               left > 0 ? hist + (pass + 1) * row : nullptr, next_mask);
            }
            ksrc = kdst;
            vsrc = vdst;
            continue;
        }
        launch_chained(radix_hist_kernel<K>, p.blocks, kSortThreads, 0, stream, ksrc, n, p.chunk, n_dev, shift,
                       (1u << dbits) - 1u, hist, 0);
        launch_chained(radix_scan_rows_kernel, kRadix, kSortThreads, 0, stream, hist, p.blocks, totals);
        auto scatter = dbits <= 5 ? radix_scatter_kernel<K, 5, false, VALS> : dbits == 6 ? radix_scatter_kernel<K, 6, false, VALS>
                     : dbits == 7 ? radix_scatter_kernel<K, 7, false, VALS> : radix_scatter_kernel<K, 8, false, VALS>;
        cudaError_t e = cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { set_cuda_error(e, "sort_pairs"); return GSTEX_ERR_CUDA; }
        launch_chained(scatter, p.blocks, kSortThreads, smem, stream, ksrc, vsrc, kdst, vdst, n, p.chunk, n_dev, shift,
                       dbits, hist, totals, nullptr, 0u);
        ksrc = kdst;
        vsrc = vdst;
    }
    return check_launch("sort_pairs", direct ? 1 + passes : 3 * passes);
}

extern "C" int gstex_sort_pairs(int n, int end_bit, const int64_t* keys_in, const int32_t* vals_in,
                                int64_t* keys_out, int32_t* vals_out, void* ws, size_t ws_bytes, gstex_stream_t s) {
    return sort_impl<uint64_t>(n, nullptr, end_bit, (const uint64_t*)keys_in, vals_in, (uint64_t*)keys_out, vals_out,
                               ws, ws_bytes, (cudaStream_t)s);
}

extern "C" int gstex_sort_pairs_dyn(int capacity, const int64_t* count, int end_bit, const int64_t* keys_in,
                                    const int32_t* vals_in, int64_t* keys_out, int32_t* vals_out, void* ws,
                                    size_t ws_bytes, gstex_stream_t s) {
    GSTEX_REQUIRE(count);
    return sort_impl<uint64_t>(capacity, count, end_bit, (const uint64_t*)keys_in, vals_in, (uint64_t*)keys_out,
                               vals_out, ws, ws_bytes, (cudaStream_t)s);
}

extern "C" int gstex_sort_pairs32(int n, const int64_t* count, int end_bit, const uint32_t* keys_in,
                                  const int32_t* vals_in, uint32_t* keys_out, int32_t* vals_out, void* ws,
                                  size_t ws_bytes, gstex_stream_t s) {
    return sort_impl<uint32_t>(n, count, end_bit, keys_in, vals_in, keys_out, vals_out, ws, ws_bytes,
                               (cudaStream_t)s);
}

extern "C" int gstex_get_tile_bin_edges(int num_isect, const int64_t* sorted, int num_tiles, int32_t* bins,
                                        gstex_stream_t s) {
    GSTEX_REQUIRE(num_isect >= 0 && num_tiles > 0 && bins);
    cudaStream_t stream = (cudaStream_t)s;
    cudaError_t e = cudaMemsetAsync(bins, 0, (size_t)num_tiles * 2 * sizeof(int32_t), stream);
    if (e != cudaSuccess) { set_cuda_error(e, "tile_bin_edges memset"); return GSTEX_ERR_CUDA; }
    if (num_isect == 0) return GSTEX_OK;
    GSTEX_REQUIRE(sorted);
    launch_chained(bin_edges_kernel<int64_t>, ceil_div(num_isect, 256 * kEdgeItems), 256, 0, stream, num_isect,
                   nullptr, sorted, 32, num_tiles, (int2*)bins, nullptr, 0u);
    return check_launch("get_tile_bin_edges");
}

extern "C" int gstex_get_tile_bin_edges_dyn(int capacity, const int64_t* count, const int64_t* sorted, int num_tiles,
                                            int32_t* bins, gstex_stream_t s) {
    GSTEX_REQUIRE(capacity >= 0 && num_tiles > 0 && bins && count);
    cudaStream_t stream = (cudaStream_t)s;
    cudaError_t e = cudaMemsetAsync(bins, 0, (size_t)num_tiles * 2 * sizeof(int32_t), stream);
    if (e != cudaSuccess) { set_cuda_error(e, "tile_bin_edges memset"); return GSTEX_ERR_CUDA; }
    if (capacity == 0) return GSTEX_OK;
    GSTEX_REQUIRE(sorted);
    launch_chained(bin_edges_kernel<int64_t>, ceil_div(capacity, 256 * kEdgeItems), 256, 0, stream, capacity, count,
                   sorted, 32, num_tiles, (int2*)bins, nullptr, 0u);
    return check_launch("get_tile_bin_edges_dyn");
}

extern "C" int gstex_get_tile_bin_edges32_dyn(int capacity, const int64_t* count, const uint32_t* sorted, int shift,
                                              int num_tiles, int32_t* bins, gstex_stream_t s) {
    GSTEX_REQUIRE(capacity >= 0 && num_tiles > 0 && bins && count && shift >= 0 && shift < 32);
    cudaStream_t stream = (cudaStream_t)s;
    cudaError_t e = cudaMemsetAsync(bins, 0, (size_t)num_tiles * 2 * sizeof(int32_t), stream);
    if (e != cudaSuccess) { set_cuda_error(e, "tile_bin_edges32 memset"); return GSTEX_ERR_CUDA; }
    if (capacity == 0) return GSTEX_OK;
    GSTEX_REQUIRE(sorted);
    launch_chained(bin_edges_kernel<uint32_t>, ceil_div(capacity, 256 * kEdgeItems), 256, 0, stream, capacity, count,
                   sorted, shift, num_tiles, (int2*)bins, nullptr, 0u);
    return check_launch("get_tile_bin_edges32_dyn");
}

// Workspace of gstex_view_order: depth keys, ids, sorted keys, counts in depth
// order, then the sort's and the scan's.
extern "C" size_t gstex_view_order_workspace_bytes(int n) {
    if (n <= kSmallItems) return 256;
    return 4 * align_up((size_t)n * 4, 256) + align_up(sort_workspace_bytes(n, 4), 256) + gstex_scan_workspace_bytes(n);
}

extern "C" int gstex_view_order(int n, const float* depths, const int32_t* counts, int32_t* order, int32_t* cum,
                                int64_t* info, void* ws, size_t ws_bytes, gstex_stream_t s) {
    GSTEX_REQUIRE(n >= 0 && info);
    cudaStream_t stream = (cudaStream_t)s;
    if (n == 0 || n > kSmallItems) {
        cudaError_t e = cudaMemsetAsync(info, 0, 2 * sizeof(int64_t), stream);
        if (e != cudaSuccess) { set_cuda_error(e, "view_order"); return GSTEX_ERR_CUDA; }
        if (n == 0) return GSTEX_OK;
    }
    GSTEX_REQUIRE(depths && counts && order && cum && ws && ((uintptr_t)ws & 15) == 0);
    if (ws_bytes < gstex_view_order_workspace_bytes(n)) return GSTEX_ERR_CAPACITY;
    if (n <= kSmallItems) {
        cudaError_t e = cudaFuncSetAttribute(view_order_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(SmallSort));
        if (e != cudaSuccess) { set_cuda_error(e, "view_order"); return GSTEX_ERR_CUDA; }
        view_order_small_kernel<<<1, kSmallThreads, sizeof(SmallSort), stream>>>(n, depths, counts, order, cum, info);
        return check_launch("view_order");
    }
    char* w = (char*)ws;
    const size_t a = align_up((size_t)n * 4, 256), sb = align_up(sort_workspace_bytes(n, 4), 256);
    uint32_t* keys = (uint32_t*)w;
    int32_t* ids = (int32_t*)(w + a);
    uint32_t* sorted = (uint32_t*)(w + 2 * a);
    int32_t* scounts = (int32_t*)(w + 3 * a);
    launch_chained(depth_keys_kernel, ceil_div(n, 256), 256, 0, stream, n, depths, counts, keys, ids, info);
    int rc = check_launch("view_order");
    if (rc) return rc;
    rc = gstex_sort_pairs32(n, nullptr, 32, keys, ids, sorted, order, w + 4 * a, sb, s);
    if (rc) return rc;
    return gstex_inclusive_scan_picked_i32(n, counts, order, scounts, cum, info, w + 4 * a + sb,
                                           gstex_scan_workspace_bytes(n), s);
}

extern "C" size_t gstex_view_bins_workspace_bytes(int num_isect) {
    if (num_isect <= kSmallItems) return 256;
    return 3 * align_up((size_t)num_isect * 4, 256) + sort_workspace_bytes(num_isect, 4);
}

extern "C" int gstex_view_bins(int n, int num_isect, const float* centers, const float* extents, const float* depths,
                               const int32_t* order, const int32_t* cum, int tiles_x, int tiles_y, int bw, int32_t* gids,
                               int32_t* bins, void* ws, size_t ws_bytes, gstex_stream_t s) {
    GSTEX_REQUIRE(n >= 0 && num_isect >= 0 && tiles_x > 0 && tiles_y > 0 && bw > 0 && bins);
    if ((long long)tiles_x * tiles_y >= (1ll << 30)) return GSTEX_ERR_UNSUPPORTED;
    const int num_tiles = tiles_x * tiles_y;
    cudaStream_t stream = (cudaStream_t)s;
    if (n == 0 || num_isect == 0) {
        cudaError_t e = cudaMemsetAsync(bins, 0, (size_t)num_tiles * 2 * sizeof(int32_t), stream);
        if (e != cudaSuccess) { set_cuda_error(e, "view_bins"); return GSTEX_ERR_CUDA; }
        return GSTEX_OK;
    }
    GSTEX_REQUIRE(centers && extents && depths && order && cum && gids && ws && ((uintptr_t)ws & 15) == 0);
    if (ws_bytes < gstex_view_bins_workspace_bytes(num_isect)) return GSTEX_ERR_CAPACITY;
    int end_bit = 1;  // keys reach num_tiles << 1 | 1
    while ((num_tiles >> (end_bit - 1)) != 0) end_bit++;
    if (num_isect <= kSmallItems) {
        cudaError_t e = cudaFuncSetAttribute(view_bins_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(SmallSort));
        if (e != cudaSuccess) { set_cuda_error(e, "view_bins"); return GSTEX_ERR_CUDA; }
        view_bins_small_kernel<<<1, kSmallThreads, sizeof(SmallSort), stream>>>(
            n, num_isect, (const float2*)centers, (const float2*)extents, depths, order, cum, tiles_x, tiles_y, bw,
            end_bit, gids, (int2*)bins);
        return check_launch("view_bins");
    }
    cudaError_t e = cudaMemsetAsync(bins, 0, (size_t)num_tiles * 2 * sizeof(int32_t), stream);
    if (e != cudaSuccess) { set_cuda_error(e, "view_bins"); return GSTEX_ERR_CUDA; }
    // Where the key (tile << 1 | real) and the id fit one word, the words are
    // sorted alone and the ids taken out with the tile ranges: 4 bytes an item
    // less to write, read and regroup in each pass (158M items, two passes 1.75
    // -> 1.45 ms; the full-HD view 11.9 -> 11.7 ms).
    int id_bits = 0;
    while (n - 1 > 0 && ((n - 1) >> id_bits) != 0) id_bits++;
    const bool packed = id_bits + end_bit <= 32;
    if (!packed) id_bits = 0;
    char* w = (char*)ws;
    const size_t a = align_up((size_t)num_isect * 4, 256);
    uint32_t* keys = (uint32_t*)w;
    int32_t* vals = packed ? nullptr : (int32_t*)(w + a);
    uint32_t* sorted = (uint32_t*)(w + 2 * a);
    const int slots = num_isect >= kEmitSlots * kEmitWarps ? kEmitSlots : (num_isect / kEmitWarps / 32 + 1) * 32;
    const int warps = (int)(((long long)num_isect + slots - 1) / slots);
    launch_chained(view_emit_kernel, ceil_div(warps, 8), 256, 0, stream, n, num_isect, slots, (const float2*)centers,
                   (const float2*)extents, depths, order, cum, tiles_x, tiles_y, bw, id_bits, keys, vals);
    int rc = check_launch("view_bins");
    if (rc) return rc;
    const size_t sort_bytes = sort_workspace_bytes(num_isect, 4);
    rc = packed ? sort_impl<uint32_t, false>(num_isect, nullptr, end_bit, keys, nullptr, sorted, nullptr, w + 3 * a,
                                             sort_bytes, stream, id_bits)
                : sort_impl<uint32_t>(num_isect, nullptr, end_bit, keys, vals, sorted, gids, w + 3 * a, sort_bytes, stream);
    if (rc) return rc;
    launch_chained(bin_edges_kernel<uint32_t>, ceil_div(num_isect, 256 * kEdgeItems), 256, 0, stream, num_isect,
                   nullptr, sorted, id_bits + 1, num_tiles, (int2*)bins, packed ? gids : nullptr,
                   (1u << id_bits) - 1u);
    return check_launch("view_bins");
}

extern "C" int gstex_batch_tile_order_small(int num_groups, const int32_t* groups, const int32_t* tile_bins,
                                            int32_t* order, gstex_stream_t s) {
    GSTEX_REQUIRE(num_groups >= 0);
    if (num_groups == 0) return GSTEX_OK;
    GSTEX_REQUIRE(groups && ((uintptr_t)groups & 15) == 0 && tile_bins && order);
    if (num_groups > kSmallItems) return GSTEX_ERR_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(tile_order_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(SmallSort));
    if (e != cudaSuccess) { set_cuda_error(e, "batch_tile_order"); return GSTEX_ERR_CUDA; }
    launch_chained(tile_order_small_kernel, 1, kSmallThreads, sizeof(SmallSort), (cudaStream_t)s, num_groups,
                   (const int4*)groups, (const int2*)tile_bins, order);
    return check_launch("batch_tile_order");
}
