// Binning: depth ordering, duplicateWithKeys, onesweep radix sort by tile,
// tile ranges (antialias/cuda_rasterizer/rasterizer_impl.cu:113-194,363-445).
//
// The reference stably sorts 64-bit (tile << 32 | depth bits) keys of all K
// pairs with a 6-pass LSD radix sort.  An LSD sort's first four passes only
// look at the depth bits, and every pair of a Gaussian carries the same
// depth, so the same permutation is obtained by (1) stably sorting the P
// Gaussians by depth bits, (2) emitting each Gaussian's pairs in that order
// (rect y-major, x-minor, as the reference does), and (3) stably sorting the
// pairs by tile id only.  The result -- sorted order, keys, ranges -- is
// identical, and the K-sized passes drop from 6 to ceil(tile_bits / 8).
//
// Every sort pass is one onesweep kernel (Adinets & Merrill 2022): chunks
// take ascending indices from an atomic counter, rank their keys with
// warp-level ballots, and learn their global offsets per digit from a
// decoupled look-back over the preceding chunks (fgs_scan.cuh: windowed,
// bounded; on timeout the kernel records FGS_ERR_TIMEOUT and moves on).
#include "fgs_common.cuh"
#include "fgs_internal.h"
#include "fgs_scan.cuh"

namespace fgs {

namespace {

constexpr int kSortTileMin = 2048;  // smallest chunk (sizes the status words)
constexpr int kSortItems = 16;      // keys per thread, at most
constexpr int kRadix = 256;

// Exclusive scan of one value per thread over the first 256 threads of a block (all
// threads call it; s_warp: 8 words).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31 && warp < 8) s_warp[warp] = x;
    __syncthreads();
    uint32_t wpre = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const uint32_t c = s_warp[w];
        if (w < warp) wpre += c;
        tot += c;
    }
    __syncthreads();
    if (total) *total = tot;
    return wpre + x - v;
}

template <int kThreads>
struct SortSmem {
    uint16_t hist[kThreads / 32][kRadix];  // per warp; a chunk holds at most 16384 keys
    uint32_t keys[kThreads * kSortItems];
    uint32_t vals[kThreads * kSortItems];
    uint32_t start[kRadix];
    uint32_t gbase[kRadix];
    uint32_t warp[8];
    uint32_t chunk;
};

// One onesweep pass over `n` 32-bit keys with 32-bit values.
//   vals_in == nullptr: values are the element indices.
//   n_dev != nullptr: the live count is min(n, *n_dev) (the grid covers n).
// Persistent: each CTA takes chunks from the counter until none is left, so a
// grid sized for a bound costs nothing for the chunks that are not live.  Per
// chunk: rank the keys (a ballot per digit bit), publish the digit counts at once, sort the
// chunk locally in shared memory (which needs no global offsets), and only
// then walk back for the global offsets -- the registers that held the keys
// are free by then, so the walk keeps 32 status loads in flight per digit.
//
// With all chunks of a pass resident at once a walk sums half of the chunks before it,
// some six instructions each on every digit's thread: in blocks of 256 threads that
// was more than half of all instructions of the tile passes (570 chunks, 211 thread
// instructions per pair), so their blocks have 1024 threads and chunks of up to 16384
// pairs (128 chunks).  The depth sort, which runs over the ~120K visible Gaussians of a
// view and beside seven other views in a batch, takes 512: at least 2048 keys per chunk
// are then four per thread instead of eight, a shorter chain of ranks.
// A 1080p view of 2M Gaussians with 2.1M pairs: the four depth passes 84 -> 70 us, the two
// tile passes 126 -> 110 (62 without the records, which place_kernel writes); a 256x256 view
// of 10K Gaussians, all six passes: 59 -> 51 us.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads)
    onesweep_kernel(const uint32_t* __restrict__ keys_in, uint32_t* __restrict__ keys_out,
                    const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ vals_out, uint32_t n, int shift,
                    int nbits, const uint32_t* __restrict__ pass_hist, uint32_t* status, uint32_t* chunk_counter,
                    unsigned* err, const unsigned long long* __restrict__ n_dev,
                    unsigned long long wait_ns = kWaitLimitNs, uint32_t skip_chunk = 0xffffffffu)
{
    constexpr int kWarps = kThreads / 32, kItemsMin = kSortTileMin / kThreads;
    extern __shared__ __align__(16) unsigned char sort_dyn[];
    SortSmem<kThreads>& sm = *reinterpret_cast<SortSmem<kThreads>*>(sort_dyn);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (n_dev) n = (uint32_t)min((unsigned long long)n, *n_dev);
    // Keys per thread from the live count: about one chunk per resident CTA, between
    // kItemsMin and kSortItems (a small sort gets more, shorter chunks; a large one
    // fewer chunks and a shorter look-back chain).  The same on every CTA.
    const uint32_t per_cta = (n + gridDim.x - 1) / gridDim.x;
    const int items = (int)min((uint32_t)kSortItems,
                               max((uint32_t)kItemsMin, (per_cta + kThreads - 1) / kThreads));
    const uint32_t tile = (uint32_t)items * kThreads;
    const uint32_t live = (n + tile - 1) / tile;
    if (blockIdx.x >= live) return;
    const uint32_t dmask = (1u << nbits) - 1u;
    // global start of every digit in this pass (the same for all chunks)
    const uint32_t gh = (uint32_t)tid <= dmask ? __ldg(pass_hist + tid) : 0u;
    const uint32_t gofs = block_excl_scan(gh, sm.warp, nullptr);
    const unsigned lt = (1u << lane) - 1u;

    for (;;) {
        if (tid == 0) sm.chunk = atomicAdd(chunk_counter, 1u);
        for (int i = tid; i < kWarps * kRadix / 2; i += kThreads) reinterpret_cast<uint32_t*>(sm.hist)[i] = 0;
        __syncthreads();
        const uint32_t chunk = sm.chunk;
        if (chunk >= live) break;
        const uint32_t base = chunk * tile;
        const uint32_t count = min(tile, n - base);

        uint32_t key[kSortItems], rank[kSortItems];
#pragma unroll
        for (int i = 0; i < kSortItems; i++) {
            if (i >= items) break;
            const uint32_t pos = warp * (items * 32) + i * 32 + lane;
            key[i] = pos < count ? __ldg(keys_in + base + pos) : 0xffffffffu;
        }
#pragma unroll
        for (int i = 0; i < kSortItems; i++) {
            if (i >= items) break;
            const uint32_t pos = warp * (items * 32) + i * 32 + lane;
            const bool valid = pos < count;
            const uint32_t dg = (key[i] >> shift) & dmask;
            // lanes with this lane's digit: one vote per digit bit (a match instruction takes longer)
            unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                if (b >= nbits) break;
                const bool one = (dg >> b) & 1u;
                const unsigned m = __ballot_sync(0xffffffffu, one);
                peers &= one ? m : ~m;
            }
            // every lane of a digit reads its count before the last of them adds to it
            uint32_t old = 0;
            if (valid) old = sm.hist[warp][dg];
            __syncwarp();
            if (valid && (peers >> lane) == 1u) sm.hist[warp][dg] = (uint16_t)(old + __popc(peers));
            rank[i] = old + __popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        // per digit (thread d): exclusive prefix over warps, chunk total, published at once
        uint32_t tot = 0;
        // skip_chunk (a test hook) never publishes: its successors wait until wait_ns runs out
        const bool publish = chunk != skip_chunk;
        if ((uint32_t)tid <= dmask) {
#pragma unroll 8
            for (int w = 0; w < kWarps; w++) {
                const uint32_t c = sm.hist[w][tid];
                sm.hist[w][tid] = (uint16_t)tot;
                tot += c;
            }
            if (publish) lookback_publish(status + tid, chunk, kRadix, tot);
        }
        const uint32_t start = block_excl_scan(tot, sm.warp, nullptr);
        if (tid < kRadix) sm.start[tid] = start;
        __syncthreads();
        // local sort of the chunk by digit
#pragma unroll
        for (int i = 0; i < kSortItems; i++) {
            if (i >= items) break;
            const uint32_t pos = warp * (items * 32) + i * 32 + lane;
            if (pos < count) {
                const uint32_t dg = (key[i] >> shift) & dmask;
                const uint32_t lp = sm.start[dg] + sm.hist[warp][dg] + rank[i];
                sm.keys[lp] = key[i];
                sm.vals[lp] = vals_in ? __ldg(vals_in + base + pos) : base + pos;
            }
        }
        // global offset of this chunk's digit run
        if ((uint32_t)tid <= dmask)
            sm.gbase[tid] = gofs + thread_lookback_walk<32>(status + tid, chunk, kRadix, tot, err, wait_ns, publish);
        __syncthreads();
        for (uint32_t p = tid; p < count; p += kThreads) {
            const uint32_t k = sm.keys[p];
            const uint32_t dg = (k >> shift) & dmask;
            const uint32_t gp = sm.gbase[dg] + (p - sm.start[dg]);
            const uint32_t v = sm.vals[p];
            if (gp >= n) {  // cannot happen with consistent histograms; never write out of bounds
                set_error(err, FGS_ERR_OVERFLOW);
                continue;
            }
            if (keys_out) keys_out[gp] = k;
            vals_out[gp] = v;
        }
        __syncthreads();  // shared buffers are reused by the next chunk
    }
}

constexpr int kDepthThreads = 512, kTileThreads = 1024;

// Histograms of the 4 depth-key bytes (one read of the keys).
__global__ void depth_hist_kernel(const uint32_t* __restrict__ keys, uint32_t n,
                                  const unsigned long long* __restrict__ n_dev, uint32_t* __restrict__ hist)
{
    __shared__ uint32_t s[4][kRadix];
    n = (uint32_t)min((unsigned long long)n, *n_dev);
    for (int i = threadIdx.x; i < 4 * kRadix; i += blockDim.x) (&s[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = __ldg(keys + i);
#pragma unroll
        for (int b = 0; b < 4; b++) atomicAdd(&s[b][(k >> (8 * b)) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * kRadix; i += blockDim.x) {
        const uint32_t c = (&s[0][0])[i];
        if (c) atomicAdd(hist + i, c);
    }
}

// duplicateWithKeys over the depth-ordered Gaussians, in two kernels.
//
// pair_offsets_kernel: the prefix sum of tiles_touched in depth order (decoupled look-back
// over chunks of 2048 Gaussians, eight per thread), and per depth rank j the tile rectangle
// its pairs walk: off[j] the first pair, corner[j] the rectangle's first tile, w[j] its
// width; per Gaussian the emission row for the sort's gather.
//
// emit_pairs_kernel: the pairs themselves, kEmitPairs consecutive ones per block whatever
// Gaussians they belong to.  A block finds its first and last Gaussian by a 32-way search of
// off[], holds their offsets in shared memory and every pair finds its Gaussian there by
// bisection.  In depth order the near Gaussians come first and cover hundreds of tiles
// each, so blocks that took a fixed number of Gaussians (one kernel with the prefix sum)
// left the SMs idle three quarters of the time behind the first few: 2.09M pairs of 130K
// Gaussians 128 us -> 16 + 19.  Also builds the tile digit histograms of the tile sort.
constexpr int kOffItems = 8;
constexpr uint32_t kOffChunk = 256u * kOffItems;
constexpr uint32_t kEmitPairs = 2048;

__global__ void __launch_bounds__(256)
    pair_offsets_kernel(const uint32_t* __restrict__ sorted_ids, const uint32_t* __restrict__ tiles,
                        const PairRecord* __restrict__ grec, const int* __restrict__ radii, uint32_t V, int gx,
                        int gy, uint32_t* status, uint32_t* chunk_counter,
                        const unsigned long long* __restrict__ V_dev, uint32_t* __restrict__ off,
                        uint32_t* __restrict__ corner, uint32_t* __restrict__ w, int2* __restrict__ erow, unsigned* err)
{
    __shared__ uint32_t s_cnt[kOffChunk];  // counts, then exclusive prefixes within the chunk
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_chunk, s_prefix;
    const int tid = threadIdx.x;
    V = (uint32_t)min((unsigned long long)V, *V_dev);
    const uint32_t live = (V + kOffChunk - 1) / kOffChunk;
    if (blockIdx.x >= live) return;
    for (;;) {
        if (tid == 0) s_chunk = atomicAdd(chunk_counter, 1u);
        __syncthreads();
        const uint32_t chunk = s_chunk;
        if (chunk >= live) break;
        const uint32_t base = chunk * kOffChunk;
        uint32_t id[kOffItems];
#pragma unroll
        for (int i = 0; i < kOffItems; i++) {
            const uint32_t j = base + i * 256 + tid;
            id[i] = j < V ? __ldg(sorted_ids + j) : 0xffffffffu;
        }
#pragma unroll
        for (int i = 0; i < kOffItems; i++) s_cnt[i * 256 + tid] = id[i] != 0xffffffffu ? __ldg(tiles + id[i]) : 0u;
        __syncthreads();
        uint32_t c[kOffItems], sum = 0;
#pragma unroll
        for (int i = 0; i < kOffItems; i++) {
            c[i] = s_cnt[tid * kOffItems + i];
            sum += c[i];
        }
        uint32_t total;
        uint32_t at = block_excl_scan(sum, s_warp, &total);
#pragma unroll
        for (int i = 0; i < kOffItems; i++) {
            s_cnt[tid * kOffItems + i] = at;
            at += c[i];
        }
        if (tid < 32) {
            const uint32_t e = warp_lookback(status, chunk, 1, total, err);
            if (tid == 0) s_prefix = e;
        }
        __syncthreads();
        const uint32_t prefix = s_prefix;
#pragma unroll
        for (int i = 0; i < kOffItems; i++) {
            if (id[i] == 0xffffffffu) continue;
            const uint32_t j = base + i * 256 + tid;
            const float2 m = *reinterpret_cast<const float2*>(&grec[id[i]].a);
            int x0, y0, x1, y1;
            tile_rect(m.x, m.y, __ldg(radii + id[i]), gx, gy, kTileX, kTileY, x0, y0, x1, y1);
            const uint32_t o = prefix + s_cnt[i * 256 + tid], wd = (uint32_t)max(1, x1 - x0);
            // Gaussian j's pairs are [off[j], off[j + 1]); the emission index of tile (tx, ty) is
            // erow.x + ty * erow.y + tx (unsigned wrap-around)
            off[j] = o;
            corner[j] = (uint32_t)y0 * (uint32_t)gx + (uint32_t)x0;
            w[j] = wd;
            erow[id[i]] = make_int2((int)(o - (uint32_t)y0 * wd - (uint32_t)x0), (int)wd);
        }
        __syncthreads();  // the shared arrays are reused by the next chunk
    }
}

// Last rank j < V with off[j] <= p (off[0] = 0), by one warp: 32 probes per step.
__device__ __forceinline__ uint32_t rank_of_pair(const uint32_t* __restrict__ off, uint32_t V, uint32_t p)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, n = V;  // the answer lies in [lo, lo + n)
    while (n > 1) {
        const uint32_t step = (n + 31) / 32, at = lane * step;
        const bool le = at < n && __ldg(off + lo + at) <= p;  // monotone over the lanes; lane 0 holds
        const uint32_t k = (uint32_t)(31 - __clz(__ballot_sync(0xffffffffu, le)));
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

// (Offsets that a look-back which ran out of time left inconsistent keep every index inside
// its array: ranks below V, at most kEmitPairs of them, tiles below num_tiles.)
__global__ void __launch_bounds__(256)
    emit_pairs_kernel(const uint32_t* __restrict__ sorted_ids, const uint32_t* __restrict__ off,
                      const uint32_t* __restrict__ corner, const uint32_t* __restrict__ w, uint32_t V, uint32_t K, int gx,
                      uint32_t num_tiles, const unsigned long long* __restrict__ totals, uint32_t* __restrict__ tile_out,
                      uint32_t* __restrict__ val_out, uint32_t* __restrict__ tile_hist, int tile_passes, unsigned* err)
{
    __shared__ uint32_t s_hist[4][kRadix];
    __shared__ uint32_t s_off[kEmitPairs];
    __shared__ uint32_t s_j[2];
    const int tid = threadIdx.x;
    V = (uint32_t)min((unsigned long long)V, totals[1]);
    if (totals[0] > K && blockIdx.x == 0 && tid == 0) set_error(err, FGS_ERR_OVERFLOW);  // truncated at the capacity
    K = (uint32_t)min((unsigned long long)K, totals[0]);
    const uint32_t chunks = (K + kEmitPairs - 1) / kEmitPairs;
    if (V == 0 || blockIdx.x >= chunks) return;
    for (int i = tid; i < tile_passes * kRadix; i += 256) (&s_hist[0][0])[i] = 0;
    for (uint32_t chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
        const uint32_t p0 = chunk * kEmitPairs, p1 = min(K, p0 + kEmitPairs);
        if (tid < 64) {
            const uint32_t j = rank_of_pair(off, V, tid < 32 ? p0 : p1 - 1);
            if ((tid & 31) == 0) s_j[tid >> 5] = j;
        }
        __syncthreads();
        const uint32_t j0 = s_j[0];
        const uint32_t nj = s_j[1] < j0 ? 1u : min(s_j[1] - j0 + 1, kEmitPairs);  // at most one Gaussian per pair
        for (uint32_t i = tid; i < nj; i += 256) s_off[i] = __ldg(off + j0 + i);
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < kEmitPairs / 256; i++) {
            const uint32_t p = p0 + i * 256 + tid;
            if (p >= p1) break;
            uint32_t lo = 0, hi = nj;  // last entry with s_off <= p lies in [lo, hi)
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_off[mid] <= p) lo = mid;
                else hi = mid;
            }
            const uint32_t j = j0 + lo, t = p - s_off[lo], wd = __ldg(w + j), c = __ldg(corner + j);
            const uint32_t ty = t / wd, tx = t - ty * wd;
            uint32_t tile = c + ty * (uint32_t)gx + tx;
            if (tile >= num_tiles) {
                set_error(err, FGS_ERR_OVERFLOW);
                tile = num_tiles - 1;
            }
            tile_out[p] = tile;
            val_out[p] = __ldg(sorted_ids + j);
            for (int b = 0; b < tile_passes; b++) atomicAdd(&s_hist[b][(tile >> (8 * b)) & 255u], 1u);
        }
        __syncthreads();  // s_j and s_off are rewritten for the next chunk
    }
    for (int i = tid; i < tile_passes * kRadix; i += 256) {
        const uint32_t c = (&s_hist[0][0])[i];
        if (c) atomicAdd(tile_hist + i, c);
    }
}

// identifyTileRanges (rasterizer_impl.cu:172-194): the first pair of every tile by a
// search of the sorted tile ids, one lane per tile, 31 tiles per warp (a tile ends where
// the next lane's starts).  Four-way, three loads in flight per step: bound by the
// latency of its ~11 dependent steps, where a pass over all pairs that compares
// neighbours needs a zeroed table first and 16 bytes per pair of traffic (9.4 us plus the
// memset for 1.75M pairs; this one 5 us for both).  The same warps list the tiles that the
// launch rule renders in units, one atomic per warp and bin.
__device__ __forceinline__ void find_ranges(const uint32_t* __restrict__ tile, uint32_t K, uint2* __restrict__ ranges,
                                            uint32_t num_tiles, uint32_t warp, const LongList& lng)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t t = warp * 31 + lane;
    uint32_t lo = 0, hi = K;  // the first pair whose tile is >= t lies in [lo, hi]
    while (lo < hi) {
        const uint32_t q = (hi - lo) >> 2;
        const uint32_t m0 = lo + q, m1 = lo + 2 * q, m2 = lo + 3 * q;  // lo <= m0 <= m1 <= m2 < hi
        const bool b0 = __ldg(tile + m0) < t, b1 = __ldg(tile + m1) < t, b2 = __ldg(tile + m2) < t;
        if (b2) lo = m2 + 1;
        else if (b1) { lo = m1 + 1; hi = m2; }
        else if (b0) { lo = m0 + 1; hi = m1; }
        else hi = m0;
    }
    const uint32_t end = __shfl_down_sync(0xffffffffu, lo, 1);
    const bool mine = lane < 31 && t < num_tiles;
    const uint32_t n = mine ? end - lo : 0u;
    if (mine) ranges[t] = n ? make_uint2(lo, end) : make_uint2(0u, 0u);
    if (!lng.list) return;
    const bool is_long = n != 0 && n >= auto_split_min(lng.totals);
    uint32_t todo = __ballot_sync(0xffffffffu, is_long);
    const int bin = is_long ? 31 - __clz(n) : 0;
    while (todo) {
        const int lead = __ffs(todo) - 1;
        const int b = __shfl_sync(0xffffffffu, bin, lead);
        const uint32_t same = __ballot_sync(0xffffffffu, is_long && bin == b);
        todo &= ~same;
        uint32_t at = 0;
        if ((int)lane == lead) {
            at = atomicAdd(lng.ctr + 2 + b, (uint32_t)__popc(same));
            atomicAdd(lng.ctr, (uint32_t)__popc(same));
        }
        at = __shfl_sync(0xffffffffu, at, lead);
        if ((same >> lane) & 1u)
            lng.list[(size_t)b * lng.cap + at + __popc(same & ((1u << lane) - 1u))] = lng.id_base + t;
        if (lng.kv_sum)
            for (uint32_t m = same; m; m &= m - 1) {
                const int l = __ffs(m) - 1;
                const uint32_t x0 = __shfl_sync(0xffffffffu, lo, l), x1 = __shfl_sync(0xffffffffu, end, l);
                for (uint32_t i = x0 + lane; i < x1; i += 32) {
                    lng.kv_sum[i] = 0.f;
                    lng.kv_cnt[i] = 0u;
                }
            }
    }
}

// What follows the tile sort: the first range_blocks blocks find the tiles' ranges, the others
// write the pairs' records in sorted order, 32 per warp.  A warp moves these as 96 items of 16
// bytes, lane by lane along the records, both from the Gaussians' table and to the sorted
// list, and meets them whole in shared memory in between.  The last sort pass wrote the records
// before, at one block of 1024 threads per SM, eight to sixteen records in a row per thread;
// with 2048 threads per SM their masks (some 200 instructions each) and the gathers overlap,
// and so do the searches, which wait for memory.  2.1M pairs: last pass and ranges
// 90 us, last pass and this launch 75.
constexpr int kPlaceThreads = 256;
__global__ void __launch_bounds__(kPlaceThreads, 6)
    place_kernel(const uint32_t* __restrict__ tile, const uint32_t* __restrict__ vals, uint32_t K,
                 const unsigned long long* __restrict__ n_dev, uint2* __restrict__ ranges, uint32_t num_tiles,
                 LongList lng, uint32_t range_blocks, const PairRecord* __restrict__ grec,
                 const int2* __restrict__ erow, uint32_t P, uint32_t gx, PairRecord* __restrict__ rec_out, unsigned* err)
{
    __shared__ float4 s_rec[kPlaceThreads / 32][96];
    if (n_dev) K = (uint32_t)min((unsigned long long)K, *n_dev);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x < range_blocks) {
        find_ranges(tile, K, ranges, num_tiles, blockIdx.x * (kPlaceThreads / 32) + warp, lng);
        return;
    }
    const uint32_t p0 = (blockIdx.x - range_blocks) * kPlaceThreads + 32 * warp, p = p0 + lane;
    if (p0 >= K) return;  // (the same on the whole warp)
    float4* W = s_rec[warp];
    uint32_t k = 0, v = 0xffffffffu;
    if (p < K) {
        k = __ldg(tile + p);
        v = __ldg(vals + p);
        if (v >= P) {  // cannot happen with consistent histograms; never read out of bounds
            set_error(err, FGS_ERR_OVERFLOW);
            v = 0xffffffffu;
        }
    }
    int2 er = make_int2(0, 0);
    if (v != 0xffffffffu) er = __ldg(erow + v);
#pragma unroll
    for (int t = 0; t < 3; t++) {
        const uint32_t q = 32 * t + lane, j = q / 3, part = q - 3 * j;
        const uint32_t vj = __shfl_sync(0xffffffffu, v, j);
        W[q] = vj != 0xffffffffu ? __ldg(reinterpret_cast<const float4*>(grec + vj) + part) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncwarp();
    if (v != 0xffffffffu) {
        // The record also carries the pair's emission index: the Gaussian's first pair plus
        // this tile's row-major place in its tile rectangle (the order in which
        // emit_pairs_kernel emitted them), from the row base and width that
        // pair_offsets_kernel left per Gaussian.  The backward writes the pair's gradients
        // there, so each Gaussian's pairs are contiguous and are summed in a fixed order.
        const PairRecord r = {W[3 * lane], W[3 * lane + 1], W[3 * lane + 2]};
        const uint32_t ty = k / gx, tx = k - ty * gx;
        W[3 * lane + 2].z = __uint_as_float(block_mask(r, (float)(tx * kTileX), (float)(ty * kTileY)));
        W[3 * lane + 2].w = __uint_as_float((uint32_t)er.x + ty * (uint32_t)er.y + tx);
    }
    __syncwarp();
    float4* out = reinterpret_cast<float4*>(rec_out + p0);
    const uint32_t n = 3 * min(32u, K - p0);
#pragma unroll
    for (int t = 0; t < 3; t++) {
        const uint32_t q = 32 * t + lane;
        if (q < n) out[q] = W[q];
    }
}

inline uint32_t chunks_of(long long n, int tile) { return (uint32_t)((n + tile - 1) / tile); }

// Test hook of the first depth-sort pass (fgs_debug_lookback_fault): the chunk
// that never publishes its counts and the wait limit of that pass.
unsigned long long g_fault_wait_ns = kWaitLimitNs;
uint32_t g_fault_skip_chunk = 0xffffffffu;

}  // namespace

void set_lookback_fault(uint32_t skip_chunk, unsigned long long wait_ns)
{
    g_fault_skip_chunk = skip_chunk;
    g_fault_wait_ns = wait_ns ? wait_ns : kWaitLimitNs;
}

int sort_chunk_size() { return kSortTileMin; }  // the smallest chunk: sizes the status words

void launch_depth_sort(const GeomState& g, int P, cudaStream_t s)
{
    // the V visible Gaussians (count on the device, bound P): keys depth_key[0..V), ids sort_ids_b[0..V)
    if (P <= 0) return;
    const uint32_t n = (uint32_t)P;
    const unsigned long long* V = g.total + 1;
    const uint32_t nch = chunks_of(n, kSortTileMin);
    const uint32_t hb0 = (n + 1023) / 1024;
    const int hb = (int)(hb0 < 1184u ? hb0 : 1184u);
    depth_hist_kernel<<<hb, 256, 0, s>>>(g.depth_key, n, V, g.hist);
    const size_t smem = sizeof(SortSmem<kDepthThreads>);
    const uint32_t grid = min(nch, resident_ctas(onesweep_kernel<kDepthThreads>, kDepthThreads, smem));
    note_launches(5);
    // ping-pong: depth_key -> sort_keys_b -> depth_key -> sort_keys_b ; ids b -> a -> b -> a -> b
    const uint32_t* kin[4] = {g.depth_key, g.sort_keys_b, g.depth_key, g.sort_keys_b};
    uint32_t* kout[4] = {g.sort_keys_b, g.depth_key, g.sort_keys_b, nullptr};
    const uint32_t* vin[4] = {g.sort_ids_b, g.sort_ids_a, g.sort_ids_b, g.sort_ids_a};
    uint32_t* vout[4] = {g.sort_ids_a, g.sort_ids_b, g.sort_ids_a, g.sort_ids_b};
    for (int pass = 0; pass < 4; pass++) {
        onesweep_kernel<kDepthThreads><<<grid, kDepthThreads, smem, s>>>(
            kin[pass], kout[pass], vin[pass], vout[pass], n, 8 * pass, 8, g.hist + pass * kRadix,
            g.status + (size_t)pass * nch * kRadix, g.counters + pass, g.err, V,
            pass ? kWaitLimitNs : g_fault_wait_ns, pass ? 0xffffffffu : g_fault_skip_chunk);
    }
}

void launch_duplicate(const GeomState& g, const BinState& b, uint32_t V, uint32_t K, int W, int H, int tile_bits,
                      cudaStream_t s)
{
    if (V == 0) return;
    const int gx = (W + kTileX - 1) / kTileX, gy = (H + kTileY - 1) / kTileY;
    const int passes = (tile_bits + 7) / 8;
    // The tile sort ping-pongs between the a/b buffers and must end in b:
    // with an odd number of passes it starts from a, with an even one from b.
    uint32_t* tout = (passes & 1) ? b.tile_a : b.tile_b;
    uint32_t* vout = (passes & 1) ? b.val_a : b.val_b;
    // the depth keys and the other id buffer are free once the Gaussians are sorted
    uint32_t *corner = g.depth_key, *w = g.sort_ids_a;
    const uint32_t grid = min(chunks_of(V, kOffChunk), resident_ctas(pair_offsets_kernel, 256));
    pair_offsets_kernel<<<grid, 256, 0, s>>>(g.sort_ids_b, g.tiles, g.grec, g.radii, V, gx, gy, b.scan_status,
                                             g.counters + 8, g.total + 1, g.pair_off, corner, w, g.erow, g.err);
    const uint32_t egrid = min(chunks_of(K, kEmitPairs), resident_ctas(emit_pairs_kernel, 256));
    emit_pairs_kernel<<<egrid, 256, 0, s>>>(g.sort_ids_b, g.pair_off, corner, w, V, K, gx, (uint32_t)(gx * gy), g.total,
                                            tout, vout, g.hist + 4 * kRadix, passes, g.err);
    note_launches(2);
}

void launch_tile_sort(const GeomState& g, const BinState& b, long long K, int tile_bits, cudaStream_t s,
                      const unsigned long long* n_dev)
{
    if (K <= 0) return;
    const uint32_t n = (uint32_t)K;
    const uint32_t nch = chunks_of(n, kSortTileMin);
    const size_t smem = sizeof(SortSmem<kTileThreads>);
    const uint32_t grid = min(nch, resident_ctas(onesweep_kernel<kTileThreads>, kTileThreads, smem));
    const int passes = (tile_bits + 7) / 8;
    const uint32_t* ki = (passes & 1) ? b.tile_a : b.tile_b;
    const uint32_t* vi = (passes & 1) ? b.val_a : b.val_b;
    for (int pass = 0; pass < passes; pass++) {
        const int nbits = min(8, tile_bits - 8 * pass);
        uint32_t* ko = (ki == b.tile_a) ? b.tile_b : b.tile_a;
        uint32_t* vo = (vi == b.val_a) ? b.val_b : b.val_a;
        onesweep_kernel<kTileThreads><<<grid, kTileThreads, smem, s>>>(
            ki, ko, vi, vo, n, 8 * pass, nbits, g.hist + (4 + pass) * kRadix,
            b.status + (size_t)pass * nch * kRadix, g.counters + 4 + pass, g.err, n_dev);
        ki = ko;
        vi = vo;
    }
    note_launches(passes);
}

void launch_ranges(const GeomState& g, const BinState& b, const ImageState& im, long long K, int P, int W, int num_tiles,
                   cudaStream_t s, const unsigned long long* n_dev, const LongList& lng)
{
    if (K <= 0) {
        cudaMemsetAsync(im.ranges, 0, sizeof(uint2) * (size_t)num_tiles, s);
        return;
    }
    const uint32_t range_blocks = chunks_of(chunks_of(num_tiles, 31), kPlaceThreads / 32);
    place_kernel<<<range_blocks + chunks_of(K, kPlaceThreads), kPlaceThreads, 0, s>>>(
        b.tile_b, b.val_b, (uint32_t)K, n_dev, im.ranges, (uint32_t)num_tiles, lng, range_blocks, g.grec, g.erow,
        (uint32_t)P, (uint32_t)((W + kTileX - 1) / kTileX), b.rec, g.err);
    note_launches(1);
}

}  // namespace fgs
