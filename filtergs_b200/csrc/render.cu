// Tile compositing, forward and backward
// (antialias/cuda_rasterizer/forward.cu:406-567, backward.cu:399-557).
//
// One CTA per 16x16 tile.  The tile's sorted pairs are contiguous 48-byte
// records (written after the tile sort), so each record batch is ONE bulk copy
// (cp.async.bulk, the TMA engine's 1-D form) into shared memory, completed on an
// mbarrier.  Three record buffers keep two batches in flight while the current
// one is composited.  A warp owns a block of pixels (PPT of one column per lane), and a
// record carries the mask of the tile's eight 8x4 blocks it can reach (block_mask,
// written with it): one ballot per 32 records tells a warp which to composite.
//
// Both directions are bound by instruction issue (80% and 77% of the issue slots of
// 1080p views), so two pixels of a lane are composited per instruction with packed
// fma / mul / add.f32x2, which round each half as the scalar operation does, and a
// record's masks are formed once, not once per warp and direction.  Sixteen 1080p views
// (27.9M pairs): forward 4.81 -> 3.67 ms, backward 7.81 -> 6.93 ms (6.55 with the sums of 8x8
// quads, whose order depended on the shape); one such view: 361 -> 296 and 505 -> 415 us with
// the gradient buffers zeroed; 10,000 Gaussians at 256x256: 72 -> 60 and 93 -> 48 us.
//
// Per-Gaussian outputs that the reference updates from every pixel (the
// racy out_point_weight max, the KPC statistics, the backward's 9 gradient
// atomics) are reduced across the warp first, then across the CTA in shared
// memory, and leave the CTA once per (tile, pair).
#include <cstddef>

#include "fgs_common.cuh"
#include "fgs_internal.h"

namespace fgs {

namespace {

constexpr int kBufs = 3;

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false (and an error bit) if the copy never lands.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned* err)
{
    WaitBound wb;
    while (!mbar_try_wait(bar, parity)) {
        if (wb.expired(kWaitLimitNs)) {
            set_error(err, FGS_ERR_TIMEOUT);
            return false;
        }
    }
    return true;
}
// 1-D bulk copy global -> shared, completion counted on `bar`.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Issue the bulk copy of records [first, first+count) into buffer `buf`.
__device__ __forceinline__ void issue_batch(PairRecord* sbuf, uint64_t* bar, const PairRecord* recs, uint32_t first,
                                            uint32_t count)
{
    const uint32_t bytes = count * (uint32_t)sizeof(PairRecord);
    mbar_expect_tx(bar, bytes);
    bulk_g2s(sbuf, recs + first, bytes, bar);
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The forward's block of pixels of this thread's warp: 8 columns x 4 PPT rows of the tile,
// lane (x, y) = (lane & 7, lane >> 3), its pixel k at row y + 4 k.
template <int PPT>
struct WarpBlock {
    int px, py0, bit;  // first pixel; the block's first bit in a record's block_mask
    __device__ __forceinline__ WarpBlock(int bx, int by)
    {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int col = w & 1, row = (w >> 1) * 4 * PPT;
        bit = 2 * (row >> 2) + col;
        px = bx * kTileX + 8 * col + (lane & 7);
        py0 = by * kTileY + row + (lane >> 3);
    }
};
// Quads of 8x8 pixels one warp's block covers (a block of PPT = 1 is half a quad), and the
// block_mask bits of one of them above the block's first bit.
template <int PPT>
constexpr int warp_quads() { return PPT == 4 ? 2 : 1; }
template <int PPT>
constexpr uint32_t quad_bits() { return PPT == 1 ? 1u : 5u; }

// ---------------------------------------------------------------- per-view render descriptors
// Everything one tile needs, for the plain launch (one view, one tile per CTA)
// and the persistent multi-view launch (CTAs pop (view, tile) work items).

// The statistics sums come last: a launch without statistics allocates the
// dynamic shared memory only up to ksum (fwd_smem_bytes), which leaves room for
// one more CTA per SM at the batch sizes the autotuner picks.
template <int kBatch>
struct FwdSmem {
    PairRecord rec[kBufs][kBatch];
    uint64_t bar[kBufs];
    uint32_t wmax[2][kBatch];
    float ksum[2][kBatch];
    uint32_t kcnt[2][kBatch];
};

constexpr int kPend = 4;  // steps that add_step_sums adds at once

// The nine sums of up to kPend (record, strip) steps of a warp, every lane's, until
// add_step_sums adds them over the lanes: a[half] holds four sums of each lane (lane l
// of the second half at l ^ 4, so that the eight lanes that read a step meet no bank
// twice), b the ninth.
struct __align__(16) StepSums {
    struct {
        float4 a[2][32];
        float b[40];
    } step[kPend];
    int rec[kPend];  // the record's index in the batch
};

// Per-record gradient sums of a batch.  With two warps per tile (PPT = 4) each has a slot of
// its own.  With more, warps 2s and 2s+1 add into slot s: a slot starts at zero and takes at
// most two additions per record, and float addition is commutative, so its value does not
// depend on which warp came first.  Slots are added in order.  Either way the result is the
// same on every run (no order-dependent float atomics anywhere in the backward).
template <int PPT>
constexpr int bwd_slots() { return PPT == 4 ? 2 : (256 / PPT / 32) / 2; }

template <int PPT, int kBatch>
struct BwdSmem {
    PairRecord rec[kBufs][kBatch];
    StepSums step[PPT == 1 ? 1 : 8 / PPT];
    uint64_t bar[kBufs];
    float acc[kBufs][bwd_slots<PPT>()][kBatch][9];
    uint32_t arrived[kBufs];  // warps that are through with a batch
    uint32_t max_last;
};

// ---------------------------------------------------------------- forward
// One (pixel, record) step of the compositing loop (forward.cu:466-544), in two
// parts.  fwd_alpha: the Gaussian's alpha at the pixel centre, or 0 where the
// reference skips the record (power > 0, alpha < 1/255); it does not depend on
// the pixel's state, so a renderer may evaluate several records ahead.
// fwd_accumulate: early termination below T = 1e-4, the colour and
// transmittance update and the pixel's strongest contributor; returns the
// weight T * alpha the record took (> 0), or 0 when it did not contribute.
//
// The multiply-adds are spelled out with round-to-nearest intrinsics (the
// contraction a compiler would pick for the reference's expressions), so that
// the compiler cannot fuse them differently in different renderers: the tile
// path at any pixels-per-thread and the band path produce the same bits.
__device__ __forceinline__ float fwd_alpha(const float4 ra, const float4 rb, float pxf, float pyf)
{
    const float dx = ra.x - pxf, dy = ra.y - pyf;
    // -0.5 * (a dx^2 + c dy^2) - b dx dy with the first product of each sum fused
    // into the multiply-add: of the orders measured, the one whose alphas agree
    // with the reference build's on the most pixels
    const float q = __fmaf_rn(__fmul_rn(ra.z, dx), dx, __fmul_rn(__fmul_rn(rb.x, dy), dy));
    const float power = __fmaf_rn(-0.5f, q, -__fmul_rn(__fmul_rn(ra.w, dx), dy));
    if (power > 0.0f) return 0.f;
    const float alpha = fminf(0.99f, __fmul_rn(rb.y, expf(power)));
    return alpha < 1.0f / 255.0f ? 0.f : alpha;
}

__device__ __forceinline__ float fwd_accumulate(float alpha, const float4 rb, const PairRecord& rec,
                                                uint32_t position, float& T, float (&C)[3], float& wmax, int& maxid,
                                                uint32_t& last, bool& done)
{
    if (done || alpha == 0.f) return 0.f;
    const float test_T = __fmul_rn(T, 1.0f - alpha);
    if (test_T < 0.0001f) {
        done = true;
        return 0.f;
    }
    const float4 rc = rec.c;
    C[0] = __fmaf_rn(__fmul_rn(rb.z, alpha), T, C[0]);
    C[1] = __fmaf_rn(__fmul_rn(rb.w, alpha), T, C[1]);
    C[2] = __fmaf_rn(__fmul_rn(rc.x, alpha), T, C[2]);
    const float w = __fmul_rn(T, alpha);
    if (w > wmax) {
        wmax = w;
        maxid = __float_as_int(rc.y);
    }
    T = test_T;
    last = position;
    return w;
}

// What a forward launch keeps beside the image: nothing (a batched view without these
// outputs), point_id / point_weight_pixel / point_weight, or those and the statistics.
enum { kImage = 0, kWeights = 1, kStats = 2 };

// One pixel's state between records: colour and the strongest contributor as in
// fwd_accumulate; T is the transmittance, negative once the pixel takes no record any more
// (it lies outside the image, or the next record would have brought T below 1e-4).

// One record on one pixel, with branches: the form for one pixel per lane, and for a
// record whose colour or position is too large for the packed form (kWild), where a
// pixel the record does not reach must not see 0 * inf.  Returns the weight T * alpha
// the record took, 0 when it did not contribute.
__device__ __forceinline__ float fwd_pixel_step(const float4 ra, const float4 rb, float c2, int id, float pxf,
                                                float pyf, uint32_t position, float& T, float& C0, float& C1,
                                                float& C2, float& wmax, int& maxid, uint32_t& last)
{
    if (T < 0.f) return 0.f;
    const float alpha = fwd_alpha(ra, rb, pxf, pyf);
    if (alpha == 0.f) return 0.f;
    const float test_T = __fmul_rn(T, 1.0f - alpha);
    if (test_T < 0.0001f) {
        T = -T;
        return 0.f;
    }
    C0 = __fmaf_rn(__fmul_rn(rb.z, alpha), T, C0);
    C1 = __fmaf_rn(__fmul_rn(rb.w, alpha), T, C1);
    C2 = __fmaf_rn(__fmul_rn(c2, alpha), T, C2);
    const float w = __fmul_rn(T, alpha);
    if (w > wmax) {
        wmax = w;
        maxid = id;
    }
    T = test_T;
    last = position;
    return w;
}

// The pixels of one lane in pairs (k = 2q, 2q + 1).
template <int NP>
struct FwdPixels {
    F2 T[NP], C[NP][3], wmax[NP], npy[NP];  // npy: -row
    int maxid[2 * NP];
    uint32_t last[2 * NP];
};

// One record on one pair of pixels, without branches: a pixel that does not take the
// record gets alpha 0, which leaves the colours and the weight as they are (C + 0 * T).
// The same operations, in the same order and rounding, as fwd_alpha and fwd_accumulate.
// A pixel that is done has T < 0, so its product with 1 - alpha is below 1e-4 for every
// record: one comparison tells both.  Returns the larger of the two weights (kImage:
// alphas): > 0 when either pixel took something.
template <int kOut, int NP>
__device__ __forceinline__ float fwd_pair_step(FwdPixels<NP>& s, int q, const float4 ra, const float4 rb, float c2,
                                               int id, float dx, float sx, float nbx, uint32_t position, F2& wsum,
                                               uint32_t& wcount)
{
    const F2 dy = f2_add(f2(ra.y), s.npy[q]);
    const F2 qf = f2_fma(f2(sx), f2(dx), f2_mul(f2_mul(f2(rb.x), dy), dy));
    const F2 power = f2_fma(f2(-0.5f), qf, f2_mul(f2(nbx), dy));
    const F2 oG = f2_mul(f2(rb.y), f2(expf(f2_lo(power)), expf(f2_hi(power))));
    const F2 a = f2(fminf(0.99f, f2_lo(oG)), fminf(0.99f, f2_hi(oG)));
    const F2 test_T = f2_mul(s.T[q], f2_fma(a, f2(-1.f), f2(1.f)));  // T (1 - alpha)
    const bool ok0 = !(f2_lo(power) > 0.f) && f2_lo(a) >= 1.0f / 255.0f;
    const bool ok1 = !(f2_hi(power) > 0.f) && f2_hi(a) >= 1.0f / 255.0f;
    const bool take0 = ok0 && !(f2_lo(test_T) < 0.0001f), take1 = ok1 && !(f2_hi(test_T) < 0.0001f);
    const F2 alpha = f2(take0 ? f2_lo(a) : 0.f, take1 ? f2_hi(a) : 0.f);
    s.C[q][0] = f2_fma(f2_mul(f2(rb.z), alpha), s.T[q], s.C[q][0]);
    s.C[q][1] = f2_fma(f2_mul(f2(rb.w), alpha), s.T[q], s.C[q][1]);
    s.C[q][2] = f2_fma(f2_mul(f2(c2), alpha), s.T[q], s.C[q][2]);
    s.last[2 * q] = take0 ? position : s.last[2 * q];
    s.last[2 * q + 1] = take1 ? position : s.last[2 * q + 1];
    float took = fmaxf(f2_lo(alpha), f2_hi(alpha));
    if constexpr (kOut != kImage) {
        const F2 w = f2_mul(s.T[q], alpha);
        const float w0 = f2_lo(w), w1 = f2_hi(w);
        const bool g0 = w0 > f2_lo(s.wmax[q]), g1 = w1 > f2_hi(s.wmax[q]);
        s.wmax[q] = f2(g0 ? w0 : f2_lo(s.wmax[q]), g1 ? w1 : f2_hi(s.wmax[q]));
        s.maxid[2 * q] = g0 ? id : s.maxid[2 * q];
        s.maxid[2 * q + 1] = g1 ? id : s.maxid[2 * q + 1];
        took = fmaxf(w0, w1);
        if constexpr (kOut == kStats) {
            wsum = f2_add(wsum, f2(fmaxf(w0, 0.f), fmaxf(w1, 0.f)));
            wcount += (int)take0 + (int)take1;
        }
    }
    // taken: T (1 - alpha); reached but not taken: done; else unchanged
    const float T0 = f2_lo(s.T[q]), T1 = f2_hi(s.T[q]);
    s.T[q] = f2(take0 ? f2_lo(test_T) : (ok0 ? -fabsf(T0) : T0), take1 ? f2_hi(test_T) : (ok1 ? -fabsf(T1) : T1));
    return took;
}

// One tile.  Callers guarantee every thread of the CTA is synchronised on
// entry and that no bulk copy is in flight.  `gb` counts the record batches
// this CTA has ever waited for: batch g lives in buffer g % 3 and completes
// phase (g / 3) & 1 of that buffer's mbarrier, so the barriers are initialised
// once per CTA and keep their phase across tiles.
template <int PPT, int kBatch, int kOut>
__device__ __forceinline__ void render_fwd_tile(FwdSmem<kBatch>& sm, const TileArgs& a, int tile, uint32_t& gb,
                                                uint32_t split_min, unsigned* err)
{
    // (every thread of the CTA takes the same way here)
    constexpr int NT = 256 / PPT;
    constexpr int NP = PPT > 1 ? PPT / 2 : 1;
    constexpr int kQuads = warp_quads<PPT>();
    const int tid = threadIdx.x;
    const int W = a.W, H = a.H;
    const int gx = (W + kTileX - 1) / kTileX;
    const int bx = tile % gx, by = tile / gx;
    const WarpBlock<PPT> blk(bx, by);
    const int px = blk.px;
    const uint2 range = a.ranges[tile];
    const uint32_t n = range.y - range.x;
    if (split_min && n >= split_min) return;  // rendered in bands (render_long_tile)
    const int nb = (int)((n + kBatch - 1) / kBatch);
    const PairRecord* recs = a.recs;

    if (tid == 0) {
        for (int b = 0; b < 2 && b < nb; b++) {
            const int buf = (int)((gb + b) % kBufs);
            issue_batch(sm.rec[buf], &sm.bar[buf], recs, range.x + b * kBatch, min((uint32_t)kBatch, n - b * kBatch));
        }
    }

    FwdPixels<NP> s;
#pragma unroll
    for (int q = 0; q < NP; q++) {
        s.C[q][0] = s.C[q][1] = s.C[q][2] = f2(0.f);
        s.wmax[q] = f2(0.f);
        s.npy[q] = f2(-(float)(blk.py0 + 8 * q), -(float)(blk.py0 + 8 * q + 4));
        float T[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const bool inside = px < W && blk.py0 + 8 * q + 4 * h < H && 2 * q + h < PPT;
            T[h] = inside ? 1.f : -1.f;  // negative: takes no record any more
            s.last[2 * q + h] = 0;
            s.maxid[2 * q + h] = -1;
        }
        s.T[q] = f2(T[0], T[1]);
    }
    const float pxf = (float)px;
    auto all_done = [&] {
        bool d = true;
#pragma unroll
        for (int k = 0; k < PPT; k++) d = d && ((k & 1) ? f2_hi(s.T[k >> 1]) : f2_lo(s.T[k >> 1])) < 0.f;
        return d;
    };
    int issued = nb < 2 ? nb : 2;
    uint32_t contributor = 0;
    bool stop = __all_sync(0xffffffffu, all_done());  // warp-uniform: no pixel of the warp takes any more
    for (int b = 0; b < nb; b++) {
        const uint32_t g = gb + b;
        const int buf = (int)(g % kBufs);
        const int acc = b & 1;
        const uint32_t cnt = min((uint32_t)kBatch, n - b * kBatch);
        // (a copy that never lands: every thread gives up on the tile, the error is recorded)
        if (__any_sync(0xffffffffu, !mbar_wait(&sm.bar[buf], (g / kBufs) & 1, err))) stop = true;
        const PairRecord* R = sm.rec[buf];
        for (uint32_t k0 = 0; k0 < cnt && !stop; k0 += 32) {
            // which of these 32 records reach this warp's quads
            const uint32_t e = k0 + (tid & 31);
            const uint32_t mask = e < cnt ? __float_as_uint(R[e].c.z) >> blk.bit : 0u;
            uint32_t quad[kQuads], live = 0;
#pragma unroll
            for (int q = 0; q < kQuads; q++) {
                quad[q] = __ballot_sync(0xffffffffu, ((mask >> (4 * q)) & quad_bits<PPT>()) != 0);
                live |= quad[q];
            }
            while (live) {
                const uint32_t bit = (uint32_t)(__ffs(live) - 1);
                const uint32_t j = k0 + bit;
                live &= live - 1;
                const uint32_t position = contributor + j + 1;
                const float4 ra = R[j].a;
                const float4 rb = R[j].b;
                const float4 rc = R[j].c;
                float wj = 0.f;
                F2 wsum = f2(0.f);
                uint32_t kc = 0;
                if (PPT == 1 || (__float_as_uint(rc.z) & kWild)) {
#pragma unroll
                    for (int k = 0; k < PPT; k++) {
                        const int q = k >> 1;
                        float T = (k & 1) ? f2_hi(s.T[q]) : f2_lo(s.T[q]);
                        float C[3], wm = (k & 1) ? f2_hi(s.wmax[q]) : f2_lo(s.wmax[q]);
#pragma unroll
                        for (int c = 0; c < 3; c++) C[c] = (k & 1) ? f2_hi(s.C[q][c]) : f2_lo(s.C[q][c]);
                        const float pyf = -((k & 1) ? f2_hi(s.npy[q]) : f2_lo(s.npy[q]));
                        const float w = fwd_pixel_step(ra, rb, rc.x, __float_as_int(rc.y), pxf, pyf, position, T, C[0],
                                                       C[1], C[2], wm, s.maxid[k], s.last[k]);
                        wj = fmaxf(wj, w);
                        wsum = f2_add(wsum, f2(w, 0.f));
                        kc += w > 0.f;
                        s.T[q] = (k & 1) ? f2(f2_lo(s.T[q]), T) : f2(T, f2_hi(s.T[q]));
                        s.wmax[q] = (k & 1) ? f2(f2_lo(s.wmax[q]), wm) : f2(wm, f2_hi(s.wmax[q]));
#pragma unroll
                        for (int c = 0; c < 3; c++)
                            s.C[q][c] = (k & 1) ? f2(f2_lo(s.C[q][c]), C[c]) : f2(C[c], f2_hi(s.C[q][c]));
                    }
                } else {
                    const float dx = ra.x - pxf;
                    const float sx = __fmul_rn(ra.z, dx), nbx = -__fmul_rn(ra.w, dx);
#pragma unroll
                    for (int q = 0; q < NP; q++)
                        if (kQuads == 1 || ((quad[q] >> bit) & 1u))
                            wj = fmaxf(wj, fwd_pair_step<kOut, NP>(s, q, ra, rb, rc.x, __float_as_int(rc.y), dx, sx,
                                                                    nbx, position, wsum, kc));
                }
                if (!__any_sync(0xffffffffu, wj > 0.f)) {
                    // a record that nobody took: perhaps because every pixel is done
                    stop = __all_sync(0xffffffffu, all_done());
                    if (stop) break;
                    continue;
                }
                if constexpr (kOut != kImage) {
                    // per-Gaussian max weight (and statistics): warp, then CTA
                    const uint32_t wm = __reduce_max_sync(0xffffffffu, __float_as_uint(wj));
                    float ks = 0.f;
                    uint32_t kcs = 0;
                    if constexpr (kOut == kStats) {
                        ks = warp_sum(f2_lo(wsum) + f2_hi(wsum));
                        kcs = __reduce_add_sync(0xffffffffu, kc);
                    }
                    if ((tid & 31) == 0) {
                        atomicMax(&sm.wmax[acc][j], wm);
                        if constexpr (kOut == kStats) {
                            atomicAdd(&sm.ksum[acc][j], ks);
                            atomicAdd(&sm.kcnt[acc][j], kcs);
                        }
                    }
                }
            }
            if (!stop) stop = __all_sync(0xffffffffu, all_done());
        }
        contributor += cnt;
        const int ndone = __syncthreads_count(stop);
        if constexpr (kOut != kImage)
            for (uint32_t e = tid; e < cnt; e += NT) {
                const uint32_t wm = sm.wmax[acc][e];
                if (wm) {
                    const int id = __float_as_int(R[e].c.y);
                    if (a.out_point_weight) atomicMax(reinterpret_cast<unsigned*>(a.out_point_weight) + id, wm);
                    sm.wmax[acc][e] = 0;
                }
                if constexpr (kOut == kStats) {
                    a.kv_sum[range.x + b * kBatch + e] = sm.ksum[acc][e];
                    a.kv_cnt[range.x + b * kBatch + e] = sm.kcnt[acc][e];
                    sm.ksum[acc][e] = 0.f;
                    sm.kcnt[acc][e] = 0;
                }
            }
        if (ndone == NT) {
            // drain the copy still in flight before the buffers are reused or the CTA exits
            if (tid == 0 && b + 1 < nb)
                mbar_wait(&sm.bar[(g + 1) % kBufs], ((g + 1) / kBufs) & 1, err);
            if constexpr (kOut == kStats) {
                // pairs never reached contribute nothing
                for (uint32_t e = (b + 1) * kBatch + tid; e < n; e += NT) {
                    a.kv_sum[range.x + e] = 0.f;
                    a.kv_cnt[range.x + e] = 0;
                }
            }
            break;
        }
        if (b + 2 < nb) {
            if (tid == 0) {
                const int nbuf = (int)((g + 2) % kBufs);
                issue_batch(sm.rec[nbuf], &sm.bar[nbuf], recs, range.x + (b + 2) * kBatch,
                            min((uint32_t)kBatch, n - (b + 2) * kBatch));
            }
            issued = b + 3;
        }
    }
    gb += (uint32_t)issued;

#pragma unroll
    for (int k = 0; k < PPT; k++) {
        const int py = blk.py0 + 4 * k, q = k >> 1;
        auto half = [&](F2 v) { return (k & 1) ? f2_hi(v) : f2_lo(v); };
        if (px < W && py < H) {
            const int pix = W * py + px;
            const float T = fabsf(half(s.T[q]));
            a.final_T[pix] = T;
            a.n_contrib[pix] = s.last[k];
            a.out_color[pix] = __fmaf_rn(T, a.bg[0], half(s.C[q][0]));
            a.out_color[H * W + pix] = __fmaf_rn(T, a.bg[1], half(s.C[q][1]));
            a.out_color[2 * H * W + pix] = __fmaf_rn(T, a.bg[2], half(s.C[q][2]));
            if constexpr (kOut != kImage) {
                if (a.out_point_id) a.out_point_id[pix] = s.maxid[k];
                if (a.out_pw_pixel) a.out_pw_pixel[pix] = half(s.wmax[q]);
            }
        }
    }
}

template <int kBatch>
__device__ __forceinline__ void fwd_smem_init(FwdSmem<kBatch>& sm, int NT, bool stats_smem)
{
    for (int e = threadIdx.x; e < 2 * kBatch; e += NT) {
        (&sm.wmax[0][0])[e] = 0;
        if (stats_smem) {
            (&sm.ksum[0][0])[e] = 0.f;
            (&sm.kcnt[0][0])[e] = 0;
        }
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kBufs; i++) mbar_init(&sm.bar[i], 1);
        mbar_fence_init();
    }
    __syncthreads();
}

// Resident CTAs per SM the forward kernels are compiled for (a register cap of
// 65536 / (CTAs x threads)): 32 warps per SM at 2 and at 4 pixels per thread (64
// registers, at 4 with a few spilled bytes; a 64- or 128-record batch's shared
// memory then lets them fill; measured faster than 24 and 28 warps without or with
// fewer spills).
template <int PPT>
constexpr int fwd_min_ctas() { return PPT == 1 ? 3 : (PPT == 2 ? 8 : 16); }

template <int PPT, int kBatch, int kOut>
__global__ void __launch_bounds__(256 / PPT, fwd_min_ctas<PPT>())
    render_fwd_kernel(TileArgs a, uint32_t split_min, unsigned* err)
{
    extern __shared__ __align__(128) unsigned char fwd_dyn[];
    FwdSmem<kBatch>& sm = *reinterpret_cast<FwdSmem<kBatch>*>(fwd_dyn);
    fwd_smem_init(sm, 256 / PPT, kOut == kStats);
    uint32_t gb = 0;
    render_fwd_tile<PPT, kBatch, kOut>(sm, a, blockIdx.x, gb, split_min, err);
}

// Persistent multi-view forward: CTAs pop work items from one queue; item i is
// tile (i - begin[v]) of view v.  Views are laid out in the caller's order.
__device__ __forceinline__ int view_of(const uint32_t* __restrict__ begin, int nviews, uint32_t item)
{
    int v = 0;
    while (v + 1 < nviews && begin[v + 1] <= item) v++;
    return v;
}

template <int PPT, int kBatch>
__global__ void __launch_bounds__(256 / PPT, fwd_min_ctas<PPT>())
    render_fwd_multi_kernel(const TileArgs* __restrict__ views, const uint32_t* __restrict__ begin, int nviews,
                            uint32_t total, uint32_t* queue, uint32_t split_min, unsigned* err)
{
    // launched without the statistics sums (the batched path keeps no statistics)
    extern __shared__ __align__(128) unsigned char fwd_dyn[];
    FwdSmem<kBatch>& sm = *reinterpret_cast<FwdSmem<kBatch>*>(fwd_dyn);
    __shared__ uint32_t s_item;
    fwd_smem_init(sm, 256 / PPT, false);
    uint32_t gb = 0;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total) break;
        const int v = view_of(begin, nviews, item);
        const TileArgs& a = views[v];  // fields read where used, not held in registers
        // (from the device descriptors: a captured graph follows fgs_batch_set_view_outputs)
        if (a.out_point_weight || a.out_point_id || a.out_pw_pixel)
            render_fwd_tile<PPT, kBatch, kWeights>(sm, a, (int)(item - begin[v]), gb, split_min, err);
        else
            render_fwd_tile<PPT, kBatch, kImage>(sm, a, (int)(item - begin[v]), gb, split_min, err);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- long tiles in bands
// A tile with a long record list (dense small splats: distant LoD levels, a
// horizon) is the critical path of the one-CTA-per-tile render: its few warps
// walk every record while the rest of the GPU has finished.  Tiles with at
// least split_min records are rendered instead in bands of BW x BH pixels, one
// warp per band and four bands per CTA (a tile's 256 / (BW BH) bands spread over
// several SMs), longest tiles first.  The CTA stages the tile's records in
// chunks of two records per thread (plain coalesced loads; the next chunk is
// loaded into registers while the current one is composited), and each thread
// works out which bands its record can reach (band_mask), so a record is tested
// once per four bands instead of once per band, and a warp finds its band's
// records with one ballot per 32.  The
// warp composites them with the tile path's per-pixel functions; a band of
// fewer than 32 pixels evaluates several records per step (lane = slot * pixels
// + pixel) and the pixel's owner lane composites them in order.  Every pixel
// composites the same records in the same order with the same arithmetic as on
// the tile path.  Per record, a contributing lane folds its weight into the
// record's shared slot; the slots leave once per chunk (atomicMax into the
// per-Gaussian max weight, atomicAdd into the statistics, which are zeroed
// before the launch when on).
//
// Order: long tiles are binned by floor(log2(records)) (kLongBuckets bins of
// capacity `cap` each); the queue hands out the bins from the longest down.
constexpr int kLongBuckets = 32;

template <int BW, int BH>
struct LongTile {
    static_assert(BW * BH <= 32 && kTileX % BW == 0 && kTileY % BH == 0, "band shape");
    static constexpr int kPix = BW * BH;                   // pixels per band
    static constexpr int kPerRow = kTileX / BW;            // bands per row of the tile
    static constexpr int kRows = kTileY / BH;
    static constexpr int kBands = kPerRow * kRows;         // bands per tile
    static constexpr int kGroup = kBands < 4 ? kBands : 4; // bands (warps) per CTA
    static constexpr int kGroups = kBands / kGroup;        // CTAs per tile
    static constexpr int kThreads = 32 * kGroup;
    static constexpr int kPer = 2;                         // records each thread stages per chunk
    static constexpr int kChunk = kPer * kThreads;
    static constexpr int kSlots = 32 / kPix;               // records evaluated per step
};

template <int kChunk>
struct LongSmem {
    PairRecord rec[kChunk];
    uint32_t mask[kChunk];  // bands each record can reach
    uint32_t wmax[kChunk];  // per record: max weight over the tile's pixels
    float ksum[kChunk];     // statistics: weight sum and count over the tile's pixels
    uint32_t kcnt[kChunk];
};

// The bands of the tile at (tx0, ty0) that a record can reach.  The record
// reaches alpha >= 1/255 only inside the ellipse Q(d) = a dx^2 + 2 b dx dy +
// c dy^2 <= 2 ln(255 o); the test uses the axis-aligned box around Q(d) <= t,
// t = 1.01 * 2 ln(255 o) + 0.1, whose half-widths are sqrt(t c / det) and
// sqrt(t a / det) (det = a c - b^2), grown by 0.01 px.  With det >= 0.01 a c the
// per-pixel float evaluation of Q errs by under 5e-7 of a dx^2 + c dy^2 +
// 2|b dx dy|, which is at most 400 Q there, far inside the 1% margin; the fast
// log and divide err by less than the 0.1 absolute margin.  So a pixel outside
// the box gets alpha < 1/255 and is skipped by the per-pixel test anyway.  Band
// k of a row covers the pixel columns tx0 + k BW .. tx0 + k BW + BW - 1, so the
// box reaches it when mx - ex <= tx0 + k BW + BW - 1 and mx + ex >= tx0 + k BW
// (rows alike).  0 when the record cannot reach alpha >= 1/255 in the tile;
// every band for a conic the box does not cover (near-degenerate, not positive
// definite, not finite) and for a mean that is not finite.
template <int BW, int BH>
__device__ __forceinline__ uint32_t band_mask(const float4 ea, const float4 eb, float tx0, float ty0)
{
    using L = LongTile<BW, BH>;
    constexpr uint32_t kAll = L::kBands == 32 ? 0xffffffffu : ((1u << L::kBands) - 1u);
    const float mx = ea.x, my = ea.y, a = ea.z, b = ea.w, c = eb.x, o = eb.y;
    if (!(o >= 1.0f / 255.0f)) return 0u;
    const float det = a * c - b * b;
    if (!(a > 0.f && c > 0.f && det >= 0.01f * a * c) || !isfinite(mx) || !isfinite(my)) return kAll;
    const float t = 1.01f * (2.f * __logf(255.f * o)) + 0.1f;
    const float s = __fdividef(t, det);
    const float ex = sqrtf(s * c) + 0.01f, ey = sqrtf(s * a) + 0.01f;
    const float lo_x = (mx - ex - tx0 - (BW - 1)) * (1.f / BW), hi_x = (mx + ex - tx0) * (1.f / BW);
    const float lo_y = (my - ey - ty0 - (BH - 1)) * (1.f / BH), hi_y = (my + ey - ty0) * (1.f / BH);
    const int c0 = (int)ceilf(fmaxf(lo_x, 0.f)), c1 = (int)floorf(fminf(hi_x, (float)(L::kPerRow - 1)));
    const int r0 = (int)ceilf(fmaxf(lo_y, 0.f)), r1 = (int)floorf(fminf(hi_y, (float)(L::kRows - 1)));
    if (c0 > c1 || r0 > r1) return 0u;
    const uint32_t cols = ((2u << (c1 - c0)) - 1u) << c0;
    uint32_t m = 0u;
    for (int r = r0; r <= r1; r++) m |= cols << (r * L::kPerRow);
    return m;
}

template <int kChunk>
__device__ __forceinline__ void long_fold(LongSmem<kChunk>& sm, uint32_t j, float w, bool stats)
{
    if (w > 0.f) {
        atomicMax(&sm.wmax[j], __float_as_uint(w));
        if (stats) {
            atomicAdd(&sm.ksum[j], w);
            atomicAdd(&sm.kcnt[j], 1u);
        }
    }
}

// Bands group * kGroup .. group * kGroup + kGroup - 1 of one long tile by one
// CTA; warp w renders band group * kGroup + w.
template <int BW, int BH>
__device__ __forceinline__ void render_long_tile(LongSmem<LongTile<BW, BH>::kChunk>& sm, const TileArgs& a,
                                                 int tile, int group)
{
    using L = LongTile<BW, BH>;
    constexpr int kPix = L::kPix, kSlots = L::kSlots, kPer = L::kPer, kChunk = L::kChunk;
    const int tid = threadIdx.x, lane = tid & 31, band = group * L::kGroup + (tid >> 5);
    const int W = a.W, H = a.H;
    const int gx = (W + kTileX - 1) / kTileX;
    const int bx = tile % gx, by = tile / gx;
    const float tx0 = (float)(bx * kTileX), ty0 = (float)(by * kTileY);
    const int ox = bx * kTileX + (band % L::kPerRow) * BW, oy = by * kTileY + (band / L::kPerRow) * BH;
    const int pix_lane = lane % kPix, slot = lane / kPix;
    const bool mine = lane < kPix;  // the pixel's owner lane keeps its state
    const int px = ox + pix_lane % BW, py = oy + pix_lane / BW;
    const uint2 range = a.ranges[tile];
    const uint32_t n = range.y - range.x;
    const bool stats = a.kv_sum != nullptr;
    const PairRecord* recs = a.recs + range.x;
    const float pxf = (float)px, pyf = (float)py;
    float T = 1.0f, C[3] = {0.f, 0.f, 0.f}, wmax = 0.f;
    uint32_t last = 0;
    int maxid = -1;
    bool done = !(mine && px < W && py < H);

    // A contributing record's per-chunk sums leave through global atomics; slot i
    // of chunk cbase is flushed by the thread that staged it, before it restages
    // the slot (no other thread touches the slot between the barriers around the
    // compositing).
    auto flush = [&](uint32_t cbase) {
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int i = q * L::kThreads + tid;
            const uint32_t e = cbase + (uint32_t)i;
            if (e >= n) continue;
            const uint32_t wm = sm.wmax[i];
            if (wm && a.out_point_weight)
                atomicMax(reinterpret_cast<unsigned*>(a.out_point_weight) + __float_as_int(sm.rec[i].c.y), wm);
            if (stats && sm.kcnt[i]) {
                atomicAdd(a.kv_sum + range.x + e, sm.ksum[i]);
                atomicAdd(a.kv_cnt + range.x + e, sm.kcnt[i]);
            }
        }
    };
    PairRecord nxt[kPer];
#pragma unroll
    for (int q = 0; q < kPer; q++)
        if ((uint32_t)(q * L::kThreads + tid) < n) nxt[q] = recs[q * L::kThreads + tid];
    uint32_t last_c = 0;
    bool pending = false;
    for (uint32_t c0 = 0; c0 < n; c0 += kChunk) {
        if (pending) flush(last_c);
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int i = q * L::kThreads + tid;
            const uint32_t e = c0 + (uint32_t)i;
            const bool have = e < n;
            if (have) sm.rec[i] = nxt[q];
            sm.mask[i] = have ? band_mask<BW, BH>(nxt[q].a, nxt[q].b, tx0, ty0) : 0u;
            sm.wmax[i] = 0u;
            if (stats) {
                sm.ksum[i] = 0.f;
                sm.kcnt[i] = 0u;
            }
            if (e + kChunk < n) nxt[q] = recs[e + kChunk];  // in flight while this chunk is composited
        }
        __syncthreads();
        for (int k = 0; k < kChunk / 32 && !__all_sync(0xffffffffu, done); k++) {
            uint32_t live = __ballot_sync(0xffffffffu, (sm.mask[k * 32 + lane] >> band) & 1u);
            const PairRecord* R = sm.rec + k * 32;
            const uint32_t k0 = c0 + (uint32_t)(k * 32);  // tile position of R[0]
            if constexpr (kSlots == 1) {
                while (live) {
                    const uint32_t j1 = (uint32_t)(__ffs(live) - 1);
                    live &= live - 1;
                    const bool two = live != 0;
                    const uint32_t j2 = two ? (uint32_t)(__ffs(live) - 1) : j1;
                    if (two) live &= live - 1;
                    const float4 ra1 = R[j1].a, rb1 = R[j1].b, ra2 = R[j2].a, rb2 = R[j2].b;
                    const float al1 = done ? 0.f : fwd_alpha(ra1, rb1, pxf, pyf);
                    const float al2 = (done || !two) ? 0.f : fwd_alpha(ra2, rb2, pxf, pyf);
                    long_fold(sm, k * 32 + j1,
                              fwd_accumulate(al1, rb1, R[j1], k0 + j1 + 1, T, C, wmax, maxid, last, done), stats);
                    long_fold(sm, k * 32 + j2,
                              fwd_accumulate(al2, rb2, R[j2], k0 + j2 + 1, T, C, wmax, maxid, last, done), stats);
                }
            } else {
                while (live) {
                    // the next kSlots live records, in order (32: none); lanes of slot s
                    // evaluate record js[s] at their pixel
                    uint32_t js[kSlots];
                    uint32_t mj = 32u;
#pragma unroll
                    for (int s = 0; s < kSlots; s++) {
                        js[s] = live ? (uint32_t)(__ffs(live) - 1) : 32u;
                        live &= live - 1;
                        if (s == slot) mj = js[s];
                    }
                    const bool pdone = __shfl_sync(0xffffffffu, done, pix_lane);
                    const float al = (mj < 32u && !pdone) ? fwd_alpha(R[mj].a, R[mj].b, pxf, pyf) : 0.f;
#pragma unroll
                    for (int s = 0; s < kSlots; s++) {
                        const float as = __shfl_sync(0xffffffffu, al, s * kPix + pix_lane);
                        const uint32_t j = js[s];
                        if (j < 32u)
                            long_fold(sm, k * 32 + j,
                                      fwd_accumulate(as, R[j].b, R[j], k0 + j + 1, T, C, wmax, maxid, last, done),
                                      stats);
                    }
                }
            }
        }
        last_c = c0;
        pending = true;
        // every pixel of this band group done: no later record can contribute (also
        // the barrier before the next chunk's staging)
        if (__syncthreads_and(done)) break;
    }
    if (pending) flush(last_c);
    if (mine && px < W && py < H) {
        const int pix = W * py + px;
        a.final_T[pix] = T;
        a.n_contrib[pix] = last;
        a.out_color[pix] = __fmaf_rn(T, a.bg[0], C[0]);
        a.out_color[H * W + pix] = __fmaf_rn(T, a.bg[1], C[1]);
        a.out_color[2 * H * W + pix] = __fmaf_rn(T, a.bg[2], C[2]);
        if (a.out_point_id) a.out_point_id[pix] = maxid;
        if (a.out_pw_pixel) a.out_pw_pixel[pix] = wmax;
    }
}

__device__ __forceinline__ void long_tile_push(uint32_t n, uint32_t id, uint32_t cap, uint32_t* __restrict__ list,
                                               uint32_t* __restrict__ ctr)
{
    const int b = 31 - __clz(n);
    const uint32_t slot = atomicAdd(ctr + 2 + b, 1u);
    list[(size_t)b * cap + slot] = id;
    atomicAdd(ctr, 1u);
}

// The long tiles of one view (ids are tiles) or of a multi-view batch (ids are
// global work items, mapped to (view, tile) by begin[]).  ctr: [0] long tiles,
// [1] tile queue, [2 + b] tiles in bin b.
__global__ void long_tiles_kernel(const uint2* __restrict__ ranges, uint32_t num_tiles, uint32_t split_min,
                                  uint32_t* __restrict__ list, uint32_t* __restrict__ ctr)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= num_tiles) return;
    const uint2 r = ranges[t];
    if (r.y - r.x >= split_min) long_tile_push(r.y - r.x, t, num_tiles, list, ctr);
}

__global__ void long_tiles_multi_kernel(const TileArgs* __restrict__ views, const uint32_t* __restrict__ begin,
                                        int nviews, uint32_t total, uint32_t split_min, uint32_t* __restrict__ list,
                                        uint32_t* __restrict__ ctr)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int v = view_of(begin, nviews, i);
    const uint2 r = views[v].ranges[i - begin[v]];
    if (r.y - r.x >= split_min) long_tile_push(r.y - r.x, i, total, list, ctr);
}

// The next (long tile, band group) for this CTA (thread 0), longest bins first.
// False when the queue is empty.
template <int kGroups>
__device__ __forceinline__ bool next_long_tile(uint32_t* ctr, const uint32_t* __restrict__ list, uint32_t cap,
                                               uint32_t& id, int& group)
{
    const uint32_t item = atomicAdd(ctr + 1, 1u);
    if (item >= *(volatile uint32_t*)ctr * kGroups) return false;
    uint32_t r = item / kGroups;
    group = (int)(item % kGroups);
    for (int b = kLongBuckets - 1; b >= 0; b--) {
        const uint32_t c = *(volatile uint32_t*)(ctr + 2 + b);
        if (r < c) {
            id = list[(size_t)b * cap + r];
            return true;
        }
        r -= c;
    }
    return false;
}

template <int BW, int BH>
__device__ __forceinline__ void long_tile_loop(unsigned char* dyn, const TileArgs* __restrict__ views,
                                               const uint32_t* __restrict__ begin, int nviews,
                                               const uint32_t* __restrict__ list, uint32_t* ctr, uint32_t cap)
{
    auto& sm = *reinterpret_cast<LongSmem<LongTile<BW, BH>::kChunk>*>(dyn);
    __shared__ uint32_t s_id;
    __shared__ int s_ok, s_group;
    for (;;) {
        if (threadIdx.x == 0) {
            uint32_t id = 0;
            int group = 0;
            s_ok = next_long_tile<LongTile<BW, BH>::kGroups>(ctr, list, cap, id, group);
            s_id = id;
            s_group = group;
        }
        __syncthreads();
        if (!s_ok) break;
        const uint32_t id = s_id;
        const int v = begin ? view_of(begin, nviews, id) : 0;
        render_long_tile<BW, BH>(sm, views[v], (int)(begin ? id - begin[v] : id), s_group);
        __syncthreads();  // s_id / s_group / s_ok are rewritten for the next item
    }
}

template <int BW, int BH>
__global__ void __launch_bounds__(LongTile<BW, BH>::kThreads)
    render_fwd_long_kernel(TileArgs a, const uint32_t* __restrict__ list, uint32_t* ctr, uint32_t cap)
{
    extern __shared__ __align__(128) unsigned char long_dyn[];
    long_tile_loop<BW, BH>(long_dyn, &a, nullptr, 1, list, ctr, cap);
}

template <int BW, int BH>
__global__ void __launch_bounds__(LongTile<BW, BH>::kThreads)
    render_fwd_long_multi_kernel(const TileArgs* __restrict__ views, const uint32_t* __restrict__ begin, int nviews,
                                 const uint32_t* __restrict__ list, uint32_t* ctr, uint32_t cap)
{
    extern __shared__ __align__(128) unsigned char long_dyn[];
    long_tile_loop<BW, BH>(long_dyn, views, begin, nviews, list, ctr, cap);
}

// ---------------------------------------------------------------- long tiles by quads
// The launch rule's form of a long tile: a CTA renders a unit of 8x4 pixels, four warps
// with a 4x2 band each, and stages only the records whose block_mask has the unit's block.
// What bounds a tile of thousands of small splats is staging, not compositing: with
// every record staged and tested by each of the tile's eight CTAs, two thirds of the
// time went there.  Here a CTA reads the 4-byte masks of kUnitIn records (the next ones
// in flight meanwhile), compacts the survivors (about a seventh) in order, loads only
// those records and tests only those against the bands.  Per pixel the same records in
// the same order with the same arithmetic as on the tile path.  8M-node LoD views at
// 1080p with 2.7M / 6.4M / 8.5M pairs: 0.60 / 1.08 / 1.06 ms with masks of 8x8 quads (a
// quarter survived; the 8x4 blocks take another tenth off: 462 -> 418 us of a smaller view);
// in bands that stage every record 0.78 / 1.42 / 1.36; one CTA per tile 1.66 / 2.63 / 5.59.
constexpr int kUnitIn = 512, kUnitRecs = 256, kUnits = 8, kUnitThreads = 128;

struct UnitSmem {
    PairRecord rec[kUnitRecs];
    uint32_t mask[kUnitRecs];  // the unit's bands each record can reach (bit = warp)
    uint32_t wmax[kUnitRecs];  // as in LongSmem
    float ksum[kUnitRecs];
    uint32_t kcnt[kUnitRecs];
    uint16_t idx[kUnitIn];     // survivors of the kUnitIn records
    uint32_t cnt[kUnitIn / 32];
};

__device__ __forceinline__ void render_unit(UnitSmem& sm, const TileArgs& a, int tile, int unit)
{
    constexpr int kPix = 8, kSlots = 4, kPer = kUnitIn / kUnitThreads;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = a.W, H = a.H;
    const int gx = (W + kTileX - 1) / kTileX;
    const int bx = tile % gx, by = tile / gx, ux = unit & 1, uy = unit >> 1;
    const float tx0 = (float)(bx * kTileX), ty0 = (float)(by * kTileY);
    const int band0 = 8 * uy + 2 * ux;  // the unit's bands in band_mask<4, 2>: band0 + {0, 1, 4, 5}
    const int mbit = 2 * uy + ux;  // the unit's bit in a record's block_mask
    const int pix_lane = lane % kPix, slot = lane / kPix;
    const int px = bx * kTileX + 8 * ux + 4 * (warp & 1) + pix_lane % 4;
    const int py = by * kTileY + 4 * uy + 2 * (warp >> 1) + pix_lane / 4;
    const bool mine = lane < kPix;  // the pixel's owner lane keeps its state
    const uint2 range = a.ranges[tile];
    const uint32_t n = range.y - range.x;
    const bool stats = a.kv_sum != nullptr;
    const PairRecord* recs = a.recs + range.x;
    const float pxf = (float)px, pyf = (float)py;
    float T = 1.0f, C[3] = {0.f, 0.f, 0.f}, wmax = 0.f;
    uint32_t last = 0;
    int maxid = -1;
    bool done = !(mine && px < W && py < H);
    const unsigned lt = (1u << lane) - 1u;

    uint32_t m[kPer];
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        const uint32_t e = (uint32_t)(i * kUnitThreads + tid);
        m[i] = e < n ? __float_as_uint(__ldg(&recs[e].c.z)) : 0u;
    }
    bool all_done = false;
    for (uint32_t c0 = 0; c0 < n && !all_done; c0 += kUnitIn) {
        uint32_t b[kPer];
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            b[i] = __ballot_sync(0xffffffffu, (m[i] >> mbit) & 1u);
            if (lane == 0) sm.cnt[i * (kUnitThreads / 32) + warp] = __popc(b[i]);
        }
#pragma unroll
        for (int i = 0; i < kPer; i++) {  // the next masks, in flight while these records are composited
            const uint32_t e = c0 + kUnitIn + (uint32_t)(i * kUnitThreads + tid);
            m[i] = e < n ? __float_as_uint(__ldg(&recs[e].c.z)) : 0u;
        }
        __syncthreads();
        uint32_t total = 0;
#pragma unroll
        for (int i = 0; i < kPer; i++)
#pragma unroll
            for (int w = 0; w < kUnitThreads / 32; w++) {
                if (w == warp && ((b[i] >> lane) & 1u))
                    sm.idx[total + __popc(b[i] & lt)] = (uint16_t)(i * kUnitThreads + tid);
                total += sm.cnt[i * (kUnitThreads / 32) + w];
            }
        __syncthreads();
        for (uint32_t s0 = 0; s0 < total && !all_done; s0 += kUnitRecs) {
            const uint32_t cnt = min((uint32_t)kUnitRecs, total - s0);
#pragma unroll
            for (int q = 0; q < kUnitRecs / kUnitThreads; q++) {
                const int e = q * kUnitThreads + tid;
                uint32_t bits = 0;
                if ((uint32_t)e < cnt) {
                    const PairRecord r = recs[c0 + sm.idx[s0 + e]];
                    const uint32_t all = band_mask<4, 2>(r.a, r.b, tx0, ty0) >> band0;
                    bits = (all & 3u) | ((all >> 2) & 12u);
                    sm.rec[e] = r;
                }
                sm.mask[e] = bits;
                sm.wmax[e] = 0u;
                if (stats) {
                    sm.ksum[e] = 0.f;
                    sm.kcnt[e] = 0u;
                }
            }
            __syncthreads();
            for (uint32_t k = 0; k < cnt && !__all_sync(0xffffffffu, done); k += 32) {
                uint32_t live = __ballot_sync(0xffffffffu, (sm.mask[k + lane] >> warp) & 1u);
                const PairRecord* R = sm.rec + k;
                while (live) {
                    // the next kSlots live records, in order (32: none); lanes of slot s
                    // evaluate record js[s] at their pixel
                    uint32_t js[kSlots];
                    uint32_t mj = 32u;
#pragma unroll
                    for (int s = 0; s < kSlots; s++) {
                        js[s] = live ? (uint32_t)(__ffs(live) - 1) : 32u;
                        live &= live - 1;
                        if (s == slot) mj = js[s];
                    }
                    const bool pdone = __shfl_sync(0xffffffffu, done, pix_lane);
                    const float al = (mj < 32u && !pdone) ? fwd_alpha(R[mj].a, R[mj].b, pxf, pyf) : 0.f;
#pragma unroll
                    for (int s = 0; s < kSlots; s++) {
                        const float as = __shfl_sync(0xffffffffu, al, s * kPix + pix_lane);
                        const uint32_t j = js[s];
                        if (j < 32u) {
                            const float w = fwd_accumulate(as, R[j].b, R[j], c0 + sm.idx[s0 + k + j] + 1, T, C, wmax,
                                                           maxid, last, done);
                            if (w > 0.f) {
                                atomicMax(&sm.wmax[k + j], __float_as_uint(w));
                                if (stats) {
                                    atomicAdd(&sm.ksum[k + j], w);
                                    atomicAdd(&sm.kcnt[k + j], 1u);
                                }
                            }
                        }
                    }
                }
            }
            // (every pixel of this unit done: no later record can contribute)
            all_done = __syncthreads_and(done);
#pragma unroll
            for (int q = 0; q < kUnitRecs / kUnitThreads; q++) {
                const uint32_t e = (uint32_t)(q * kUnitThreads + tid);
                const uint32_t wm = e < cnt ? sm.wmax[e] : 0u;
                if (!wm) continue;
                if (a.out_point_weight)
                    atomicMax(reinterpret_cast<unsigned*>(a.out_point_weight) + __float_as_int(sm.rec[e].c.y), wm);
                if (stats) {
                    const uint32_t at = range.x + c0 + sm.idx[s0 + e];
                    atomicAdd(a.kv_sum + at, sm.ksum[e]);
                    atomicAdd(a.kv_cnt + at, sm.kcnt[e]);
                }
            }
        }
    }
    if (mine && px < W && py < H) {
        const int pix = W * py + px;
        a.final_T[pix] = T;
        a.n_contrib[pix] = last;
        a.out_color[pix] = __fmaf_rn(T, a.bg[0], C[0]);
        a.out_color[H * W + pix] = __fmaf_rn(T, a.bg[1], C[1]);
        a.out_color[2 * H * W + pix] = __fmaf_rn(T, a.bg[2], C[2]);
        if (a.out_point_id) a.out_point_id[pix] = maxid;
        if (a.out_pw_pixel) a.out_pw_pixel[pix] = wmax;
    }
}

// Units of long tiles from the queue until it is empty (all threads of the CTA).
__device__ __forceinline__ void unit_loop(unsigned char* dyn, const TileArgs* __restrict__ views,
                                          const uint32_t* __restrict__ begin, int nviews,
                                          const uint32_t* __restrict__ list, uint32_t* ctr, uint32_t cap)
{
    UnitSmem& sm = *reinterpret_cast<UnitSmem*>(dyn);
    __shared__ uint32_t s_id;
    __shared__ int s_ok, s_unit;
    for (;;) {
        if (threadIdx.x == 0) {
            uint32_t id = 0;
            int unit = 0;
            s_ok = next_long_tile<kUnits>(ctr, list, cap, id, unit);
            s_id = id;
            s_unit = unit;
        }
        __syncthreads();
        if (!s_ok) break;
        const uint32_t id = s_id;
        const int v = begin ? view_of(begin, nviews, id) : 0;
        render_unit(sm, views[v], (int)(begin ? id - begin[v] : id), s_unit);
        __syncthreads();  // s_id / s_unit / s_ok are rewritten for the next item
    }
}

// ---------------------------------------------------------------- the launch rule's forward
// Used until a caller sets a shape or a split: 2 pixels per lane and 128-record batches,
// and the long tiles (listed by place_kernel) in units by the same launch: its first
// blocks, one resident set, take them from the queue before the tiles' own blocks start,
// so a view without long tiles pays for no second kernel and no listing pass (10 us of
// 300), only for blocks that leave at once.  Against the best of the nine shapes without
// long tiles, in us: a 1237x823 view of 300K Gaussians 199 / 194, one of 2M at 1080p 296 / 289
// (4 pixels, 64 records), sixteen of these 3679 / 3486 (4, 64), six of mixed sizes 859 / 838, four
// of 1600x900 692 / 677 (4, 64); 10K Gaussians at 256x256 53 / 35 (1, 256: more warps for few tiles).
// In a batch the units share the tiles' registers: with every output per view, not the image
// alone, sixteen 1080p views take 5365 against 4880 in the same shape without them, mixed sizes
// 3054 / 2722; a tuned shape gets that back.  LoD views of 5.4M pairs 1.50 ms, 10.1 without long
// tiles, 1.58 in the best bands.
constexpr int kRulePpt = 2, kRuleBatch = 128;
static_assert(kUnitThreads == 256 / kRulePpt, "one block size for tiles and units");
static_assert(sizeof(UnitSmem) <= offsetof(FwdSmem<kRuleBatch>, ksum), "shared memory");

template <int kOut>
__global__ void __launch_bounds__(256 / kRulePpt, fwd_min_ctas<kRulePpt>())
    render_fwd_rule_kernel(TileArgs a, int long_ctas, const uint32_t* __restrict__ list, uint32_t* ctr, uint32_t cap,
                           unsigned* err)
{
    extern __shared__ __align__(128) unsigned char fwd_dyn[];
    if ((int)blockIdx.x < long_ctas) {
        if (*(volatile uint32_t*)ctr) unit_loop(fwd_dyn, &a, nullptr, 1, list, ctr, cap);
        return;
    }
    FwdSmem<kRuleBatch>& sm = *reinterpret_cast<FwdSmem<kRuleBatch>*>(fwd_dyn);
    fwd_smem_init(sm, 256 / kRulePpt, kOut == kStats);
    uint32_t gb = 0;
    render_fwd_tile<kRulePpt, kRuleBatch, kOut>(sm, a, (int)blockIdx.x - long_ctas, gb, auto_split_min(a.totals), err);
}

__global__ void __launch_bounds__(256 / kRulePpt, fwd_min_ctas<kRulePpt>())
    render_fwd_multi_rule_kernel(const TileArgs* __restrict__ views, const uint32_t* __restrict__ begin, int nviews,
                                 uint32_t total, uint32_t* queue, const uint32_t* __restrict__ list, uint32_t* ctr,
                                 unsigned* err)
{
    extern __shared__ __align__(128) unsigned char fwd_dyn[];
    if (*(volatile uint32_t*)ctr) {
        unit_loop(fwd_dyn, views, begin, nviews, list, ctr, total);
        __syncthreads();
    }
    FwdSmem<kRuleBatch>& sm = *reinterpret_cast<FwdSmem<kRuleBatch>*>(fwd_dyn);
    __shared__ uint32_t s_item;
    fwd_smem_init(sm, 256 / kRulePpt, false);
    uint32_t gb = 0;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total) break;
        const int v = view_of(begin, nviews, item);
        const TileArgs& a = views[v];  // fields read where used, not held in registers
        const uint32_t split = auto_split_min(a.totals);
        // (from the device descriptors: a captured graph follows fgs_batch_set_view_outputs)
        if (a.out_point_weight || a.out_point_id || a.out_pw_pixel)
            render_fwd_tile<kRulePpt, kRuleBatch, kWeights>(sm, a, (int)(item - begin[v]), gb, split, err);
        else
            render_fwd_tile<kRulePpt, kRuleBatch, kImage>(sm, a, (int)(item - begin[v]), gb, split, err);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- backward
// The backward's pixels: a warp owns PPT / 2 strips of 16x4 (half a strip at one pixel per
// lane), lane (x, y) = (lane & 15, lane >> 4) with the rows 2 y and 2 y + 1 of each strip, so
// that all of a lane's pixels share a column.  In pairs (k = 2q, 2q + 1: a strip's).
// The reference's accum_rec recurrence (the colour composited behind the current Gaussian,
// backward.cu:513-520) enters dL/dalpha only through its dot product with dL/dpixel, so a
// pixel carries that dot product (acc): one value instead of six.  bgT: the numerator
// -T_final (bg . dL/dpixel) of the background term of dL/dalpha.
template <int NP>
struct BwdPixels {
    F2 T[NP], acc[NP], d[NP][3], bgT[NP], npy[NP];
    F2 d01[NP][2];  // channels 0 and 1 of either pixel
    uint32_t last[2 * NP];
};

// A record's nine sums over a lane's pixels of one strip, with w = G dL/dalpha:
// alpha T dL/dpixel (channels 0, 1), w dx, w dy, w dx dx, w dx dy, w dy dy, w and
// alpha T dL/dpixel (channel 2): neighbours come from one packed instruction.  Pixels are
// added one after the other, lanes by warp_transpose_sum9 and strips as (0 + 1) + (2 + 3),
// at two and at four pixels per lane alike (one pixel per lane adds half strips in four
// slots, in turn): a training step carries the last bits of these sums on to the
// next one, where they decide comparisons.

// 1 / x for x in [0.01, 1], with the bits of __fdividef(1, x) there, which spends its time on
// guarding the ends of the range.
__device__ __forceinline__ float rcp_unit(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// One record on one pixel, with branches (see fwd_pixel_step for when).
template <bool kConsistent>
__device__ __forceinline__ bool bwd_pixel_step(const float4 ra, const float4 rb, float c2, float pxf, float pyf,
                                               bool before_last, float& T, float& acc, float d0, float d1, float d2,
                                               float bgT, float (&g)[9])
{
    if (!before_last) return false;
    const float dx = ra.x - pxf, dy = ra.y - pyf;
    const float qf = __fmaf_rn(__fmul_rn(ra.z, dx), dx, __fmul_rn(__fmul_rn(rb.x, dy), dy));
    const float power = __fmaf_rn(-0.5f, qf, -__fmul_rn(__fmul_rn(ra.w, dx), dy));
    if (power > 0.0f) return false;
    const float G = expf(power);
    const float oG = __fmul_rn(rb.y, G);
    const float alpha = fminf(0.99f, oG);
    if (alpha < 1.0f / 255.0f) return false;
    const float inv = rcp_unit(1.f - alpha);
    T = __fmul_rn(T, inv);
    const float wc = __fmul_rn(alpha, T);
    g[0] = __fmaf_rn(wc, d0, g[0]);
    g[1] = __fmaf_rn(wc, d1, g[1]);
    g[8] = __fmaf_rn(wc, d2, g[8]);
    const float cdot = __fmaf_rn(c2, d2, __fmaf_rn(rb.z, d0, __fmul_rn(rb.w, d1)));
    const float diff = cdot - acc;
    float dL_dalpha = __fmul_rn(diff, T);
    if (bgT != 0.f) dL_dalpha = __fmaf_rn(bgT, inv, dL_dalpha);
    if (kConsistent && oG > 0.99f) dL_dalpha = 0.f;
    acc = __fmaf_rn(alpha, diff, acc);
    const float w = __fmul_rn(G, dL_dalpha), u = __fmul_rn(w, dx), v = __fmul_rn(w, dy);
    g[2] = __fadd_rn(g[2], u);
    g[3] = __fadd_rn(g[3], v);
    g[4] = __fmaf_rn(u, dx, g[4]);
    g[5] = __fmaf_rn(u, dy, g[5]);
    g[6] = __fmaf_rn(v, dy, g[6]);
    g[7] = __fadd_rn(g[7], w);
    return true;
}

// One record on one pair of pixels, without branches: a pixel the record does not
// reach (or that ended before it) takes alpha 0, which leaves its T and acc as they are,
// and w 0.  G and alpha are formed with the forward's operations and rounding, so this
// pass skips exactly the (pixel, record) pairs the forward skipped.  All values are
// below 1e15 here (kWild records and warps take bwd_pixel_step), so no 0 * inf arises.
template <bool kConsistent, int NP>
__device__ __forceinline__ bool bwd_pair_step(BwdPixels<NP>& s, int q, const float4 ra, const float4 rb, float c2,
                                              float dx, float sx, float nbx, uint32_t contributor, float (&g)[9])
{
    const F2 dy = f2_add(f2(ra.y), s.npy[q]);
    const F2 qf = f2_fma(f2(sx), f2(dx), f2_mul(f2_mul(f2(rb.x), dy), dy));
    const F2 power = f2_fma(f2(-0.5f), qf, f2_mul(f2(nbx), dy));
    const F2 G = f2(expf(f2_lo(power)), expf(f2_hi(power)));
    const F2 oG = f2_mul(f2(rb.y), G);
    const float a0 = fminf(0.99f, f2_lo(oG)), a1 = fminf(0.99f, f2_hi(oG));
    const bool ok0 = contributor < s.last[2 * q] && !(f2_lo(power) > 0.f) && !(a0 < 1.0f / 255.0f);
    const bool ok1 = contributor < s.last[2 * q + 1] && !(f2_hi(power) > 0.f) && !(a1 < 1.0f / 255.0f);
    const F2 alpha = f2(ok0 ? a0 : 0.f, ok1 ? a1 : 0.f);
    const F2 rem = f2_fma(alpha, f2(-1.f), f2(1.f));
    // (fast reciprocal: 1 - alpha >= 0.01)
    const F2 inv = f2(rcp_unit(f2_lo(rem)), rcp_unit(f2_hi(rem)));
    s.T[q] = f2_mul(s.T[q], inv);  // transmittance before this Gaussian
    const F2 wc = f2_mul(alpha, s.T[q]);
    const F2 c01 = f2_fma(f2(f2_hi(wc)), s.d01[q][1], f2_mul(f2(f2_lo(wc)), s.d01[q][0]));
    g[0] = f2_lo(c01);
    g[1] = f2_hi(c01);
    g[8] = __fmaf_rn(f2_hi(wc), f2_hi(s.d[q][2]), __fmul_rn(f2_lo(wc), f2_lo(s.d[q][2])));
    const F2 cdot = f2_fma(f2(c2), s.d[q][2], f2_fma(f2(rb.z), s.d[q][0], f2_mul(f2(rb.w), s.d[q][1])));
    const F2 diff = f2_fma(s.acc[q], f2(-1.f), cdot);
    s.acc[q] = f2_fma(alpha, diff, s.acc[q]);
    const F2 dL_dalpha = f2_fma(s.bgT[q], inv, f2_mul(diff, s.T[q]));
    const F2 Gd = f2_mul(G, dL_dalpha);
    const float w0 = ok0 && !(kConsistent && f2_lo(oG) > 0.99f) ? f2_lo(Gd) : 0.f;
    const float w1 = ok1 && !(kConsistent && f2_hi(oG) > 0.99f) ? f2_hi(Gd) : 0.f;
    const F2 xy0 = f2(dx, f2_lo(dy)), xy1 = f2(dx, f2_hi(dy));
    const F2 uv0 = f2_mul(f2(w0), xy0), uv1 = f2_mul(f2(w1), xy1);
    const F2 uv = f2_add(uv0, uv1);
    const F2 uxy = f2_fma(f2(f2_lo(uv1)), xy1, f2_mul(f2(f2_lo(uv0)), xy0));
    g[2] = f2_lo(uv);
    g[3] = f2_hi(uv);
    g[4] = f2_lo(uxy);
    g[5] = f2_hi(uxy);
    g[6] = __fmaf_rn(f2_hi(uv1), f2_hi(dy), __fmul_rn(f2_hi(uv0), f2_lo(dy)));
    g[7] = __fadd_rn(w0, w1);
    return ok0 || ok1;
}

// Adds the warp's `count` pending steps over the lanes and into `acc`, in the order of
// warp_transpose_sum9 (lanes 16 apart first, then 8, 4, 2, 1): eight lanes per step, of which
// each takes four sums of every fourth lane (128-bit loads, packed adds) through the first
// three levels; two exchanges halve the four sums a lane still holds.  The two strips of one
// record are added to each other first.  kAtomic: two warps share a slot.
// What bounds the backward is instructions issued (77% of the slots; about 125 per step of 32
// lanes x 2 pixels).  A butterfly over one step's nine sums takes 12 shuffles and 46
// instructions, this about 20 with the stores: with it, and with warps that do not wait for
// one another at each batch, the backward of a 1237x823 view of 300K Gaussians takes 263 us
// (308 before), of 2M at 1080p 465 (476), of 16 such views 7.07 ms (7.25), of six smaller
// views 1.70 ms (2.03), of 10K at 256x256 50 us (62).  (The single-view figures hold the zeroing of
// the gradient buffers, whose shares each thread then still divided for: 415 us at 2M without.)  Two steps at a time, in half the shared
// memory and with one more CTA per SM: 491 us at 2M.
template <bool kAtomic>
__device__ __forceinline__ void add_step_sums(const StepSums& u, float (*acc)[9], int count)
{
    const int lane = threadIdx.x & 31, step = lane >> 3, r = lane & 3, x = lane & 4;
    __syncwarp();
    const ulonglong2* A = reinterpret_cast<const ulonglong2*>(u.step[step].a[x >> 2]);
    F2 v[4][2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const ulonglong2 p = A[(r + 4 * k) ^ x], q = A[(r + 4 * k + 16) ^ x];
        v[k][0] = f2_add(p.x, q.x);
        v[k][1] = f2_add(p.y, q.y);
    }
    const float* B = u.step[step].b + (lane & 7);
    float z = (B[0] + B[16]) + (B[8] + B[24]);
    const int rec = u.rec[step];
#pragma unroll
    for (int c = 0; c < 2; c++) v[0][c] = f2_add(f2_add(v[0][c], v[2][c]), f2_add(v[1][c], v[3][c]));
    const float v0 = f2_lo(v[0][0]), v1 = f2_hi(v[0][0]), v2 = f2_lo(v[0][1]), v3 = f2_hi(v[0][1]);
    const bool b2 = r & 2, b1 = r & 1;
    const float s0 = (b2 ? v2 : v0) + __shfl_xor_sync(0xffffffffu, b2 ? v0 : v2, 2);
    const float s1 = (b2 ? v3 : v1) + __shfl_xor_sync(0xffffffffu, b2 ? v1 : v3, 2);
    float tot = (b1 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, b1 ? s0 : s1, 1);  // sum number lane & 7
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    bool on = step < count;
    if constexpr (!kAtomic) {
        const int after = __shfl_down_sync(0xffffffffu, rec, 8), before = __shfl_up_sync(0xffffffffu, rec, 8);
        const float t2 = __shfl_down_sync(0xffffffffu, tot, 8), z2 = __shfl_down_sync(0xffffffffu, z, 8);
        if (step + 1 < count && after == rec) {
            tot += t2;
            z += z2;
        }
        if (step > 0 && before == rec) on = false;
    }
    if (on) {
        float* dst = acc[rec];
        if constexpr (kAtomic) {
            atomicAdd(dst + (lane & 7), tot);
            if ((lane & 7) == 0) atomicAdd(dst + 8, z);
        } else {
            dst[lane & 7] += tot;
            if ((lane & 7) == 0) dst[8] += z;
        }
    }
    __syncwarp();
}

// kConsistent: the exact-gradient backward mode (FGS_BACKWARD_CONSISTENT), a
// compile-time switch so that the reference mode pays nothing for it per pixel.
template <int PPT, int kBatch, bool kConsistent>
__device__ __forceinline__ void render_bwd_tile(BwdSmem<PPT, kBatch>& sm, const TileArgs& a, int tile, uint32_t& gb,
                                                unsigned* err)
{
    constexpr int kSlots = bwd_slots<PPT>();
    constexpr bool kOwnSlot = PPT == 4;
    constexpr int NT = 256 / PPT;
    constexpr int NP = PPT > 1 ? PPT / 2 : 1;
    constexpr int NG = 9;  // dcolor r,g,b ; dmean2D x,y ; dconic x,y,w ; dopacity
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int W = a.W, H = a.H;
    const int gx = (W + kTileX - 1) / kTileX;
    const int bx = tile % gx, by = tile / gx;
    const int px = bx * kTileX + (lane & 15);
    // first row of the lane's pair in the warp's first strip (its row at one pixel per lane)
    const int py0 = by * kTileY + 2 * PPT * warp + (PPT > 1 ? 2 : 1) * (lane >> 4);
    const uint2 range = a.ranges[tile];
    const PairRecord* recs = a.recs;

    BwdPixels<NP> s;
    const float bg0 = a.bg[0], bg1 = a.bg[1], bg2 = a.bg[2];
    uint32_t my_max = 0;
    bool tame = true;
#pragma unroll
    for (int q = 0; q < NP; q++) {
        float T[2], d[2][3], bgT[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int py = py0 + 4 * q + h;
            const bool inside = px < W && py < H && 2 * q + h < PPT;
            const int pix = W * py + px;
            T[h] = inside ? a.final_T[pix] : 0.f;
            s.last[2 * q + h] = inside ? a.n_contrib[pix] : 0;
            my_max = max(my_max, s.last[2 * q + h]);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                d[h][c] = inside ? a.dL_dpix[c * H * W + pix] : 0.f;
                tame = tame && fabsf(d[h][c]) < 1e15f;
            }
            bgT[h] = -T[h] * (bg0 * d[h][0] + bg1 * d[h][1] + bg2 * d[h][2]);
            tame = tame && fabsf(bgT[h]) < 1e30f;
        }
        s.T[q] = f2(T[0], T[1]);
        s.bgT[q] = f2(bgT[0], bgT[1]);
        s.acc[q] = f2(0.f);
        s.npy[q] = f2(-(float)(py0 + 4 * q), -(float)(py0 + 4 * q + 1));
#pragma unroll
        for (int c = 0; c < 3; c++) s.d[q][c] = f2(d[0][c], d[1][c]);
        s.d01[q][0] = f2(d[0][0], d[0][1]);
        s.d01[q][1] = f2(d[1][0], d[1][1]);
    }
    // a gradient too large for the packed form (or not finite) sends the warp the other way
    const uint32_t wild_warp = __all_sync(0xffffffffu, tame) ? 0u : kWild;
    const float pxf = (float)px;
    const int mbit = PPT == 4 ? 4 * warp : 2 * (warp * PPT / 2);  // the first strip's bits in a block_mask
    const float ddelx_dx = 0.5 * W;
    const float ddely_dy = 0.5 * H;
    const int q_lane = (lane & 1) ? 15 : sum9_component((unsigned)lane);
    StepSums& steps = sm.step[PPT == 1 ? 0 : warp];
    int pending = 0;

    if (tid == 0) sm.max_last = 0;
    __syncthreads();
    const uint32_t warp_last = __reduce_max_sync(0xffffffffu, my_max);
    if (lane == 0) atomicMax(&sm.max_last, warp_last);
    __syncthreads();
    // Entries at or beyond the largest n_contrib of the tile touch no pixel.
    const uint32_t n = min(range.y - range.x, sm.max_last);
    const int nb = (int)((n + kBatch - 1) / kBatch);
    // batch b holds entries [lo_b, hi_b) with hi_b = n - b*kBatch (back to front)
    auto issue = [&](int b) {
        const uint32_t hi = n - b * kBatch, lo = hi > (uint32_t)kBatch ? hi - kBatch : 0;
        const int buf = (int)((gb + b) % kBufs);
        issue_batch(sm.rec[buf], &sm.bar[buf], recs, range.x + lo, hi - lo);
    };
    if (tid == 0)
        for (int b = 0; b < kBufs && b < nb; b++) issue(b);

    // Warps go through the batches on their own: a batch's sums are written out by the warp
    // that is through with it last, which then has the batch three later copied into its
    // buffer; a warp that waits for that copy also knows that the sums it will add to are
    // zero again.  (With the block waiting twice per batch of 32 a fifth of the warps' time
    // went there.)
    for (int b = 0; b < nb; b++) {
        const uint32_t g = gb + b;
        const int buf = (int)(g % kBufs);
        const uint32_t hi = n - b * kBatch, lo = hi > (uint32_t)kBatch ? hi - kBatch : 0;
        const uint32_t cnt = hi - lo;
        mbar_wait(&sm.bar[buf], (g / kBufs) & 1, err);
        const PairRecord* R = sm.rec[buf];
        for (int k0 = (int)((cnt - 1) & ~31u); k0 >= 0; k0 -= 32) {
            // records of this chunk that sit before some pixel's last contributor and reach
            // this warp's strips, walked back to front
            const uint32_t e = (uint32_t)k0 + lane;
            const uint32_t mask = e < cnt && lo + e < warp_last ? __float_as_uint(R[e].c.z) >> mbit : 0u;
            uint32_t strip[NP], live = 0;
#pragma unroll
            for (int q = 0; q < NP; q++) {
                strip[q] = __ballot_sync(0xffffffffu, ((mask >> (2 * q)) & 3u) != 0);
                live |= strip[q];
            }
            while (live) {
                const int bit = 31 - __clz(live);
                live &= ~(1u << bit);
                const int j = k0 + bit;
                const uint32_t contributor = lo + (uint32_t)j;  // 0-based position in the tile list
                const float4 ra = R[j].a;
                const float4 rb = R[j].b;
                const float2 rc = make_float2(R[j].c.x, R[j].c.z);
                const float dx = ra.x - pxf;
                const bool branchy = PPT == 1 || ((__float_as_uint(rc.y) | wild_warp) & kWild);
                const float sx = __fmul_rn(ra.z, dx), nbx = -__fmul_rn(ra.w, dx);
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    if (NP > 1 && !((strip[q] >> bit) & 1u)) continue;
                    float g[NG];
                    bool any = false;
                    if (branchy) {
#pragma unroll
                        for (int i = 0; i < NG; i++) g[i] = 0.f;
#pragma unroll
                        for (int h = 0; h < 2 && 2 * q + h < PPT; h++) {
                            auto half = [&](F2 x) { return h ? f2_hi(x) : f2_lo(x); };
                            float T = half(s.T[q]), acc = half(s.acc[q]);
                            any |= bwd_pixel_step<kConsistent>(
                                ra, rb, rc.x, pxf, -half(s.npy[q]), contributor < s.last[2 * q + h], T, acc,
                                half(s.d[q][0]), half(s.d[q][1]), half(s.d[q][2]), half(s.bgT[q]), g);
                            s.T[q] = h ? f2(f2_lo(s.T[q]), T) : f2(T, f2_hi(s.T[q]));
                            s.acc[q] = h ? f2(f2_lo(s.acc[q]), acc) : f2(acc, f2_hi(s.acc[q]));
                        }
                    } else {
                        any = bwd_pair_step<kConsistent, NP>(s, q, ra, rb, rc.x, dx, sx, nbx, contributor, g);
                    }
                    if (!__any_sync(0xffffffffu, any)) continue;
                    if constexpr (PPT == 1) {
                        const float tot = warp_transpose_sum9(g);
                        if (q_lane < NG) atomicAdd(&sm.acc[buf][warp >> 1][j][q_lane], tot);
                    } else {
                        auto& st = steps.step[pending];
                        st.a[0][lane] = make_float4(g[0], g[1], g[2], g[3]);
                        st.a[1][lane ^ 4] = make_float4(g[4], g[5], g[6], g[7]);
                        st.b[lane] = g[8];
                        if (lane == 0) steps.rec[pending] = j;
                        if (++pending == kPend) {
                            add_step_sums<!kOwnSlot>(steps, sm.acc[buf][kOwnSlot ? warp : warp >> 1], kPend);
                            pending = 0;
                        }
                    }
                }
            }
        }
        if (PPT > 1 && pending) {
            add_step_sums<!kOwnSlot>(steps, sm.acc[buf][kOwnSlot ? warp : warp >> 1], pending);
            pending = 0;
        }
        uint32_t through = 0;
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            through = atomicAdd(&sm.arrived[buf], 1u);
            __threadfence_block();
        }
        if (__shfl_sync(0xffffffffu, through, 0) != NT / 32 - 1) continue;
        // this batch's per-pair gradients, at each pair's emission index: the slot sums times
        // the pair's own factors (opacity, conic, -W/2, -H/2, -1/2 of backward.cu:537-551)
        for (uint32_t e = lane; e < cnt; e += 32) {
            float* dst = a.pgrad + (size_t)__float_as_uint(R[e].c.w) * NG;
            float sum[NG];
#pragma unroll
            for (int q = 0; q < NG; q++) sum[q] = 0.f;
#pragma unroll
            for (int sl = 0; sl < kSlots; sl++) {
                float* acc = sm.acc[buf][sl][e];
#pragma unroll
                for (int q = 0; q < NG; q++) {
                    sum[q] += acc[q];
                    acc[q] = 0.f;
                }
            }
            const float4 ea = R[e].a, eb = R[e].b;  // conic (ea.z, ea.w, eb.x), opacity eb.y
            const float o = eb.y;
            dst[0] = sum[0];
            dst[1] = sum[1];
            dst[2] = sum[8];
            dst[3] = -ddelx_dx * (o * __fmaf_rn(ea.z, sum[2], __fmul_rn(ea.w, sum[3])));
            dst[4] = -ddely_dy * (o * __fmaf_rn(eb.x, sum[3], __fmul_rn(ea.w, sum[2])));
            dst[5] = -0.5f * (o * sum[4]);
            dst[6] = -0.5f * (o * sum[5]);
            dst[7] = -0.5f * (o * sum[6]);
            dst[8] = sum[7];
        }
        __syncwarp();
        if (lane == 0) {
            sm.arrived[buf] = 0;
            __threadfence_block();
            if (b + kBufs < nb) issue(b + kBufs);
        }
    }
    __syncthreads();  // (the buffers and counters are free for the next tile)
    gb += (uint32_t)nb;
    // pairs at or past the tile's largest n_contrib touch no pixel: zero gradients
    for (uint32_t e = n + tid; e < range.y - range.x; e += NT) {
        float* dst = a.pgrad + (size_t)__float_as_uint(recs[range.x + e].c.w) * NG;
#pragma unroll
        for (int q = 0; q < NG; q++) dst[q] = 0.f;
    }
}

template <typename Smem>
__device__ __forceinline__ void bwd_smem_init(Smem& sm, int NT)
{
    float* acc = &sm.acc[0][0][0][0];
    if (threadIdx.x < kBufs) sm.arrived[threadIdx.x] = 0;
    for (int e = threadIdx.x; e < (int)(sizeof(sm.acc) / sizeof(float)); e += NT) acc[e] = 0.f;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kBufs; i++) mbar_init(&sm.bar[i], 1);
        mbar_fence_init();
    }
    __syncthreads();
}

// Resident CTAs per SM the multi-view backward is compiled for: 28 warps at 2 pixels per
// thread (what the shared memory of 32-record batches lets in) and 24 at 4 (80 registers and
// a few spilled bytes instead of the 94 the compiler takes when left alone).  The
// single-view kernel keeps the compiler's allocation.
template <int PPT>
constexpr int bwd_multi_min_ctas() { return PPT == 2 ? 7 : (PPT == 4 ? 12 : 1); }

template <int PPT, int kBatch, bool kConsistent>
__global__ void __launch_bounds__(256 / PPT) render_bwd_kernel(TileArgs a, ZeroList zero, unsigned* err)
{
    extern __shared__ __align__(128) unsigned char bwd_dyn[];
    BwdSmem<PPT, kBatch>& sm = *reinterpret_cast<BwdSmem<PPT, kBatch>*>(bwd_dyn);
    bwd_smem_init(sm, 256 / PPT);
    uint32_t gb = 0;
    render_bwd_tile<PPT, kBatch, kConsistent>(sm, a, blockIdx.x, gb, err);
    // last, so that the first blocks composite while later ones have not yet anything to store
    zero_share(zero, blockIdx.x);
}

template <int PPT, int kBatch, bool kConsistent>
__global__ void __launch_bounds__(256 / PPT, bwd_multi_min_ctas<PPT>())
    render_bwd_multi_kernel(const TileArgs* __restrict__ views, const uint32_t* __restrict__ begin, int nviews,
                            uint32_t total, uint32_t* queue, ZeroList zero, int zero_shift, unsigned* err)
{
    // (a share of `zero` after one tile in 1 << zero_shift)
    extern __shared__ __align__(128) unsigned char bwd_dyn[];
    BwdSmem<PPT, kBatch>& sm = *reinterpret_cast<BwdSmem<PPT, kBatch>*>(bwd_dyn);
    __shared__ uint32_t s_item;
    bwd_smem_init(sm, 256 / PPT);
    uint32_t gb = 0;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total) break;
        const int v = view_of(begin, nviews, item);
        const TileArgs& a = views[v];  // fields read where used, not held in registers
        render_bwd_tile<PPT, kBatch, kConsistent>(sm, a, (int)(item - begin[v]), gb, err);
        if (!(item & ((1u << zero_shift) - 1u))) zero_share(zero, item >> zero_shift);
        __syncthreads();
    }
}

}  // namespace

namespace {
RenderConfig g_cfg{0, 0, 0, 0, 0, -1};

// Dynamic shared memory of a forward launch: the whole FwdSmem with statistics,
// up to its statistics sums without.
template <int kBatch>
size_t fwd_smem_bytes(bool stats)
{
    return stats ? sizeof(FwdSmem<kBatch>) : offsetof(FwdSmem<kBatch>, ksum);
}

// Dynamic shared memory of a long-tile kernel (opted in once per process and device
// ordinal; Tag tells the kernels apart: single-view 0, multi-view 1).
template <int BW, int BH, int Tag, typename Kern>
size_t long_smem_bytes(Kern k)
{
    static bool done[64] = {};
    const size_t bytes = sizeof(LongSmem<LongTile<BW, BH>::kChunk>);
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !done[dev]) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    return bytes;
}

// Band shapes (fgs_set_render_split): 0 = 16x2, 1 = 8x4, 2 = 4x4, 3 = 4x2 pixels per warp.
template <int BW, int BH>
void long_launch(const TileArgs& a, const uint32_t* list, uint32_t* ctr, uint32_t cap, cudaStream_t s)
{
    constexpr int kThreads = LongTile<BW, BH>::kThreads;
    const size_t smem = long_smem_bytes<BW, BH, 0>(render_fwd_long_kernel<BW, BH>);
    render_fwd_long_kernel<BW, BH><<<resident_ctas(render_fwd_long_kernel<BW, BH>, kThreads), kThreads, smem, s>>>(
        a, list, ctr, cap);
}
void launch_long_kernel(int shape, const TileArgs& a, const uint32_t* list, uint32_t* ctr, uint32_t cap,
                        cudaStream_t s)
{
    if (shape == 1) long_launch<8, 4>(a, list, ctr, cap, s);
    else if (shape == 2) long_launch<4, 4>(a, list, ctr, cap, s);
    else if (shape == 3) long_launch<4, 2>(a, list, ctr, cap, s);
    else long_launch<16, 2>(a, list, ctr, cap, s);
}
template <int BW, int BH>
void long_multi_launch(const TileArgs* views, const uint32_t* begin, int nviews, const uint32_t* list, uint32_t* ctr,
                       uint32_t cap, cudaStream_t s)
{
    constexpr int kThreads = LongTile<BW, BH>::kThreads;
    const size_t smem = long_smem_bytes<BW, BH, 1>(render_fwd_long_multi_kernel<BW, BH>);
    render_fwd_long_multi_kernel<BW, BH>
        <<<resident_ctas(render_fwd_long_multi_kernel<BW, BH>, kThreads), kThreads, smem, s>>>(views, begin, nviews,
                                                                                             list, ctr, cap);
}
void launch_long_multi_kernel(int shape, const TileArgs* views, const uint32_t* begin, int nviews,
                              const uint32_t* list, uint32_t* ctr, uint32_t cap, cudaStream_t s)
{
    if (shape == 1) long_multi_launch<8, 4>(views, begin, nviews, list, ctr, cap, s);
    else if (shape == 2) long_multi_launch<4, 4>(views, begin, nviews, list, ctr, cap, s);
    else if (shape == 3) long_multi_launch<4, 2>(views, begin, nviews, list, ctr, cap, s);
    else long_multi_launch<16, 2>(views, begin, nviews, list, ctr, cap, s);
}

template <int PPT, int B>
void fwd_launch(int grid, const ImageState& im, const BinState& b, long long K, int W, int H, const float* bg,
                float* out_color, int* point_id, float* pw_pixel, float* point_weight, bool stats, int split,
                int band_shape, unsigned* err, cudaStream_t s)
{
    TileArgs a{};
    a.ranges = im.ranges; a.recs = b.rec; a.W = W; a.H = H; a.bg = bg;
    a.out_color = out_color; a.final_T = im.final_T; a.n_contrib = im.n_contrib; a.out_point_id = point_id;
    a.out_pw_pixel = pw_pixel; a.out_point_weight = point_weight;
    a.kv_sum = stats ? b.kv_sum : nullptr; a.kv_cnt = stats ? b.kv_cnt : nullptr;
    if (split > 0) {
        // long tiles first, in bands; the tile kernel then skips them
        cudaMemsetAsync(im.long_ctr, 0, (2 + kLongBuckets) * sizeof(uint32_t), s);
        if (stats && K > 0) {
            cudaMemsetAsync(b.kv_sum, 0, sizeof(float) * (size_t)K, s);
            cudaMemsetAsync(b.kv_cnt, 0, sizeof(uint32_t) * (size_t)K, s);
        }
        long_tiles_kernel<<<(grid + 255) / 256, 256, 0, s>>>(im.ranges, (uint32_t)grid, (uint32_t)split, im.long_list,
                                                             im.long_ctr);
        launch_long_kernel(band_shape, a, im.long_list, im.long_ctr, (uint32_t)grid, s);
        note_launches(2);
    }
    const uint32_t split_min = (uint32_t)(split > 0 ? split : 0);
    if (stats)
        render_fwd_kernel<PPT, B, kStats><<<grid, 256 / PPT, fwd_smem_bytes<B>(true), s>>>(a, split_min, err);
    else
        render_fwd_kernel<PPT, B, kWeights><<<grid, 256 / PPT, fwd_smem_bytes<B>(false), s>>>(a, split_min, err);
}

// Dynamic shared memory of a backward kernel instantiation (opted in once per process
// and device ordinal; Tag tells the kernels apart: single-view 0, multi-view 1, +2 in the
// consistent mode).
template <int PPT, int B, int Tag, typename Kern>
size_t bwd_smem_bytes(Kern k)
{
    static bool done[64] = {};
    const size_t bytes = sizeof(BwdSmem<PPT, B>);
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !done[dev]) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    return bytes;
}

template <int PPT, int B>
void bwd_launch(int grid, const ImageState& im, const BinState& b, int W, int H, const float* bg, const float* dL,
                int consistent, const ZeroList& zero, unsigned* err, cudaStream_t s)
{
    TileArgs a{};
    a.ranges = im.ranges; a.recs = b.rec; a.W = W; a.H = H; a.bg = bg;
    a.final_T = im.final_T; a.n_contrib = im.n_contrib;
    a.dL_dpix = dL; a.pgrad = b.pgrad;
    if (consistent) {
        const size_t smem = bwd_smem_bytes<PPT, B, 2>(render_bwd_kernel<PPT, B, true>);
        render_bwd_kernel<PPT, B, true><<<grid, 256 / PPT, smem, s>>>(a, ZeroList(zero).split((size_t)grid), err);
    } else {
        const size_t smem = bwd_smem_bytes<PPT, B, 0>(render_bwd_kernel<PPT, B, false>);
        render_bwd_kernel<PPT, B, false><<<grid, 256 / PPT, smem, s>>>(a, ZeroList(zero).split((size_t)grid), err);
    }
}

#define FGS_RENDER_DISPATCH(FN, PPT_, B_, ...)                                            \
    do {                                                                                  \
        const int ppt_ = (PPT_), b_ = (B_);                                               \
        if (ppt_ == 1 && b_ == 64) FN<1, 64>(__VA_ARGS__);                                \
        else if (ppt_ == 1 && b_ == 128) FN<1, 128>(__VA_ARGS__);                         \
        else if (ppt_ == 1) FN<1, 256>(__VA_ARGS__);                                      \
        else if (ppt_ == 2 && b_ == 64) FN<2, 64>(__VA_ARGS__);                           \
        else if (ppt_ == 2 && b_ == 128) FN<2, 128>(__VA_ARGS__);                         \
        else if (ppt_ == 2) FN<2, 256>(__VA_ARGS__);                                      \
        else if (ppt_ == 4 && b_ == 64) FN<4, 64>(__VA_ARGS__);                           \
        else if (ppt_ == 4 && b_ == 128) FN<4, 128>(__VA_ARGS__);                         \
        else FN<4, 256>(__VA_ARGS__);                                                     \
    } while (0)
}  // namespace

bool valid_render_config(const RenderConfig& c)
{
    auto shape = [](int p, int b) {
        return (p == 0 && b == 0) || ((p == 1 || p == 2 || p == 4) && (b == 64 || b == 128 || b == 256));
    };
    const bool split = c.own_split() ? c.fwd_split >= 0 && c.fwd_band <= 3 : c.fwd_split == 0 && c.fwd_band == -1;
    return shape(c.fwd_ppt, c.fwd_batch) && shape(c.bwd_ppt, c.bwd_batch) && split;
}
void set_render_config(const RenderConfig& c) { g_cfg = c; }
RenderConfig get_render_config() { return g_cfg; }

namespace {
template <int kOut>
void fwd_rule_launch(int tiles, const TileArgs& a, const ImageState& im, unsigned* err, cudaStream_t s)
{
    const int long_ctas = (int)resident_ctas(render_fwd_rule_kernel<kOut>, 256 / kRulePpt);
    render_fwd_rule_kernel<kOut><<<long_ctas + tiles, 256 / kRulePpt, fwd_smem_bytes<kRuleBatch>(kOut == kStats), s>>>(
        a, long_ctas, im.long_list, im.long_ctr, (uint32_t)tiles, err);
}
}  // namespace

void launch_render_fwd(const RenderConfig& c, int W, int H, const ImageState& im, const BinState& b, long long K,
                       const unsigned long long* totals, const float* bg, float* out_color, int* point_id,
                       float* pw_pixel, float* point_weight, bool stats, unsigned* err, cudaStream_t s)
{
    const int gx = (W + kTileX - 1) / kTileX, gy = (H + kTileY - 1) / kTileY;
    note_launches(1);
    if (c.rule_long()) {
        TileArgs a{};
        a.ranges = im.ranges; a.recs = b.rec; a.W = W; a.H = H; a.bg = bg;
        a.out_color = out_color; a.final_T = im.final_T; a.n_contrib = im.n_contrib; a.out_point_id = point_id;
        a.out_pw_pixel = pw_pixel; a.out_point_weight = point_weight;
        a.kv_sum = stats ? b.kv_sum : nullptr; a.kv_cnt = stats ? b.kv_cnt : nullptr;
        a.totals = totals;
        if (stats) fwd_rule_launch<kStats>(gx * gy, a, im, err, s);
        else fwd_rule_launch<kWeights>(gx * gy, a, im, err, s);
        return;
    }
    FGS_RENDER_DISPATCH(fwd_launch, c.own_fwd() ? c.fwd_ppt : kRulePpt, c.own_fwd() ? c.fwd_batch : kRuleBatch,
                        gx * gy, im, b, K, W, H, bg, out_color, point_id, pw_pixel, point_weight, stats, c.fwd_split,
                        c.fwd_band, err, s);
}

namespace {
template <int PPT, int B>
void fwd_multi_launch(const TileArgs* views, const uint32_t* begin, int nviews, uint32_t total, uint32_t* queue,
                      uint32_t* long_list, uint32_t* long_ctr, int split, int band_shape, unsigned* err,
                      cudaStream_t s)
{
    if (split > 0) {
        cudaMemsetAsync(long_ctr, 0, (2 + kLongBuckets) * sizeof(uint32_t), s);
        long_tiles_multi_kernel<<<(total + 255) / 256, 256, 0, s>>>(views, begin, nviews, total, (uint32_t)split,
                                                                    long_list, long_ctr);
        launch_long_multi_kernel(band_shape, views, begin, nviews, long_list, long_ctr, total, s);
        note_launches(2);
    }
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = fwd_smem_bytes<B>(false);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_fwd_multi_kernel<PPT, B>, 256 / PPT, smem);
    const int grid = sms * (per_sm > 0 ? per_sm : 1);
    render_fwd_multi_kernel<PPT, B><<<grid, 256 / PPT, smem, s>>>(views, begin, nviews, total, queue,
                                                               (uint32_t)(split > 0 ? split : 0), err);
}

template <int PPT, int B, bool kConsistent>
void bwd_multi_launch_mode(const TileArgs* views, const uint32_t* begin, int nviews, uint32_t total, uint32_t* queue,
                           const ZeroList& zero, unsigned* err, cudaStream_t s)
{
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = bwd_smem_bytes<PPT, B, kConsistent ? 3 : 1>(render_bwd_multi_kernel<PPT, B, kConsistent>);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_bwd_multi_kernel<PPT, B, kConsistent>, 256 / PPT,
                                                  smem);
    const int grid = sms * (per_sm > 0 ? per_sm : 1);
    int shift = 0;
    while (shift < 4 && (total >> (shift + 1)) >= 4u * (uint32_t)grid) shift++;
    const size_t parts = (total + (1u << shift) - 1u) >> shift;
    render_bwd_multi_kernel<PPT, B, kConsistent><<<grid, 256 / PPT, smem, s>>>(
        views, begin, nviews, total, queue, ZeroList(zero).split(parts), shift, err);
}

template <int PPT, int B>
void bwd_multi_launch(const TileArgs* views, const uint32_t* begin, int nviews, uint32_t total, uint32_t* queue,
                      const ZeroList& zero, int consistent, unsigned* err, cudaStream_t s)
{
    if (consistent)
        bwd_multi_launch_mode<PPT, B, true>(views, begin, nviews, total, queue, zero, err, s);
    else
        bwd_multi_launch_mode<PPT, B, false>(views, begin, nviews, total, queue, zero, err, s);
}
}  // namespace

void launch_render_fwd_multi(const RenderConfig& c, const TileArgs* views, const uint32_t* begin, int nviews,
                             uint32_t total_tiles, uint32_t* queue, uint32_t* long_list, uint32_t* long_ctr,
                             unsigned* err, cudaStream_t s)
{
    cudaMemsetAsync(queue, 0, sizeof(uint32_t), s);
    note_launches(1);
    if (c.rule_long()) {
        int dev = 0, sms = 148, per_sm = 1;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const size_t smem = fwd_smem_bytes<kRuleBatch>(false);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_fwd_multi_rule_kernel, 256 / kRulePpt, smem);
        render_fwd_multi_rule_kernel<<<sms * (per_sm > 0 ? per_sm : 1), 256 / kRulePpt, smem, s>>>(
            views, begin, nviews, total_tiles, queue, long_list, long_ctr, err);
        return;
    }
    FGS_RENDER_DISPATCH(fwd_multi_launch, c.own_fwd() ? c.fwd_ppt : kRulePpt, c.own_fwd() ? c.fwd_batch : kRuleBatch,
                        views, begin, nviews, total_tiles, queue, long_list, long_ctr, c.fwd_split, c.fwd_band, err,
                        s);
}

// The backward's shapes.  Its batches hold 32 records whatever batch a caller sets: the gradients'
// bits do not depend on it, and as warps do not wait for one another at a batch, larger ones only
// take shared memory from resident warps.  Until a caller sets a shape it is 2 pixels per lane.
// Measured, in us, at (2, 32) / (2, 64) / (4, 32): a view of 256 tiles 50 / 49 / 81, 4056 tiles 263 /
// 274 / 279, 8160 tiles 465 / 493 / 452, 16 of these 7065 / 7703 / 7218, six views of 1200 to 5700
// tiles 1705 / 1745 / 2045.
constexpr int kBwdRulePpt = 2, kBwdBatch = 32;
#define FGS_BWD_DISPATCH(FN, ...)                                        \
    do {                                                                 \
        const int ppt_ = g_cfg.own_bwd() ? g_cfg.bwd_ppt : kBwdRulePpt;  \
        if (ppt_ == 1) FN<1, kBwdBatch>(__VA_ARGS__);                    \
        else if (ppt_ == 2) FN<2, kBwdBatch>(__VA_ARGS__);               \
        else FN<4, kBwdBatch>(__VA_ARGS__);                              \
    } while (0)

// Whether the compositing launch zeroes the buffers, a share per tile, or a launch of its own before
// it, at the memory's rate.  A block stores 15 to 50 GB/s, so with few tiles the shares are the
// backward's time: 2M Gaussians with SH 3 (568 MB), one view, shares / own launch in us: 1 tile
// 9606 / 176, 16 tiles 731 / 178, 64 tiles 238 / 186, 256 tiles 195 / 193, 1024 tiles 231 / 237, 8160 tiles
// 660 / 737; two views in one launch, tiles of both: 32 852 / 178, 128 318 / 193, 512 218 / 215, 1024
// 214 / 232.  200K Gaussians: 64 tiles (888 KB each) 61 / 56, 256 tiles (222 KB) 53 / 60; 20K: 4 tiles
// (1.4 MB) 63 / 45, 16 (355 KB) 43 / 44, 64 (89 KB) 42 / 51.  From four tiles per SM on the blocks together
// store at the memory's rate, and up to 256 KB a share costs less than the launch.
bool zeroed_in_shares(const ZeroList& z, uint32_t tiles)
{
    size_t words = 0;
    for (int b = 0; b < z.n; b++) words += z.words[b];
    if (words * 4 <= (size_t)tiles * (256 << 10)) return true;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return tiles >= 4u * (uint32_t)sms;
}

void launch_render_bwd_multi(const TileArgs* views, const uint32_t* begin, int nviews, uint32_t total_tiles,
                             uint32_t* queue, const ZeroList& zero, int consistent, unsigned* err, cudaStream_t s)
{
    cudaMemsetAsync(queue, 0, sizeof(uint32_t), s);
    const bool shares = zeroed_in_shares(zero, total_tiles);
    if (!shares) launch_zero(zero, s);
    FGS_BWD_DISPATCH(bwd_multi_launch, views, begin, nviews, total_tiles, queue, shares ? zero : ZeroList{}, consistent,
                     err, s);
    note_launches(1);
}

void launch_render_bwd(int W, int H, const ImageState& im, const BinState& b, const float* bg,
                       const float* dL_dpix, int consistent, const ZeroList& zero, unsigned* err, cudaStream_t s)
{
    const int gx = (W + kTileX - 1) / kTileX, gy = (H + kTileY - 1) / kTileY;
    const bool shares = zeroed_in_shares(zero, (uint32_t)(gx * gy));
    if (!shares) launch_zero(zero, s);
    FGS_BWD_DISPATCH(bwd_launch, gx * gy, im, b, W, H, bg, dL_dpix, consistent, shares ? zero : ZeroList{}, err, s);
    note_launches(1);
}

}  // namespace fgs
