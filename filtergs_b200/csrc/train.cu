// Training-step kernels around the rasterizer (the loss, the optimizer and the
// densification statistics of LoG's training loop):
//
//   loss       LoG/render/loss.py:6-44 (SSIM, 11x11 Gaussian window, sigma 1.5,
//              no padding: "valid" outputs) and renderer.py:260-273
//              (0.8 * L1 + 0.2 * (1 - SSIM)), forward and gradient in two tiled
//              kernels per image channel, partial sums reduced in a fixed order.
//   activate   LoG/model/activation.py (exp scale, sigmoid opacity, normalised
//              quaternion) from the raw parameters.
//   adam       LoG/model/sparse_optimizer.py:41-78,163-196: Adam with bias
//              correction from the global step, eps 1e-15, on the rows that were
//              visible this step only; the gradients w.r.t. the activated values
//              are chained through the activations first, and the activated values
//              of the updated rows are rewritten for the next forward.
//   densify    LoG/model/counter.py:36-83 (reduced to the two statistics the
//              training step keeps): sum of |dL/dmean2D[:, :2]| and the visibility
//              count per Gaussian, plus this step's visible flag.
#include <cmath>
#include <cstring>
#include <initializer_list>

#include "fgs_common.cuh"
#include "fgs_internal.h"

namespace fgs {

namespace {

constexpr int kWin = 11;           // SSIM window
constexpr int kHalo = kWin - 1;    // valid outputs lose kHalo rows / columns
constexpr int kTX = 32, kTY = 32;  // output (or pixel) tile of one CTA
constexpr int kIn = kTY + kHalo;   // rows of a tile with its halo
constexpr int kPitch = 44;         // its columns, rounded up to whole 16-byte items
constexpr int kLead = 2;           // columns loaded before the gradient's halo, to start on 16 bytes
constexpr float kC1 = 0.01f * 0.01f, kC2 = 0.03f * 0.03f;

// The window is symmetric: weights 0 .. 5, each twice (one operand for both halves of a
// packed multiply-add).  Kernels pin them in registers: left as parameters they were
// fetched again for every tap, as many instructions as the multiply-adds themselves.
constexpr int kTaps = kWin / 2 + 1;
struct Window {
    F2 g[kTaps];
};
__device__ __forceinline__ constexpr int tap(int j) { return j < kTaps ? j : kWin - 1 - j; }
__device__ __forceinline__ void pin_window(const Window& win, F2 (&w)[kTaps])
{
#pragma unroll
    for (int j = 0; j < kTaps; j++) {
        w[j] = win.g[j];
        asm volatile("" : "+l"(w[j]));
    }
}

// ---------------------------------------------------------------- staging
// Rows y0 .. y0 + kIn - 1, columns x0 .. x0 + kPitch - 1 of a plane of h rows, w columns and
// `pitch` floats per row into shared memory by asynchronous copies, all in flight at once and
// without registers; zeros outside the plane.  kVec: 16-byte copies (x0, w and pitch are
// multiples of 4 and the plane starts on 16 bytes), else 4-byte ones.
template <bool kVec>
__device__ __forceinline__ void stage_tile(float (*dst)[kPitch], const float* __restrict__ src, int x0, int y0, int w,
                                           int h, int pitch)
{
    constexpr int kW = kVec ? 4 : 1, kItems = kPitch / kW;
    for (int i = threadIdx.x; i < kIn * kItems; i += kTX * kTY / 8) {
        const int r = i / kItems, c = (i - r * kItems) * kW;
        const int gx = x0 + c, gy = y0 + r;
        const bool in = gx >= 0 && gx < w && gy >= 0 && gy < h;
        const float* p = in ? src + (size_t)gy * pitch + gx : src;
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(&dst[r][c]);
        if constexpr (kVec)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(p), "r"(in ? 16 : 0) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(p), "r"(in ? 4 : 0) : "memory");
    }
}
__device__ __forceinline__ void stage_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}
// kSeg + kHalo consecutive values of a staged row from column c (a multiple of 4): 16-byte
// loads; lanes in consecutive rows are free of bank conflicts at this pitch.
template <int kN>
__device__ __forceinline__ void row_window(const float* __restrict__ row, int c, float (&v)[kN])
{
    static_assert(kN % 4 == 0, "whole 16-byte loads");
#pragma unroll
    for (int k = 0; k < kN; k += 4) {
        const float4 q = *reinterpret_cast<const float4*>(row + c + k);
        v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
    }
}

// ---------------------------------------------------------------- SSIM forward + coefficient maps
// One CTA: a 32x32 tile of valid outputs of one channel.  The 11-tap Gaussian is applied
// along rows (an item makes kSeg outputs of one row from kSeg + 10 staged pixels) into
// shared memory, then down columns (kRowsPer outputs of one column per thread from
// kRowsPer + 10 values) to x and y (packed: two multiply-adds per instruction), x^2 and
// y^2 (packed) and x y, every output summing its taps in window order.  The tile arrives by
// asynchronous copies: with plain loads, a few in flight per thread, the kernel waited for
// them two thirds of its time.  Lanes of the row pass take consecutive rows, whose pitches
// are free of bank conflicts.  Per output q the loss gradient w.r.t. the five local means
// is kept as three maps (d/dmu_x, d/dE[x^2], d/dE[xy]) of `gpitch` floats per row, zero past
// the last output; the SSIM values of the tile are summed in a fixed order.
// 1920x1080, three channels: 118 -> 80 us (scalar sums, 32x16 tiles before), the same bits.
constexpr int kRowsPer = 8;   // outputs of one column per thread
constexpr int kLossThreads = kTX * kTY / kRowsPer;
constexpr int kSeg = 8;       // outputs of one row per row-pass item
constexpr int kSumRows = 16;  // rows of values that one float32 partial sum spans

// A tile's float32 partial sums, one per kSumRows rows, from a thread's sums over the upper and
// lower four of its eight rows: lanes by a tree, then the four strips of four rows in turn.
// (Sums over all 32 rows would carry twice as many values in float32 before the double sum of
// loss_reduce_kernel.)  Partials lie [channel][rows / kSumRows][tile column].
constexpr int kStrips = kSumRows / (kRowsPer / 2);
static_assert(kStrips == 4 && kLossThreads / 32 * 2 == kTY / kSumRows * kStrips, "two strips per warp");
__device__ __forceinline__ void tile_partials(float upper, float lower, float (&red)[kTY / kSumRows][kStrips], int rows,
                                              float* __restrict__ partial)
{
    const int tid = threadIdx.x;
    // both trees at once: after lanes 16 apart, the lower half warp goes on with the upper rows' sum
    const bool second = tid & 16;
    float v = (second ? lower : upper) + __shfl_xor_sync(0xffffffffu, second ? upper : lower, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 15) == 0) (&red[0][0])[tid >> 4] = v;
    __syncthreads();
    const int blocks = (rows + kSumRows - 1) / kSumRows, by = blockIdx.y * (kTY / kSumRows) + tid;
    if (tid < kTY / kSumRows && by < blocks) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < kStrips; k++) t += red[tid][k];
        partial[((size_t)blockIdx.z * blocks + by) * gridDim.x + blockIdx.x] = t;
    }
}

template <bool kVec>
__global__ void __launch_bounds__(kLossThreads)
    ssim_forward_kernel(int W, int H, const float* __restrict__ pred, const float* __restrict__ target, Window win,
                        float ssim_grad_scale, float* __restrict__ gmap, int gpitch, float* __restrict__ partial)
{
    __shared__ __align__(16) float sx[kIn][kPitch], sy[kIn][kPitch];
    __shared__ ulonglong2 hq[kIn][kTX + 1];  // {mean x, mean y}, {mean x^2, mean y^2} along the row
    __shared__ float hp[kIn][kTX + 1];       // mean x y
    __shared__ float red[kTY / kSumRows][kStrips];
    const int Wo = W - kHalo, Ho = H - kHalo;
    const int c = blockIdx.z;
    const int ox0 = blockIdx.x * kTX, oy0 = blockIdx.y * kTY;
    const int tid = threadIdx.x, lane = tid & 31;
    stage_tile<kVec>(sx, pred + (size_t)c * W * H, ox0, oy0, W, H, W);
    stage_tile<kVec>(sy, target + (size_t)c * W * H, ox0, oy0, W, H, W);
    stage_wait();
    F2 w[kTaps];
    pin_window(win, w);
    for (int i = tid; i < kIn * (kTX / kSeg); i += kLossThreads) {
        const int r = i % kIn, c0 = (i / kIn) * kSeg;
        float u[kSeg + 12], v[kSeg + 12];
        row_window(sx[r], c0, u);
        row_window(sy[r], c0, v);
        F2 m[kSeg], e[kSeg];
        float p[kSeg];
#pragma unroll
        for (int k = 0; k < kSeg; k++) {
            m[k] = e[k] = f2(0.f);
            p[k] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < kSeg + kHalo; k++) {
            const F2 p2 = f2(u[k], v[k]), s2 = f2_mul(p2, p2);
            const float uv = __fmul_rn(u[k], v[k]);
#pragma unroll
            for (int q = 0; q < kSeg; q++) {
                const int j = k - q;  // the output's tap: ascending as k runs
                if (j < 0 || j >= kWin) continue;
                m[q] = f2_fma(w[tap(j)], p2, m[q]);
                e[q] = f2_fma(w[tap(j)], s2, e[q]);
                p[q] = __fmaf_rn(f2_lo(w[tap(j)]), uv, p[q]);
            }
        }
#pragma unroll
        for (int k = 0; k < kSeg; k++) {
            hq[r][c0 + k] = make_ulonglong2(m[k], e[k]);
            hp[r][c0 + k] = p[k];
        }
    }
    __syncthreads();
    const int tx = lane, ty0 = (tid >> 5) * kRowsPer;
    F2 m[kRowsPer], e[kRowsPer];
    float p[kRowsPer];
#pragma unroll
    for (int k = 0; k < kRowsPer; k++) {
        m[k] = e[k] = f2(0.f);
        p[k] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < kRowsPer + kHalo; k++) {
        const ulonglong2 v = hq[ty0 + k][tx];
        const float uv = hp[ty0 + k][tx];
#pragma unroll
        for (int q = 0; q < kRowsPer; q++) {
            const int j = k - q;
            if (j < 0 || j >= kWin) continue;
            m[q] = f2_fma(w[tap(j)], v.x, m[q]);
            e[q] = f2_fma(w[tap(j)], v.y, e[q]);
            p[q] = __fmaf_rn(f2_lo(w[tap(j)]), uv, p[q]);
        }
    }
    float s[2] = {0.f, 0.f};
    const size_t plane = (size_t)gpitch * Ho;
    float* gm = gmap + (size_t)c * 3 * plane;
#pragma unroll
    for (int rr = 0; rr < kRowsPer; rr++) {
        const int ox = ox0 + tx, oy = oy0 + ty0 + rr;
        if (ox < Wo && oy < Ho) {
            const float m1 = f2_lo(m[rr]), m2 = f2_hi(m[rr]);
            const float s11 = f2_lo(e[rr]) - m1 * m1, s22 = f2_hi(e[rr]) - m2 * m2, s12 = p[rr] - m1 * m2;
            const float A = 2.f * m1 * m2 + kC1, B = 2.f * s12 + kC2;
            const float Cc = m1 * m1 + m2 * m2 + kC1, D = s11 + s22 + kC2;
            const float CD = Cc * D;
            const float ss = (A * B) / CD;
            // d ssim / d(mu_x, E[x^2], E[xy]); the loss is 0.2 (1 - mean ssim): scale by -ssim_grad_scale
            const float d_m1 = (2.f * m2 * B - 2.f * m2 * A) / CD - ss * (2.f * m1 / Cc - 2.f * m1 / D);
            const float d_e11 = -ss / D;
            const float d_e12 = 2.f * A / CD;
            const size_t o = (size_t)oy * gpitch + ox;
            gm[o] = -ssim_grad_scale * d_m1;
            gm[plane + o] = -ssim_grad_scale * d_e11;
            gm[2 * plane + o] = -ssim_grad_scale * d_e12;
            s[rr / (kRowsPer / 2)] += ss;
        } else if (ox < gpitch && oy < Ho) {
            const size_t o = (size_t)oy * gpitch + ox;
            gm[o] = gm[plane + o] = gm[2 * plane + o] = 0.f;
        }
    }
    tile_partials(s[0], s[1], red, Ho, partial);
}

// ---------------------------------------------------------------- loss gradient per pixel
// dL/dx_p = sum over the outputs q whose window covers p of w(q, p) *
// (G1(q) + 2 x_p G11(q) + y_p G12(q)), a transposed separable convolution of the
// three coefficient maps, plus the L1 term w_l1 * sign(x_p - y_p).  One CTA: a 32x32
// pixel tile of one channel, the two passes as in ssim_forward_kernel with {G1, G11}
// packed and G12 beside them; also sums |x - y| over the tile.  1920x1080, three
// channels: 120 -> 56 us.
__global__ void __launch_bounds__(kLossThreads)
    loss_grad_kernel(int W, int H, const float* __restrict__ pred, const float* __restrict__ target, Window win,
                     const float* __restrict__ gmap, int gpitch, float l1_grad_scale, float* __restrict__ dpred,
                     float* __restrict__ partial)
{
    __shared__ __align__(16) float sg[3][kIn][kPitch];  // from column px0 - kHalo - kLead
    __shared__ float2 ha[kIn][kTX + 1];
    __shared__ float hb[kIn][kTX + 1];
    __shared__ float red[kTY / kSumRows][kStrips];
    const int Ho = H - kHalo;
    const int c = blockIdx.z;
    const int px0 = blockIdx.x * kTX, py0 = blockIdx.y * kTY;
    const size_t plane = (size_t)gpitch * Ho;
    const float* gm = gmap + (size_t)c * 3 * plane;
    const int tid = threadIdx.x, lane = tid & 31;
    // outputs q in [p - kHalo, p]: rows py0 - kHalo .. py0 + kTY - 1
#pragma unroll
    for (int k = 0; k < 3; k++)
        stage_tile<true>(sg[k], gm + k * plane, px0 - kHalo - kLead, py0 - kHalo, gpitch, Ho, gpitch);
    stage_wait();
    F2 w[kTaps];
    pin_window(win, w);
    // along rows: T(r, p) = sum_j g_j G(r, p - j), window columns c0 .. c0 + kSeg + kHalo
    for (int i = tid; i < kIn * (kTX / kSeg); i += kLossThreads) {
        const int r = i % kIn, c0 = (i / kIn) * kSeg;
        float g0[kSeg + 12], g1[kSeg + 12], g2[kSeg + 12];
        row_window(sg[0][r], c0, g0);
        row_window(sg[1][r], c0, g1);
        row_window(sg[2][r], c0, g2);
        F2 a[kSeg];
        float b[kSeg];
#pragma unroll
        for (int k = 0; k < kSeg; k++) {
            a[k] = f2(0.f);
            b[k] = 0.f;
        }
#pragma unroll
        for (int k = kSeg + kHalo - 1; k >= 0; k--) {
            const float v = g2[k + kLead];
            const F2 u2 = f2(g0[k + kLead], g1[k + kLead]);
#pragma unroll
            for (int q = 0; q < kSeg; q++) {
                const int j = q + kHalo - k;
                if (j < 0 || j >= kWin) continue;
                a[q] = f2_fma(w[tap(j)], u2, a[q]);
                b[q] = __fmaf_rn(f2_lo(w[tap(j)]), v, b[q]);
            }
        }
#pragma unroll
        for (int k = 0; k < kSeg; k++) {
            ha[r][c0 + k] = make_float2(f2_lo(a[k]), f2_hi(a[k]));
            hb[r][c0 + k] = b[k];
        }
    }
    __syncthreads();
    const int tx = lane, ty0 = (tid >> 5) * kRowsPer;
    const int px = px0 + tx;
    const size_t o0 = (size_t)c * W * H + px;
    float xs[kRowsPer], ys[kRowsPer];  // in flight during the column pass
#pragma unroll
    for (int rr = 0; rr < kRowsPer; rr++) {
        const int py = py0 + ty0 + rr;
        const bool in = px < W && py < H;
        xs[rr] = in ? __ldg(pred + o0 + (size_t)py * W) : 0.f;
        ys[rr] = in ? __ldg(target + o0 + (size_t)py * W) : 0.f;
    }
    F2 a[kRowsPer];
    float b[kRowsPer];
#pragma unroll
    for (int k = 0; k < kRowsPer; k++) {
        a[k] = f2(0.f);
        b[k] = 0.f;
    }
#pragma unroll
    for (int k = kRowsPer + kHalo - 1; k >= 0; k--) {
        const float2 u = ha[ty0 + k][tx];
        const F2 u2 = f2(u.x, u.y);
        const float v = hb[ty0 + k][tx];
#pragma unroll
        for (int q = 0; q < kRowsPer; q++) {
            const int j = q + kHalo - k;
            if (j < 0 || j >= kWin) continue;
            a[q] = f2_fma(w[tap(j)], u2, a[q]);
            b[q] = __fmaf_rn(f2_lo(w[tap(j)]), v, b[q]);
        }
    }
    float l1[2] = {0.f, 0.f};
#pragma unroll
    for (int rr = 0; rr < kRowsPer; rr++) {
        const int py = py0 + ty0 + rr;
        if (px < W && py < H) {
            const size_t o = o0 + (size_t)py * W;
            const float xv = xs[rr], yv = ys[rr];
            const float d = xv - yv;
            const float sgn = d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f);
            dpred[o] = f2_lo(a[rr]) + 2.f * xv * f2_hi(a[rr]) + yv * b[rr] + l1_grad_scale * sgn;
        }
        l1[rr / (kRowsPer / 2)] += fabsf(xs[rr] - ys[rr]);  // (0 outside the image)
    }
    tile_partials(l1[0], l1[1], red, H, partial);
}

// Thread t's sum of p[t], p[t + 1024], ... in turn, 16 loads in flight (1920x1080 has twelve per
// thread; one at a time their latency is the kernel's time).
__device__ __forceinline__ double partial_sum(const float* __restrict__ p, int n)
{
    double a = 0.0;
    for (int i = threadIdx.x; i < n; i += 16 * 1024) {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = i + k * 1024 < n ? __ldg(p + i + k * 1024) : 0.f;
#pragma unroll
        for (int k = 0; k < 16; k++) a += v[k];
    }
    return a;
}

// sums[0] += sum(l1 partials), sums[1] += sum(ssim partials), by one block in a
// fixed order: thread t adds partials t, t + blockDim.x, ... in turn, a butterfly of
// shuffles adds the warp's 32 values (every lane ends with the same bits: each step
// adds the same two operands on both lanes), and thread 0 adds the warp totals in
// warp order.  Every call with the same partials gives the same sums.
__global__ void __launch_bounds__(1024) loss_reduce_kernel(const float* __restrict__ l1p, int nl1,
                                                           const float* __restrict__ sp, int ns,
                                                           double* __restrict__ sums)
{
    __shared__ double s_a[32], s_b[32];
    double a = partial_sum(l1p, nl1), b = partial_sum(sp, ns);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_a[threadIdx.x >> 5] = a;
        s_b[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            ta += s_a[w];
            tb += s_b[w];
        }
        sums[0] += ta;
        sums[1] += tb;
    }
}

// ---------------------------------------------------------------- activation, densification, Adam
__device__ __forceinline__ float sigmoidf(float x) { return 1.f / (1.f + expf(-x)); }

__global__ void activate_kernel(int P, const float* __restrict__ log_scale, const float* __restrict__ rot_raw,
                                const float* __restrict__ opac_logit, float* __restrict__ scale,
                                float* __restrict__ rot, float* __restrict__ opac)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int k = 0; k < 3; k++) scale[3 * i + k] = expf(log_scale[3 * i + k]);
        const float q0 = rot_raw[4 * i], q1 = rot_raw[4 * i + 1], q2 = rot_raw[4 * i + 2], q3 = rot_raw[4 * i + 3];
        const float n = fmaxf(sqrtf(q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3), 1e-12f);
        rot[4 * i] = q0 / n; rot[4 * i + 1] = q1 / n; rot[4 * i + 2] = q2 / n; rot[4 * i + 3] = q3 / n;
        opac[i] = sigmoidf(opac_logit[i]);
    }
}

// Plain path: one view's dense screen-space gradient and radii.
__global__ void densify_dense_kernel(int P, const int* __restrict__ radii, const float* __restrict__ dmean2D,
                                     float* __restrict__ grad_sum, int* __restrict__ vis_count,
                                     uint8_t* __restrict__ flag)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
        if (radii[i] <= 0) continue;
        const float gx = dmean2D[3 * i], gy = dmean2D[3 * i + 1];
        grad_sum[i] += sqrtf(gx * gx + gy * gy);
        vis_count[i] += 1;
        flag[i] = 1;
    }
}

// sparse_optimizer.py:54-76 with torch's float32 arithmetic: the Python-float
// coefficients beta and 1 - beta (formed in double) are rounded to float.  The fused
// products are spelled out, so that no parameter's last bits hang on how a caller's loop
// is compiled.
__device__ __forceinline__ void adam_update(float& p, float& m, float& v, float g, float b1, float omb1, float b2,
                                            float omb2, float step_size, float bc2_sqrt, float eps)
{
    m = __fmaf_rn(g, omb1, __fmul_rn(m, b1));
    v = __fmaf_rn(__fmul_rn(omb2, g), g, __fmul_rn(v, b2));
    const float denom = sqrtf(v) / bc2_sqrt + eps;
    p = __fmaf_rn(-step_size, m / denom, p);
}

}  // namespace

// Bias corrections of the global step, as the reference forms them (double), and the
// float coefficients of the update.
struct AdamCoef {
    double bc1;
    float bc2s, b1, b2, omb1, omb2, eps;
};

__device__ __noinline__ AdamCoef adam_coef(double beta1, double beta2, float eps, int t)
{
    AdamCoef c;
    c.bc1 = 1.0 - pow(beta1, (double)t);
    c.bc2s = (float)sqrt(1.0 - pow(beta2, (double)t));
    c.b1 = (float)beta1;
    c.b2 = (float)beta2;
    c.omb1 = (float)(1.0 - beta1);
    c.omb2 = (float)(1.0 - beta2);
    c.eps = eps;
    return c;
}

// One Adam step of the visible rows, every parameter in one launch: a block takes 256
// consecutive rows and lists the visible ones; blocks of blockIdx.y 0 update their SH
// coefficients, of 1 the rest.  Bound by HBM traffic (per visible row 59 floats of value,
// moments and gradient read and the first three written, 16 SH coefficients), so every
// thread holds one item (16 bytes of an SH row, a float of a mean or a scale, a
// quaternion) of the four arrays in flight, and a block issues its first loads before the
// barrier behind which one thread forms the bias corrections: as double powers formed by
// every thread they cost more than the traffic.  1M rows, 30% of them visible (506 MB):
// 281 -> 114 us, at 40 to 64 resident warps per SM alike; a warp per row and a thread per row, as before, keep too little in
// flight, and so did a warp per 32 rows with two items per lane (64 registers: 302 us).
struct AdamShared {
    AdamCoef c;
    float ss[5];  // step sizes: means, SH, opacity, scale, rotation
    uint32_t count[8];
    uint8_t row[256];
};

__device__ __forceinline__ void adam_one(const AdamShared& sh, int which, float& p, float& m, float& v, float g)
{
    adam_update(p, m, v, g, sh.c.b1, sh.c.omb1, sh.c.b2, sh.c.omb2, sh.ss[which], sh.c.bc2s, sh.c.eps);
}

// kW floats, in one access when the array is aligned for it.
template <int kW>
__device__ __forceinline__ void load_w(const float* __restrict__ p, bool vec, float (&o)[kW])
{
    if (kW == 4 && vec) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        o[0] = q.x; o[kW > 1 ? 1 : 0] = q.y; o[kW > 2 ? 2 : 0] = q.z; o[kW > 3 ? 3 : 0] = q.w;
    } else {
#pragma unroll
        for (int k = 0; k < kW; k++) o[k] = p[k];
    }
}
template <int kW>
__device__ __forceinline__ void store_w(float* __restrict__ p, bool vec, const float (&o)[kW])
{
    if (kW == 4 && vec) {
        *reinterpret_cast<float4*>(p) = make_float4(o[0], o[kW > 1 ? 1 : 0], o[kW > 2 ? 2 : 0], o[kW > 3 ? 3 : 0]);
    } else {
#pragma unroll
        for (int k = 0; k < kW; k++) p[k] = o[k];
    }
}

// The SH rows, in items of kW floats; per: items per row, per_inv = ceil(2^32 / per).
template <int kW>
__device__ __forceinline__ void adam_sh_rows(const fgs_adam_args& a, AdamShared& sh, size_t i0, uint32_t visible,
                                             uint32_t per, uint32_t per_inv)
{
    const uint32_t n = visible * per;
    float p[kW], m[kW], v[kW], g[kW];
    bool ready = false;
    for (uint32_t it0 = 0; it0 < n; it0 += 256) {
        const uint32_t it = it0 + threadIdx.x;
        const uint32_t r = __umulhi(it, per_inv), q = it - r * per;  // it / per
        const size_t j = it < n ? ((i0 + sh.row[r]) * per + q) * kW : 0;
        if (it < n) {
            load_w<kW>(a.shs + j, true, p);
            load_w<kW>(a.m_shs + j, true, m);
            load_w<kW>(a.v_shs + j, true, v);
            load_w<kW>(a.g_shs + j, true, g);
        }
        if (!ready) __syncthreads();  // the coefficients, while the first loads are in flight
        ready = true;
        if (it >= n) continue;
#pragma unroll
        for (int k = 0; k < kW; k++) adam_one(sh, 1, p[k], m[k], v[k], g[k]);
        store_w<kW>(a.shs + j, true, p);
        store_w<kW>(a.m_shs + j, true, m);
        store_w<kW>(a.v_shs + j, true, v);
    }
}

// Means and scales as single floats, opacities and quaternions by row.
__device__ __forceinline__ void adam_small_rows(const fgs_adam_args& a, AdamShared& sh, size_t i0, uint32_t visible,
                                                bool vec)
{
    const uint32_t n = 3 * visible;
    bool ready = false;
    for (uint32_t it0 = 0; it0 < n; it0 += 256) {
        const uint32_t it = it0 + threadIdx.x, r = it / 3;
        const size_t j = it < n ? 3 * (i0 + sh.row[r]) + (it - 3 * r) : 0;
        float px, mx, vx, gx, ps, ms, vs, gs, sc;
        if (it < n) {
            px = a.xyz[j]; mx = a.m_xyz[j]; vx = a.v_xyz[j]; gx = a.g_xyz[j];
            ps = a.log_scale[j]; ms = a.m_scale[j]; vs = a.v_scale[j]; gs = a.g_scale[j]; sc = a.scale[j];
        }
        if (!ready) __syncthreads();
        ready = true;
        if (it >= n) continue;
        adam_one(sh, 0, px, mx, vx, gx);
        a.xyz[j] = px; a.m_xyz[j] = mx; a.v_xyz[j] = vx;
        // scale: d/dlog = d/dscale * scale
        adam_one(sh, 3, ps, ms, vs, gs * sc);
        a.log_scale[j] = ps; a.m_scale[j] = ms; a.v_scale[j] = vs;
        a.scale[j] = expf(ps);
    }
    if (threadIdx.x >= visible) return;
    const size_t i = i0 + sh.row[threadIdx.x];
    float po = a.opac_logit[i], mo = a.m_opac[i], vo = a.v_opac[i];
    const float go = a.g_opac[i], so = a.opac[i];
    float q[4], qh[4], gh[4], mq[4], vq[4];
    load_w<4>(a.rot_raw + 4 * i, vec, q);
    load_w<4>(a.rot + 4 * i, vec, qh);
    load_w<4>(a.g_rot + 4 * i, vec, gh);
    load_w<4>(a.m_rot + 4 * i, vec, mq);
    load_w<4>(a.v_rot + 4 * i, vec, vq);
    // opacity: d/dlogit = d/dopacity * s (1 - s)
    adam_one(sh, 2, po, mo, vo, go * (so * (1.f - so)));
    a.opac_logit[i] = po; a.m_opac[i] = mo; a.v_opac[i] = vo;
    a.opac[i] = sigmoidf(po);
    // rotation: d/dq = (d/dq_hat - q_hat (q_hat . d/dq_hat)) / |q|
    float n2 = 0.f, dot = 0.f;
#pragma unroll
    for (int k = 0; k < 4; k++) n2 += q[k] * q[k];
    const float norm = fmaxf(sqrtf(n2), 1e-12f);
#pragma unroll
    for (int k = 0; k < 4; k++) dot += qh[k] * gh[k];
    float m2 = 0.f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        adam_one(sh, 4, q[k], mq[k], vq[k], (gh[k] - qh[k] * dot) / norm);
        m2 += q[k] * q[k];
    }
    const float nn = fmaxf(sqrtf(m2), 1e-12f);
#pragma unroll
    for (int k = 0; k < 4; k++) qh[k] = q[k] / nn;
    store_w<4>(a.rot_raw + 4 * i, vec, q);
    store_w<4>(a.m_rot + 4 * i, vec, mq);
    store_w<4>(a.v_rot + 4 * i, vec, vq);
    store_w<4>(a.rot + 4 * i, vec, qh);
}

// vec_rot / vec_sh: the quaternions / SH rows of every array start on 16-byte boundaries
// (vec_sh: an item is four floats, else one).
__global__ void __launch_bounds__(256)
    adam_kernel(fgs_adam_args a, const uint8_t* __restrict__ flag, const int* __restrict__ step, bool vec_rot,
                bool vec_sh, uint32_t per, uint32_t per_inv)
{
    __shared__ AdamShared sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t i0 = (size_t)blockIdx.x * 256, i = i0 + threadIdx.x;
    const bool on = i < (size_t)a.P && flag[i] != 0;
    const uint32_t mask = __ballot_sync(0xffffffffu, on);
    if (lane == 0) sh.count[warp] = __popc(mask);
    __syncthreads();
    uint32_t before = 0, visible = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        if (w < warp) before += sh.count[w];
        visible += sh.count[w];
    }
    if (visible == 0) return;
    if (on) sh.row[before + __popc(mask & ((1u << lane) - 1u))] = (uint8_t)threadIdx.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        sh.c = adam_coef(a.beta1, a.beta2, a.eps, *step);
        for (int k = 0; k < 5; k++) sh.ss[k] = (float)(a.lr[k] / sh.c.bc1);
    }
    if (blockIdx.y == 1) adam_small_rows(a, sh, i0, visible, vec_rot);
    else if (vec_sh) adam_sh_rows<4>(a, sh, i0, visible, per, per_inv);
    else adam_sh_rows<1>(a, sh, i0, visible, per, per_inv);
}

__global__ void step_tick_kernel(int* step) { *step += 1; }

namespace {
Window make_window()
{
    // loss.py:7-10: exp(-(x - 5)^2 / (2 * 1.5^2)) in double, stored as float32, normalised in float32
    float g[kWin], sum = 0.f;
    for (int i = 0; i < kWin; i++) {
        g[i] = (float)std::exp(-(double)((i - kWin / 2) * (i - kWin / 2)) / (2.0 * 1.5 * 1.5));
        sum += g[i];
    }
    Window w;
    for (int i = 0; i < kTaps; i++) {  // (the exponent is an integer squared: g[i] and g[10 - i] are equal)
        const float v[2] = {g[i] / sum, g[i] / sum};
        std::memcpy(&w.g[i], v, sizeof(F2));
    }
    return w;
}
}  // namespace

}  // namespace fgs

using namespace fgs;

extern "C" {

size_t fgs_loss_scratch_bytes(int width, int height)
{
    if (width <= kHalo || height <= kHalo) return 0;
    const size_t Wo = (size_t)width - kHalo, Ho = (size_t)height - kHalo;
    const size_t nso = 3 * ((Wo + kTX - 1) / kTX) * ((Ho + kSumRows - 1) / kSumRows);
    const size_t nl1 = 3 * (((size_t)width + kTX - 1) / kTX) * (((size_t)height + kSumRows - 1) / kSumRows);
    return sizeof(float) * (9 * ((Wo + 3) / 4 * 4) * Ho + nso + nl1) + 256;
}

int fgs_loss_l1_ssim(int width, int height, const float* pred, const float* target, float* dL_dpred,
                     float l1_grad_scale, float ssim_grad_scale, double* sums, void* scratch, void* stream)
{
    if (width <= kHalo || height <= kHalo || !pred || !target || !dL_dpred || !sums || !scratch) return FGS_ERR_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int Wo = width - kHalo, Ho = height - kHalo;
    // coefficient maps of 16-byte rows, from the first 16-byte boundary of the scratch
    float* gmap = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(scratch) + 15) & ~(uintptr_t)15);
    const int gpitch = (Wo + 3) / 4 * 4;
    const dim3 go((Wo + kTX - 1) / kTX, (Ho + kTY - 1) / kTY, 3);
    const dim3 gp((width + kTX - 1) / kTX, (height + kTY - 1) / kTY, 3);
    float* sp = gmap + (size_t)9 * gpitch * Ho;
    const int nso = (int)(3 * go.x) * ((Ho + kSumRows - 1) / kSumRows);
    const int nl1 = (int)(3 * gp.x) * ((height + kSumRows - 1) / kSumRows);
    float* l1p = sp + nso;
    static const Window win = make_window();
    const bool vec = width % 4 == 0 && ((reinterpret_cast<uintptr_t>(pred) | reinterpret_cast<uintptr_t>(target)) & 15u) == 0;
    if (vec)
        ssim_forward_kernel<true><<<go, kLossThreads, 0, s>>>(width, height, pred, target, win, ssim_grad_scale, gmap,
                                                              gpitch, sp);
    else
        ssim_forward_kernel<false><<<go, kLossThreads, 0, s>>>(width, height, pred, target, win, ssim_grad_scale, gmap,
                                                               gpitch, sp);
    loss_grad_kernel<<<gp, kLossThreads, 0, s>>>(width, height, pred, target, win, gmap, gpitch, l1_grad_scale,
                                                 dL_dpred, l1p);
    loss_reduce_kernel<<<1, 1024, 0, s>>>(l1p, nl1, sp, nso, sums);
    note_launches(3);
    return cudaGetLastError() == cudaSuccess ? FGS_OK : FGS_ERR_CUDA;
}

int fgs_train_activate(int P, const float* log_scale, const float* rot_raw, const float* opac_logit, float* scale,
                       float* rot, float* opac, void* stream)
{
    if (P < 0 || (P > 0 && (!log_scale || !rot_raw || !opac_logit || !scale || !rot || !opac))) return FGS_ERR_ARG;
    if (P == 0) return FGS_OK;
    activate_kernel<<<(P + 255) / 256 < 4096 ? (P + 255) / 256 : 4096, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        P, log_scale, rot_raw, opac_logit, scale, rot, opac);
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? FGS_OK : FGS_ERR_CUDA;
}

int fgs_densify_dense(int P, const int* radii, const float* dL_dmeans2D, float* grad_sum, int* vis_count,
                      unsigned char* flag, void* stream)
{
    if (P < 0 || (P > 0 && (!radii || !dL_dmeans2D || !grad_sum || !vis_count || !flag))) return FGS_ERR_ARG;
    if (P == 0) return FGS_OK;
    densify_dense_kernel<<<(P + 255) / 256 < 4096 ? (P + 255) / 256 : 4096, 256, 0,
                           static_cast<cudaStream_t>(stream)>>>(P, radii, dL_dmeans2D, grad_sum, vis_count, flag);
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? FGS_OK : FGS_ERR_CUDA;
}

int fgs_adam_step(const fgs_adam_args* a, const unsigned char* flag, int* step, void* stream)
{
    if (!a || !flag || !step || a->P < 0 || a->M < 0) return FGS_ERR_ARG;
    if (!a->xyz || !a->opac_logit || !a->log_scale || !a->rot_raw || !a->opac || !a->scale || !a->rot) return FGS_ERR_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    step_tick_kernel<<<1, 1, 0, s>>>(step);
    int n = 1;
    if (a->P > 0) {
        auto al = [](std::initializer_list<const void*> ps) {
            for (const void* p : ps)
                if (reinterpret_cast<uintptr_t>(p) & 15u) return false;
            return true;
        };
        const bool vec_rot = al({a->rot_raw, a->rot, a->g_rot, a->m_rot, a->v_rot});
        const uint32_t floats = a->shs ? 3u * (uint32_t)a->M : 0u;
        const bool vec_sh = floats % 4 == 0 && al({a->shs, a->m_shs, a->v_shs, a->g_shs});
        const uint32_t per = vec_sh ? floats / 4 : floats;
        const uint32_t per_inv = per ? (uint32_t)((0x100000000ull + per - 1) / per) : 0u;  // per is 0 or at least 3
        // (without SH rows the blocks of y = 0 would have nothing to do: y = 1 alone cannot be
        // launched, so they leave after the list)
        adam_kernel<<<dim3(((uint32_t)a->P + 255) / 256, 2), 256, 0, s>>>(*a, flag, step, vec_rot, vec_sh, per, per_inv);
        n++;
    }
    note_launches(n);
    return cudaGetLastError() == cudaSuccess ? FGS_OK : FGS_ERR_CUDA;
}

}  // extern "C"
