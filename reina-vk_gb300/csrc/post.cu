// Post-process kernels: bloom (shaders/postprocessing/bloom/{blurCommon.h,blurX.comp,blurY.comp,
// combine.comp}.glsl) and tone mapping (shaders/postprocessing/tonemap/tonemapping.comp.glsl), as
// Reina::applyBloom / applyTonemapping run them (src/Reina.cpp:472-577):
//   blurX(accum -> ping, with threshold)   blurY(ping), combine(accum, blurred), tonemap -> rgba8
// The reference's kernel has kernelSize = int(radiusPx * 3 + 0.5) taps on each side.  Its sums run over the taps
// in order (so do these), a NaN or infinite pixel spreads over the whole kernel as it does there, and the
// sum of the weights counts out-of-image and thresholded taps (blurCommon.h.glsl:24-31).
// 1920x1080, radius 5 (289 and 163 taps a side, 72 of them not zero): 0.152 ms, against 1.561 ms with a thread
// per pixel that summed every tap; 671x296, radius 0.86: 19 us against 37 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "launch_chain.cuh"
#include "post.h"

namespace rt {

constexpr int kPostBlock = 256;

// gauss(x, sigma) = exp(-x^2 / (2 sigma^2)) is exactly 0 in float beyond |x| = sqrt(2 * 104) |sigma| (exp(-104) is
// below half of the smallest subnormal): such taps add p * 0 to the sums, which changes them only where p
// is not finite.  The passes below therefore sum the `near` taps, |i| <= near, of the finite values (the others stand
// as zeros), and blocks that another value reaches add those to the sums afterwards, over the kernel's whole width
// (one NaN pixel: 1920x1080 at radius 5 0.163 ms, 0.602 ms when such blocks summed every tap; 320x200 at radius 9
// 50 us against 111 us).
static int near_taps(int K, float sigma) {
    const double reach = std::ceil(14.45 * std::fabs((double)sigma)) + 1.0;
    return reach < (double)K ? (int)reach : K;   // (a NaN sigma keeps K)
}

// Taps summed per step of the passes' unrolled loops, and outputs per thread: X, a window of kXOut + 3 pixels
// in registers takes 4 new ones per 4 taps; Y, a window of kYOut weights takes one new one per row.
constexpr int kXOut = 9, kXStep = kXOut + 3;
constexpr int kYOut = 12;
constexpr int kXChunk = 32 * kXOut;             // outputs of one warp in one channel
constexpr int kXSeg = 4 * kXChunk;              // an X block's outputs: consecutive pixels of a row
constexpr int kXThreads = 3 * 4 * 32;           // a warp per chunk and channel
constexpr int kYWarps = 4;    // a Y block's outputs: 48 consecutive rows of 32 columns
constexpr int kYRows = 24;    // rows of the input a Y block holds per stage of its ring
constexpr int kYStages = 3;
static_assert(kXSeg % 32 == 0, "a Y block's columns lie in one X segment");
constexpr int kWeightPart = 1024;   // weights summed from shared memory at a time
constexpr size_t kXMaxShared = 200 * 1024;

struct BloomTaps {
    int K, near;      // kernel half-width, and the half-width of its non-zero taps
    float* w;         // X: padded behind, Y: on both sides, with zeros (w_at)
    float* sum;       // float sum of the weights for x = -K..K, in that order
};
static size_t x_words(int near) { return (size_t)(2 * near + 1 + kXStep + 3) / 4 * 4; }
static size_t y_words(int near) { return (size_t)(2 * near + 1 + 3 * kYOut + 3) / 4 * 4; }

// Both passes' weights, one block each: the exponentials in parallel, their sum by one thread in order (the
// zero taps leave it as it is).  One thread for all of it took 47 us at 1920x1080 and radius 5.
__global__ void __launch_bounds__(kPostBlock) k_bloom_weights(BloomTaps tx, BloomTaps ty, int x_total, int y_total, float sigma) {
    let_next_start();
    const bool X = blockIdx.x == 0;
    const BloomTaps t = X ? tx : ty;
    const int total = X ? x_total : y_total, pad = X ? 0 : kYOut, n = 2 * t.near + 1;
    for (int k = threadIdx.x; k < total; k += blockDim.x) {
        const int i = k - pad;
        float g = 0.0f;
        if (i >= 0 && i < n) {
            const float x = (float)(i - t.near);
            g = expf(-x * x / (2.0f * sigma * sigma));
        }
        t.w[k] = g;
    }
    __shared__ float part[kWeightPart];
    float sum = 0.0f;
    for (int base = 0; base < n; base += kWeightPart) {
        const int m = min(kWeightPart, n - base);
        __syncthreads();
        for (int k = threadIdx.x; k < m; k += blockDim.x) part[k] = t.w[pad + base + k];
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll 8
            for (int i = 0; i < m; ++i) sum += part[i];
        }
    }
    if (threadIdx.x == 0) *t.sum = sum;
}

// c / wsum.  A quotient of a tiny c would take the division's slow path, and where little passes the threshold
// most sums are zeros or the Gaussian's tails: those are divided at 2^64 times their size.  Scaled back, a
// subnormal quotient is rounded a second time, which goes wrong only where the first one left it midway between
// two subnormals: settle() lets the division's remainder decide on which side of the midpoint it lies.  (Leaving
// subnormal quotients to the plain division took 33 us instead of 19 us for 671x296 at radius 0.86 with few
// pixels above the threshold.)  The reference's guard against weight sums below 0.0001 has nothing to guard: the
// middle weight is exp(-0) = 1, or the sum is NaN (radius 0), and so are the image's pixels.
struct Mean {
    float n, q, r;   // scaled dividend and quotient, c / wsum but for settle()
    __device__ __forceinline__ Mean(float c, float wsum) {
        const bool tiny = fabsf(c) < 0x1p-60f, zero = c == 0.0f;
        n = zero ? wsum : (tiny ? c * 0x1p64f : c);
        q = n / wsum;
        r = zero ? c : (tiny ? q * 0x1p-64f : q);
    }
    __device__ __forceinline__ void settle(float wsum) {
        const float left = q - r * 0x1p64f, rest = fmaf(-q, wsum, n);   // exact where r is subnormal
        if (fabsf(left) == 0x1p-86f && rest != 0.0f && (rest > 0.0f) == (left > 0.0f)) r += copysignf(0x1p-149f, left);
    }
};
constexpr float kSettle = 0x1p-62f;   // means with |q| below it may be subnormal
__device__ __forceinline__ bool not_finite(float a, float b, float c) {
    return !(fabsf(a) < INFINITY && fabsf(b) < INFINITY && fabsf(c) < INFINITY);
}

// a ka + b kb + c kc with the products fused so.  The sums of three products below say which product is rounded by
// itself: left to the compiler that changed with the code around them, and bytes of the image with it.
__device__ __forceinline__ float sum3(float a, float ka, float b, float kb, float c, float kc) {
    return __fmaf_rn(c, kc, __fmaf_rn(a, ka, __fmul_rn(b, kb)));
}
__device__ __forceinline__ bool below(const float4& p, float threshold) {
    return sum3(p.x, 0.299f, p.y, 0.587f, p.z, 0.114f) < threshold;
}

// What the values that a warp left out of its sums (they are not finite) add to them: to every output they reach, at
// weight zero NaN.  stage: the warp's sums of channel ch for the pixels from xw on.  (This function and its like for
// blurY stay out of line: inlined they cost every block a microsecond of instruction fetches.)
__device__ __noinline__ void add_not_finite_x(float* stage, const float4* __restrict__ src, int W, int xw, int xe, int ch,
                                              const BloomTaps t, float threshold) {
    const int lane = threadIdx.x & 31;
    auto weight = [&](int d) { return d < -t.near || d > t.near ? 0.0f : t.w[t.near + d]; };
    auto value = [&](int x) {
        const float4 p = __ldg(src + x);
        return below(p, threshold) ? 0.0f : (ch == 0 ? p.x : (ch == 1 ? p.y : p.z));
    };
    uint32_t nan_to = 0u;   // outputs xw + 32 k + lane that a NaN reaches
    const int first = max(0, xw - t.K), last = min(W - 1, min(xw + kXChunk, xe) - 1 + t.K);
    bool infinite = false;
    for (int pass = 0; pass < 2; ++pass) {   // NaNs; then infinities, if there are any
#pragma unroll 2
        for (int x32 = first; x32 <= last; x32 += 32) {
            const float v = x32 + lane <= last ? value(x32 + lane) : 0.0f;
            infinite = infinite || fabsf(v) == INFINITY;
            for (uint32_t m = __ballot_sync(0xFFFFFFFFu, pass == 0 ? !(v == v) : fabsf(v) == INFINITY); m; m &= m - 1u) {
                const int from = __ffs(m) - 1, at = x32 + from;
                const float u = __shfl_sync(0xFFFFFFFFu, v, from);
#pragma unroll 1
                for (int k = 0; k < kXOut; ++k) {
                    const int x = xw + 32 * k + lane, d = at - x;
                    if (d < -t.K || d > t.K || x >= xe) continue;
                    if (pass == 0) nan_to |= 1u << k;
                    else stage[32 * k + lane] += u * weight(d);
                }
            }
        }
        if (pass == 1 || !__any_sync(0xFFFFFFFFu, infinite)) break;
#pragma unroll 1
        for (int k = 0; k < kXOut; ++k) {   // finite values whose sum overflows: in order, the infinities among them
            const int x = xw + 32 * k + lane;
            if (x >= xe || !not_finite(stage[32 * k + lane], 0.0f, 0.0f)) continue;
            float sum = 0.0f;
            for (int i = max(-t.K, -x); i <= min(t.K, W - 1 - x); ++i) sum += value(x + i) * weight(i);
            stage[32 * k + lane] = sum;
        }
    }
    for (; nan_to; nan_to &= nan_to - 1u) stage[32 * (__ffs(nan_to) - 1) + lane] = NAN;
    __syncwarp();
}

// blurX of one segment (kXSeg pixels) of a row per block, into one plane per channel.  The thresholded pixels of
// the segment and its `near` neighbours lie in shared memory, a plane per channel (zeros stand for taps
// outside the image, below the threshold and not finite); a warp has a channel of a quarter of the segment (four
// warps that took the channels in turn left a small image's few blocks waiting: 671x296 at radius 0.86, 43 us a
// call, 34 us so), and a thread sums kXOut neighbouring outputs from a register window, so a tap costs kXOut FMAs,
// one shared load and a quarter of a weight load (kXOut is odd: the threads' windows start in different banks).  A
// warp's outputs go through shared memory to leave in full lines.  The pixels that only taps of weight zero reach
// are read for values that are not finite.  Bound by the FP32 issue rate.
__global__ void __launch_bounds__(kXThreads, 3) k_blur_x(const float4* __restrict__ in, float* __restrict__ out, int W, int H, int pitch,
                                                         size_t plane, BloomTaps t, float threshold, int* __restrict__ flags) {
    extern __shared__ float row[];
    const int y = (int)(blockIdx.x % (unsigned)H), seg = (int)(blockIdx.x / (unsigned)H);
    const int xs = seg * kXSeg, xe = min(W, xs + kXSeg);
    const int stride = xe - xs + 2 * t.near + 2 * kXStep;   // plane length: from pixel xs - near, and zeros behind
    const float4* src = in + (size_t)y * W;
    float* dst = out + (size_t)y * pitch;
    bool bad = false;
#pragma unroll 4
    for (int j = threadIdx.x; j < stride; j += kXThreads) {
        const int x = xs + j - t.near;
        float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (x >= 0 && x < W) p = __ldg(src + x);
        if (below(p, threshold)) p.x = p.y = p.z = 0.0f;
        if (not_finite(p.x, p.y, p.z)) {
            bad = true;
            p.x = not_finite(p.x, 0.0f, 0.0f) ? 0.0f : p.x;
            p.y = not_finite(p.y, 0.0f, 0.0f) ? 0.0f : p.y;
            p.z = not_finite(p.z, 0.0f, 0.0f) ? 0.0f : p.z;
        }
        row[j] = p.x;
        row[stride + j] = p.y;
        row[2 * stride + j] = p.z;
    }
    const int far = t.K - t.near;
    for (int j = threadIdx.x; j < 2 * far; j += blockDim.x) {
        const int x = j < far ? xs - t.K + j : xe + t.near + (j - far);
        if (x < 0 || x >= W) continue;
        const float4 p = __ldg(src + x);
        bad = bad || (!below(p, threshold) && not_finite(p.x, p.y, p.z));
    }
    wait_for_previous();   // the weights; the pixels above were there before the call's first kernel began
    const float wsum = *t.sum;
    const int any_bad = __syncthreads_or(bad ? 1 : 0);
    bool flag = false;
    const int steps = (2 * t.near + 1 + kXStep - 1) / kXStep;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ch = warp / 4;
    float* stage = row + 3 * stride + warp * kXChunk;
    const int x0 = (warp % 4) * kXChunk, xw = xs + x0;   // the warp's first output
    if (xw < xe) {
        float acc[kXOut], win[kXStep];   // win[k % kXStep] holds v[k]
#pragma unroll
        for (int r = 0; r < kXOut; ++r) acc[r] = 0.0f;
        if (xw + lane * kXOut < xe) {
            const float* v = row + ch * stride + x0 + lane * kXOut;   // output r sums v[r + i] w[i], i in order
            const float4* w4 = reinterpret_cast<const float4*>(t.w);
#pragma unroll
            for (int r = 0; r < kXOut; ++r) win[r] = v[r];
#pragma unroll 1
            for (int s = 0; s < steps; ++s) {
#pragma unroll
                for (int g = 0; g < kXStep / 4; ++g) {
                    const float4 wg = __ldg(w4 + g);
                    const float wk[4] = {wg.x, wg.y, wg.z, wg.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int i = 4 * g + k;
                        win[(i + kXOut) % kXStep] = v[i + kXOut];
#pragma unroll
                        for (int r = 0; r < kXOut; ++r) acc[r] += win[(i + r) % kXStep] * wk[k];
                    }
                }
                v += kXStep;
                w4 += kXStep / 4;
            }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kXOut; ++r) stage[lane * kXOut + r] = acc[r];
        __syncwarp();
        if (any_bad) add_not_finite_x(stage, src, W, xw, xe, ch, t, threshold);
#pragma unroll
        for (int k = 0; k < kXOut; ++k) {
            const int x = xw + 32 * k + lane;
            if (x >= xe) break;
            Mean m(stage[32 * k + lane], wsum);
            if (fabsf(m.q) < kSettle) m.settle(wsum);
            flag = flag || !(fabsf(m.r) < INFINITY);
            dst[ch * plane + x] = m.r;
        }
    }
    const int any_flag = __syncthreads_or(flag ? 1 : 0);
    if (threadIdx.x == 0) flags[(size_t)seg * H + y] = any_flag;
}

// blurX of `rows` whole rows or, with rows = 1, of one segment of a row per block, a thread per output, every tap
// read from memory and summed in order as the reference does: kernels too wide for a block's shared memory, and
// images so narrow that a block per row would be nearly empty (below 32 pixels: 1x65536 at radius 0.05 252 us with
// k_blur_x and 45 us here, 24x20000 at radius 0.1 92 and 33 us; 31x31 the same).
__global__ void __launch_bounds__(kXThreads) k_blur_x_all_taps(const float4* __restrict__ in, float* __restrict__ out, int W, int H,
                                                               int pitch, size_t plane, BloomTaps t, float threshold,
                                                               int* __restrict__ flags, int rows) {
    __shared__ int row_flags[kXThreads];
    const unsigned blocks = (unsigned)((H + rows - 1) / rows);
    const int y0 = (int)(blockIdx.x % blocks) * rows, seg = (int)(blockIdx.x / blocks);
    const int xs = seg * kXSeg, n = min(W, xs + kXSeg) - xs;
    if ((int)threadIdx.x < rows) row_flags[threadIdx.x] = 0;
    wait_for_previous();
    const float wsum = *t.sum;
    __syncthreads();
    for (int j = threadIdx.x; j < min(rows, H - y0) * n; j += kXThreads) {
        const int dy = j / n, x = xs + j % n;
        const float4* src = in + (size_t)(y0 + dy) * W;
        float* dst = out + (size_t)(y0 + dy) * pitch + x;
        float cr = 0.0f, cg = 0.0f, cb = 0.0f;
        const int i0 = max(-t.K, -x), i1 = min(t.K, W - 1 - x);
        for (int i = i0; i <= i1; ++i) {
            const float4 p = __ldg(src + x + i);
            if (below(p, threshold)) continue;
            const float wgt = i < -t.near || i > t.near ? 0.0f : t.w[t.near + i];
            cr += p.x * wgt;
            cg += p.y * wgt;
            cb += p.z * wgt;
        }
        Mean mr(cr, wsum), mg(cg, wsum), mb(cb, wsum);
        mr.settle(wsum);
        mg.settle(wsum);
        mb.settle(wsum);
        if (not_finite(mr.r, mg.r, mb.r)) row_flags[dy] = 1;
        dst[0] = mr.r;
        dst[plane] = mg.r;
        dst[2 * plane] = mb.r;
    }
    __syncthreads();
    if ((int)threadIdx.x < min(rows, H - y0)) flags[(size_t)seg * H + y0 + threadIdx.x] = row_flags[threadIdx.x];
}

// combine.comp.glsl:15-27 then tonemapping.comp.glsl:66-84 (exposure, ACES fitted, clamp, RGBA8 UNORM).
__device__ __forceinline__ uint8_t to_unorm8(float v) {
    if (!(v == v)) return 0;   // NaN stores as 0
    v = fminf(fmaxf(v, 0.0f), 1.0f);
    return (uint8_t)__float2uint_rn(v * 255.0f);
}

__device__ __forceinline__ float3 aces_fitted(float3 c) {
    // color * ACESInputMat: GLSL row vector times a matrix built from columns -> dot with each column
    float3 v = make_float3(sum3(c.x, 0.59719f, c.y, 0.35458f, c.z, 0.04823f), sum3(c.x, 0.07600f, c.y, 0.90834f, c.z, 0.01566f),
                           sum3(c.x, 0.02840f, c.y, 0.13383f, c.z, 0.83777f));
    auto fit = [](float x) {
        const float a = __fmaf_rn(x, x + 0.0245786f, -0.000090537f);
        const float b = __fmaf_rn(x, __fmaf_rn(0.983729f, x, 0.4329510f), 0.238081f);
        return a / b;
    };
    v = make_float3(fit(v.x), fit(v.y), fit(v.z));
    return make_float3(sum3(v.x, 1.60475f, v.y, -0.53108f, v.z, -0.07367f), sum3(v.y, 1.10813f, v.x, -0.10208f, v.z, -0.00605f),
                       sum3(v.x, -0.00327f, v.y, -0.07276f, v.z, 1.07602f));
}

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// The same for a thread's kYOut outputs of blurY.
constexpr int kSumCh = 32 * kYWarps;
__device__ __noinline__ void add_not_finite(float* sums, const float* __restrict__ blurred_x, int pitch, size_t plane, int W, int H,
                                            int x, int y0, const BloomTaps t, const int* __restrict__ flags) {
    const int lane = threadIdx.x & 31;
    auto weight = [&](int d) { return d < -t.near || d > t.near ? 0.0f : __ldg(t.w + kYOut + t.near + d); };
    const int first = max(0, y0 - t.K), last = min(H - 1, y0 + kYOut - 1 + t.K);
    uint32_t nan_to[3] = {0u, 0u, 0u};   // per channel: outputs that a NaN reaches
    bool infinite = false;
    for (int pass = 0; pass < 2; ++pass) {   // NaNs; then infinities, if there are any
        for (int y32 = first; y32 <= last; y32 += 32) {   // a lane per row's flag, then the flagged rows, four at a time
            const bool flagged = y32 + lane <= last && __ldg(flags + (size_t)((x - lane) / kXSeg) * H + y32 + lane) != 0;
            for (uint32_t m = __ballot_sync(0xFFFFFFFFu, flagged); m;) {
                int ys[4];
                float v[4][3];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    ys[j] = m ? y32 + __ffs(m) - 1 : -1;
                    m &= m - 1u;
                    const float* p = blurred_x + (size_t)ys[j] * pitch + x;
                    for (int ch = 0; ch < 3; ++ch) v[j][ch] = ys[j] >= 0 && x < W ? __ldg(p + ch * plane) : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int r0 = max(0, ys[j] - t.K - y0), r1 = min(kYOut - 1, ys[j] + t.K - y0);
                    for (int ch = 0; ch < 3; ++ch) {
                        infinite = infinite || fabsf(v[j][ch]) == INFINITY;
                        if (pass == 0 && !(v[j][ch] == v[j][ch])) nan_to[ch] |= (2u << r1) - (1u << r0);
                        if (pass == 1 && fabsf(v[j][ch]) == INFINITY)
                            for (int r = r0; r <= r1; ++r) sums[(3 * r + ch) * kSumCh] += v[j][ch] * weight(ys[j] - y0 - r);
                    }
                }
            }
        }
        if (pass == 1 || !__any_sync(0xFFFFFFFFu, infinite)) break;
#pragma unroll 1
        for (int k = 0; k < 3 * kYOut && x < W; ++k) {   // finite values whose sum overflows: in order, the infinities among them
            if (!not_finite(sums[k * kSumCh], 0.0f, 0.0f)) continue;
            const float* p = blurred_x + (k % 3) * plane + x;
            const int at = y0 + k / 3;
            float sum = 0.0f;
            for (int y = max(first, at - t.K); y <= min(last, at + t.K); ++y) sum += __ldg(p + (size_t)y * pitch) * weight(y - at);
            sums[k * kSumCh] = sum;
        }
    }
    for (int ch = 0; ch < 3; ++ch)
        for (; nan_to[ch]; nan_to[ch] &= nan_to[ch] - 1u) sums[(3 * (__ffs(nan_to[ch]) - 1) + ch) * kSumCh] = NAN;
}

// blurY, combine and tone map: a lane per column, kYOut consecutive rows per thread, 32 columns x 48 rows a block.
// The input rows pass through a shared-memory ring filled by asynchronous copies (rows outside the image
// as zeros); every row a warp reads feeds kYOut sums, whose weights move through a register window, so a row
// costs 3 kYOut FMAs and three shared loads.  The blurred value stays in the registers and the bloomed and
// tone-mapped pixels are written at once (the former passes wrote and re-read a blurred image).  Bound by
// the FP32 issue rate (66 % of the issue slots used); the same loop over rows read from L1 and L2 by each warp
// waited on them (164 us against 84 us under the profiler, 1920x1080 at radius 5).
__global__ void __launch_bounds__(32 * kYWarps, 6) k_blur_y_tonemap(const float* __restrict__ blurred_x, int pitch, size_t plane,
                                                                    const float4* __restrict__ orig, float4* __restrict__ combined,
                                                                    uchar4* __restrict__ out, int W, int H, BloomTaps t,
                                                                    const int* __restrict__ flags, float intensity,
                                                                    float exposure_scale) {
    __shared__ __align__(16) float ring[kYStages][kYRows * 3 * 32];   // [row][channel][column]
    const int cols = (W + 31) / 32;   // blocks per row of blocks
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = (int)(blockIdx.x % cols) * 32 + lane;
    const int yb = (int)(blockIdx.x / cols) * (kYOut * kYWarps);
    const int y0 = yb + warp * kYOut;
    wait_for_previous();
    const float wsum = *t.sum;
    // rows that a tap of this block reaches and that hold a value that is not finite
    bool bad = false;
    const int f0 = max(0, yb - t.K), f1 = min(H - 1, yb + kYOut * kYWarps - 1 + t.K);
    for (int y = f0 + (int)threadIdx.x; y <= f1; y += blockDim.x)
        bad = bad || __ldg(flags + (size_t)((x - lane) / kXSeg) * H + y) != 0;
    const int any_bad = __syncthreads_or(bad ? 1 : 0);
    // the sums of a thread's outputs, [output][channel][thread] over the ring once it is read: the epilogue then loops
    // (unrolled over the outputs with their divisions it had a small image wait on instruction fetches)
    float* sums = &ring[0][0] + threadIdx.x;
    static_assert(sizeof(ring) >= sizeof(float) * kYOut * 3 * kSumCh);
    float cr[kYOut], cg[kYOut], cb[kYOut];
#pragma unroll
    for (int r = 0; r < kYOut; ++r) cr[r] = cg[r] = cb[r] = 0.0f;
    // chunk c: rows [yb - near + kYRows c, + kYRows); those with a row of the image only
    const int base = yb - t.near;
    const int c0 = base < 0 ? -base / kYRows : 0;
    const int c1 = (min(2 * t.near + kYOut * kYWarps, H - base) + kYRows - 1) / kYRows;
    const float* col = blurred_x + (x - lane);
    auto fill = [&](int c) {
        if (c < c1) {
            float* dst = ring[c % kYStages];
            for (int k = threadIdx.x; k < kYRows * 3 * 8; k += 32 * kYWarps) {
                const int row = k / 24, ch = k / 8 % 3, part = k % 8, y = base + c * kYRows + row;
                const bool in_image = y >= 0 && y < H && x - lane + 4 * part < pitch;
                copy16_or_zero(dst + 4 * k, in_image ? col + ch * plane + (size_t)y * pitch + 4 * part : blurred_x, in_image);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int c = 0; c < kYStages - 1; ++c) fill(c0 + c);
    float win[kYOut];   // win[(s - r) mod kYOut]: the weight of step s (row y0 - near + s) for output r
#pragma unroll
    for (int r = 0; r < kYOut; ++r) win[r] = 0.0f;
    bool begun = false;
    for (int c = c0; c < c1; ++c) {
        fill(c + kYStages - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(kYStages - 1) : "memory");
        __syncthreads();
        if (any_bad) {   // values that are not finite are left out here: the window pads the kernel with zeros
            float* chunk = ring[c % kYStages];
            for (int k = threadIdx.x; k < kYRows * 3 * 32; k += 32 * kYWarps)
                if (not_finite(chunk[k], 0.0f, 0.0f)) chunk[k] = 0.0f;
            __syncthreads();
        }
#pragma unroll 1
        for (int g = 0; g < kYRows / kYOut; ++g) {
            const int s = c * kYRows + g * kYOut - warp * kYOut;
            if (s < 0 || s >= 2 * t.near + kYOut) continue;
            const float* w = t.w + kYOut + s;   // zeros before and after the 2 near + 1 weights
            if (!begun) {   // the window before this warp's first step
#pragma unroll
                for (int r = 1; r < kYOut; ++r) win[kYOut - r] = __ldg(w - r);
                begun = true;
            }
            const float* p = ring[c % kYStages] + g * (kYOut * 3 * 32) + lane;
            float4 wg;
#pragma unroll
            for (int k = 0; k < kYOut; ++k) {
                if (k % 4 == 0) wg = __ldg(reinterpret_cast<const float4*>(w + k));
                win[k] = k % 4 == 0 ? wg.x : (k % 4 == 1 ? wg.y : (k % 4 == 2 ? wg.z : wg.w));
                const float pr = p[(3 * k + 0) * 32], pg = p[(3 * k + 1) * 32], pb = p[(3 * k + 2) * 32];
#pragma unroll
                for (int r = 0; r < kYOut; ++r) {
                    const float wgt = win[(k - r + kYOut) % kYOut];
                    cr[r] += pr * wgt;
                    cg[r] += pg * wgt;
                    cb[r] += pb * wgt;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kYOut; ++r) {
        sums[(3 * r + 0) * kSumCh] = cr[r];
        sums[(3 * r + 1) * kSumCh] = cg[r];
        sums[(3 * r + 2) * kSumCh] = cb[r];
    }
    if (any_bad) add_not_finite(sums, blurred_x, pitch, plane, W, H, x, y0, t, flags);
    if (x >= W) return;
    const int rows = min(kYOut, H - y0);
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
        const size_t i = (size_t)(y0 + r) * W + x;
        const float4 o = __ldg(orig + i);
        Mean mr(sums[(3 * r + 0) * kSumCh], wsum), mg(sums[(3 * r + 1) * kSumCh], wsum), mb(sums[(3 * r + 2) * kSumCh], wsum);
        if (fminf(fminf(fabsf(mr.q), fabsf(mg.q)), fabsf(mb.q)) < kSettle) {   // one branch for the three
            mr.settle(wsum);
            mg.settle(wsum);
            mb.settle(wsum);
        }
        const float3 c = make_float3(o.x + mr.r * intensity, o.y + mg.r * intensity, o.z + mb.r * intensity);
        if (combined) combined[i] = make_float4(c.x, c.y, c.z, 1.0f);
        const float3 m = aces_fitted(make_float3(c.x * exposure_scale, c.y * exposure_scale, c.z * exposure_scale));
        out[i] = make_uchar4(to_unorm8(m.x), to_unorm8(m.y), to_unorm8(m.z), 255);
    }
}

void PostWorkspace::ensure(size_t pixels, size_t words) {
    if (pixels > cap_px_) {
        ping.alloc(pixels * 3 * sizeof(float));
        cap_px_ = pixels;
    }
    if (words > cap_w_) {
        weights.alloc(words * sizeof(float));
        cap_w_ = words;
    }
}

static int bloom_kernel_size(int side, float radius) {
    const float radius_px = (float)side * radius / 100.0f;   // blurCommon.h.glsl:19
    return (int)(radius_px * 3.0f + 0.5f);
}

void postprocess(PostWorkspace& ws, const float* d_accum, int W, int H, const BloomPushConsts& bloom,
                 const TonemappingPushConsts& tm, uint8_t* d_rgba8, float* d_combined, cudaStream_t st) {
    const size_t n = (size_t)W * H;
    if (n == 0) return;
    BloomTaps tx{}, ty{};
    tx.K = bloom_kernel_size(W, bloom.radius);
    ty.K = bloom_kernel_size(H, bloom.radius);
    if (tx.K < 0 || ty.K < 0 || tx.K > (1 << 20) || ty.K > (1 << 20)) fail(REINA_ERR_INVALID, "bloom radius out of range");
    tx.near = near_taps(tx.K, bloom.radius);
    ty.near = near_taps(ty.K, bloom.radius);
    // one buffer: the two sums, both weight tables (16-byte aligned), a flag per row and X segment
    const size_t xw = x_words(tx.near), yw = y_words(ty.near);
    const int pitch = (W + 3) / 4 * 4;   // blurX's rows start on 16 bytes
    const size_t plane = (size_t)pitch * H;
    const int segs = (W + kXSeg - 1) / kXSeg;
    ws.ensure(plane, 4 + xw + yw + (size_t)segs * H);
    float* buf = ws.weights.as<float>();
    tx.sum = buf;
    ty.sum = buf + 1;
    tx.w = buf + 4;
    ty.w = tx.w + xw;
    int* flags = reinterpret_cast<int*>(ty.w + yw);
    const float4* accum = reinterpret_cast<const float4*>(d_accum);
    // The three kernels of a call are chained by programmatic launches, which take a launch's latency out of each gap
    // (671x296, radius 2: 27.8 us without, 22.8 us with): a kernel waits (wait_for_previous) before it reads what
    // the one before it wrote.  The first is launched plainly, so nothing of a call starts before the work ahead of it
    // on the stream is done, and it lets blurX start at once, whose blocks load their pixels meanwhile.  blurX does
    // not: blurY's blocks would fill the slots that blurX leaves on some SMs and crowd there (35 us).
    k_bloom_weights<<<2, kPostBlock, 0, st>>>(tx, ty, (int)xw, (int)yw, bloom.radius);
    check_cuda(cudaGetLastError(), "postprocess launch");
    float* ping = ws.ping.as<float>();
    const size_t shared = sizeof(float) * (3 * ((size_t)std::min(W, kXSeg) + 2 * (size_t)tx.near + 2 * kXStep) + 3 * kXSeg);
    // Images up to 31 pixels wide give a block of the general form little to do but its launch and its barriers.
    const int rows = W < 32 ? kXThreads / W : 1;
    if (rows == 1 && shared <= kXMaxShared) {
        if (shared > 48 * 1024)
            check_cuda(cudaFuncSetAttribute(k_blur_x, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kXMaxShared),
                       "cudaFuncSetAttribute");
        launch_after(k_blur_x, (unsigned)segs * (unsigned)H, kXThreads, shared, st, accum, ping, W, H, pitch, plane, tx, bloom.threshold,
                     flags);
    } else {
        launch_after(k_blur_x_all_taps, (unsigned)segs * (unsigned)((H + rows - 1) / rows), kXThreads, 0, st, accum, ping, W, H, pitch,
                     plane, tx, bloom.threshold, flags, rows);
    }
    const unsigned blocks = (unsigned)((W + 31) / 32) * (unsigned)((H + kYOut * kYWarps - 1) / (kYOut * kYWarps));
    launch_after(k_blur_y_tonemap, blocks, 32 * kYWarps, 0, st, ping, pitch, plane, accum, reinterpret_cast<float4*>(d_combined),
                 reinterpret_cast<uchar4*>(d_rgba8), W, H, ty, flags, bloom.intensity, exp2f(tm.exposure));
}

}  // namespace rt
