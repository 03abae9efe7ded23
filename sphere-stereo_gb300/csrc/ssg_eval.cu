// Evaluation of RGB-D panoramas against ground truth (python/utils.py:206-250): PSNR and SSIM of
// the colour panorama, MAE, RMSE and bad-pixel ratios of the inverse-distance panorama, for a
// batch of frames, as device reductions.
//
// The metrics follow scikit-image's published definitions as the reference calls them
// (structural_similarity(gt, est, multichannel=True) and peak_signal_noise_ratio(gt, est) on
// float32 images in [0, 1]) and numpy's element-wise arithmetic:
//   - colour values x = u8 / 255 in float32;
//   - PSNR: mse = mean over all values of the float32 square of the float32 difference, summed in
//     float64; psnr = 10 log10(1 / mse) (data range 1: float images with no negative value);
//   - SSIM per channel on float64 values: 7x7 uniform windows, sample covariances (49 / 48),
//     data range 2 (the float dtype's range -1..1), C1 = (0.01 * 2)^2, C2 = (0.03 * 2)^2, the
//     map cropped by 3 pixels on each side and averaged; the mean over the 3 channels;
//   - err = |est - gt| in float32; MAE = sum(err) / n, RMSE = sqrt(sum(err * err) / n) with the
//     float32 products summed in float64; bad-pixel ratio = 100 * count(err > t) / n, t rounded to
//     float32 as numpy compares a float32 array with a Python float.
// Sums are taken per block in a fixed order and reduced in a fixed order, so results do not
// depend on scheduling.
#include <algorithm>

#include "ssg_common.cuh"

namespace ssg {

constexpr int kEvalBlocks = 304;  // blocks per frame: two per SM
constexpr int kEvalThreads = 256;
constexpr int kEvalWarps = kEvalThreads / 32;
constexpr int kSsimWin = 7, kSsimHalf = 3;

struct EvalParams {
    int cols, rows, frames, thresholds;
    float threshold[SSG_EVAL_MAX_THRESHOLDS];
};

// slots of a block's partial sums
enum { kSlotSq = 0, kSlotErr = 1, kSlotErr2 = 2, kSlotSsim = 3, kSlotBad = 4 };

__device__ __forceinline__ int eval_slots(const EvalParams& p) { return kSlotBad + p.thresholds; }

// fixed-order sum of one value per thread of the block (thread 0 returns it)
__device__ __forceinline__ double block_sum(double v, double* sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();  // sh is free
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
    return s;
}

__device__ __forceinline__ float unit_value(uint8_t v) { return __fdiv_rn((float)v, 255.0f); }

// FP64 runs at a sixty-fourth of the FP32 rate on this GPU (an FP64 operation per colour value of a
// 2048x1024 panorama costs 11 us), so the sums are kept without it: colour errors as exact
// integers, distance errors and SSIM values in two floats.

// s.hi + s.lo += v (and + low), the rounding error of the sum kept in lo (Knuth's TwoSum, "The Art of
// Computer Programming" vol. 2, 4.2.2).  The sum has to stay in float32's range.
struct TwoFloat {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float v, float low = 0.0f)
    {
        const float t = __fadd_rn(hi, v), b = __fsub_rn(t, hi);
        lo += (__fsub_rn(hi, __fsub_rn(t, b)) + __fsub_rn(v, b)) + low;
        hi = t;
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Sum of float32 squares d2 in [0, 1] that are multiples of 2^-40, exact: every d2 is split into a
// multiple of 2^-23 (the sum 1 + d2) and the rest (a multiple of 2^-40 below 2^-24), both read from
// the bits of float sums.
struct SquareSum {
    uint32_t hi = 0, lo = 0;  // of at most 64 values, with the bits of the two biases
    __device__ __forceinline__ void add(float d2)
    {
        const float r = __fadd_rn(d2, 1.0f);
        hi += __float_as_uint(r) - 0x3F800000u;
        const float rest = __fsub_rn(d2, __fsub_rn(r, 1.0f));
        lo += __float_as_uint(__fmaf_rn(rest, 1099511627776.0f, 12582912.0f)) - 0x4B400000u;
    }
    __device__ __forceinline__ long long units() const  // multiples of 2^-40
    {
        return ((long long)hi << 17) + (long long)(int32_t)lo;
    }
};

// Per-pixel sums: squared colour differences, inverse-distance errors and bad-pixel counts.
// blockIdx.y: frame.  kVec: the frame's arrays are read 16 bytes at a time (all four 16-byte aligned
// in every frame).  Bound by instruction issue: 4 frames of 2048x1024 (117 MB) 450 -> 57 us.
template <bool kVec>
__global__ void __launch_bounds__(kEvalThreads) eval_pointwise_kernel(const __grid_constant__ EvalParams p,
                                                                      const uint8_t* __restrict__ rgb,
                                                                      const uint8_t* __restrict__ gt_rgb,
                                                                      const float* __restrict__ inv,
                                                                      const float* __restrict__ gt_inv,
                                                                      double* __restrict__ partials)
{
    __shared__ double sh[kEvalWarps];
    __shared__ float unit[256];  // u8 / 255
    unit[threadIdx.x] = unit_value((uint8_t)threadIdx.x);
    __syncthreads();
    const int64_t n = (int64_t)p.cols * p.rows, bytes = 3 * n;
    const int frame = blockIdx.y;
    rgb += frame * bytes;
    gt_rgb += frame * bytes;
    inv += frame * n;
    gt_inv += frame * n;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    const auto square = [&](uint32_t g, uint32_t e) {
        const float d = __fsub_rn(unit[g], unit[e]);
        return __fmul_rn(d, d);
    };
    long long sq = 0;  // multiples of 2^-40
    const int64_t groups = kVec ? bytes / 16 : 0;
    for (int64_t i = first; i < groups; i += stride) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(gt_rgb) + i), b = __ldg(reinterpret_cast<const uint4*>(rgb) + i);
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
        SquareSum s;
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int k = 0; k < 4; ++k) s.add(square((aw[w] >> (8 * k)) & 255u, (bw[w] >> (8 * k)) & 255u));
        sq += s.units();
    }
    for (int64_t i = 16 * groups + first; i < bytes; i += stride) {
        SquareSum s;
        s.add(square(__ldg(gt_rgb + i), __ldg(rgb + i)));
        sq += s.units();
    }
    TwoFloat err, err2;
    float largest = 0.0f;
    int bad[SSG_EVAL_MAX_THRESHOLDS];
#pragma unroll
    for (int k = 0; k < SSG_EVAL_MAX_THRESHOLDS; ++k) bad[k] = 0;
    const auto distance = [&](float a, float b) {
        const float e = fabsf(__fsub_rn(a, b));
        err.add(e);
        err2.add(__fmul_rn(e, e));
        largest = fmaxf(largest, e);
#pragma unroll
        for (int k = 0; k < SSG_EVAL_MAX_THRESHOLDS; ++k) {
            if (k >= p.thresholds) break;
            bad[k] += e > p.threshold[k] ? 1 : 0;
        }
    };
    const int64_t quads = kVec ? n / 4 : 0;
    for (int64_t i = first; i < quads; i += stride) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(inv) + i), b = __ldg(reinterpret_cast<const float4*>(gt_inv) + i);
        distance(a.x, b.x);
        distance(a.y, b.y);
        distance(a.z, b.z);
        distance(a.w, b.w);
    }
    for (int64_t i = 4 * quads + first; i < n; i += stride) distance(__ldg(inv + i), __ldg(gt_inv + i));
    double sum = err.value(), sum2 = err2.value();
    if (largest >= 0x1p48f) {
        // the two floats hold fewer than 2^31 squares below 2^96: larger errors (a NaN is never the largest, and
        // stays one in the two floats) are summed once more in FP64
        sum = sum2 = 0.0;
        const auto again = [&](int64_t i) {
            const float e = fabsf(__fsub_rn(__ldg(inv + i), __ldg(gt_inv + i)));
            sum += (double)e;
            sum2 += (double)__fmul_rn(e, e);
        };
        for (int64_t i = first; i < quads; i += stride)
            for (int k = 0; k < 4; ++k) again(4 * i + k);
        for (int64_t i = 4 * quads + first; i < n; i += stride) again(i);
    }
    double* out = partials + ((int64_t)frame * gridDim.x + blockIdx.x) * eval_slots(p);
    double s = block_sum((double)sq * 0x1p-40, sh);
    if (threadIdx.x == 0) out[kSlotSq] = s;
    s = block_sum(sum, sh);
    if (threadIdx.x == 0) out[kSlotErr] = s;
    s = block_sum(sum2, sh);
    if (threadIdx.x == 0) out[kSlotErr2] = s;
#pragma unroll
    for (int k = 0; k < SSG_EVAL_MAX_THRESHOLDS; ++k) {
        if (k >= p.thresholds) break;
        s = block_sum((double)bad[k], sh);
        if (threadIdx.x == 0) out[kSlotBad + k] = s;
    }
}

// ---------------------------------------------------------------------------------------------
// SSIM in integers.  A colour value is x = RN(u / 255) in float32: a multiple of 2^-31, so with
// eps(u) = 255 * 2^31 x - 2^31 u, an integer of at most 16320, x = (u + eps(u) 2^-31) / 255 exactly.
// The window sums of x, x^2 and xy are then integer sums of u and u^2, exact in 32 bits, plus
// corrections linear in eps (below 2^-24 of them, so that float32 carries them to 2^-48; terms in
// eps^2 are below 2^-48 and dropped).  With p = u + v and m = u - v, over the N = 49 pixels of a
// window,
//     (sum p)^2 -+ (sum m)^2                               are 4 UV and 2 (U^2 + V^2),
//     N (sum p^2 -+ sum m^2) - ((sum p)^2 -+ (sum m)^2)    are N^2 times 4 cov and 2 (var + var),
// so the four factors of the SSIM ratio are, up to a common scale, those integers plus a constant
// each: the variances suffer no cancellation.  The ratio is formed in two floats (error 2^-43).
// Against 113-bit sums the mean of an image is within 2e-14 (FP64 window sums: 5e-15).
//
// Bound by instruction issue (about 130 per value).  FP64 sums per window took 7471 us for 4 frames
// of 2048x1024, this form takes 167 us.
// ---------------------------------------------------------------------------------------------
constexpr int kSsimCols = 58;  // map columns of a warp: two per lane, the last three lanes are halo
constexpr int kSums = 8;

// the integer and the fractional part of the constants of the two kinds of factors
constexpr double kSsimN = kSsimWin * kSsimWin, kSsimScale = 255.0 * 255.0 * kSsimN * kSsimN;
constexpr double kSsimC1 = 2.0 * (0.01 * 2.0) * (0.01 * 2.0) * kSsimScale;
constexpr double kSsimC2 = 2.0 * (0.03 * 2.0) * (0.03 * 2.0) * kSsimScale * (kSsimN - 1.0) / kSsimN;

// i + frac + correction as two floats (|i| < 2^31)
__device__ __forceinline__ void ssim_factor(int i, float rest, float& hi, float& lo)
{
    hi = __int2float_rn(i);
    // |i - hi| <= 64, read through the bits of a float
    lo = __fsub_rn(__int_as_float(0x4B400000 + (i - __float2int_rn(hi))), 12582912.0f) + rest;
}

// SSIM of one window from its sums of p, m, p^2, m^2, eps_p, eps_m, p eps_p and m eps_m
__device__ __forceinline__ void ssim_value(const int (&w)[kSums], float& value, float& low)
{
    constexpr int kI1 = (int)kSsimC1, kI2 = (int)kSsimC2, kN = kSsimWin * kSsimWin;
    constexpr float kF1 = (float)(kSsimC1 - kI1), kF2 = (float)(kSsimC2 - kI2), kUnit = 0x1p-30f;  // 2 x 2^-31
    const int pp = w[0] * w[0], mm = w[1] * w[1];
    const float pe = (float)w[0] * (float)w[4], me = (float)w[1] * (float)w[5];
    const float cp = fmaf((float)kN, (float)w[6], -pe), cm = fmaf((float)kN, (float)w[7], -me);
    float a1, a1l, b1, b1l, a2, a2l, b2, b2l;
    ssim_factor(pp - mm + kI1, fmaf(kUnit, pe - me, kF1), a1, a1l);
    ssim_factor(pp + mm + kI1, fmaf(kUnit, pe + me, kF1), b1, b1l);
    ssim_factor(kN * (w[2] - w[3]) - (pp - mm) + kI2, fmaf(kUnit, cp - cm, kF2), a2, a2l);
    ssim_factor(kN * (w[2] + w[3]) - (pp + mm) + kI2, fmaf(kUnit, cp + cm, kF2), b2, b2l);
    const float num = __fmul_rn(a1, a2), den = __fmul_rn(b1, b2);
    const float num_l = fmaf(a1, a2l, fmaf(a1l, a2, __fmaf_rn(a1, a2, -num)));
    const float den_l = fmaf(b1, b2l, fmaf(b1l, b2, __fmaf_rn(b1, b2, -den)));
    const float r = rcp_approx(den);
    value = __fmul_rn(num, r);
    low = (__fmaf_rn(-value, den, num) + fmaf(-value, den_l, num_l)) * r;
}

// The products of one column of a row: (p, m) and their eps packed as 16-bit halves
struct SsimPixel {
    uint32_t pm, eps;
    __device__ __forceinline__ void set(uint32_t u, uint32_t v, const int* __restrict__ table)
    {
        const int eu = table[u], ev = table[v];
        pm = ((u + v) & 0xFFFFu) | ((u - v) << 16);
        eps = ((uint32_t)(eu + ev) & 0xFFFFu) | ((uint32_t)(eu - ev) << 16);
    }
    // adds (kSign = 1) or subtracts its products
    template <int kSign>
    __device__ __forceinline__ void into(int (&s)[kSums]) const
    {
        const int p = (int16_t)pm, m = (int)pm >> 16, ep = (int16_t)eps, em = (int)eps >> 16;
        s[0] += kSign * p;
        s[1] += kSign * m;
        s[2] += kSign * (p * p);
        s[3] += kSign * (m * m);
        s[4] += kSign * ep;
        s[5] += kSign * em;
        s[6] += kSign * (p * ep);
        s[7] += kSign * (m * em);
    }
};

// SSIM map sums over the cropped region [3, rows - 3) x [3, cols - 3), all three channels.  A warp takes
// kSsimCols map columns of one channel and marches down `strip_rows` map rows: every lane keeps
// the 7-row sums of its two image columns (the rows that leave the window are kept packed in
// registers), and the 7-column sums come from the neighbouring lanes.  blockIdx.y: frame.
__global__ void __launch_bounds__(kEvalThreads, 3) eval_ssim_kernel(const __grid_constant__ EvalParams p, int strips,
                                                                    int strip_rows, const uint8_t* __restrict__ rgb,
                                                                    const uint8_t* __restrict__ gt_rgb,
                                                                    double* __restrict__ partials)
{
    __shared__ int table[256];
    __shared__ double sh[kEvalWarps];
    {
        const int u = threadIdx.x;
        const uint32_t x31 = (uint32_t)__fmul_rn(unit_value((uint8_t)u), 2147483648.0f);  // exact
        table[u] = (int)(255u * x31 - ((uint32_t)u << 31));
    }
    __syncthreads();
    const int64_t n = (int64_t)p.cols * p.rows;
    const int frame = blockIdx.y;
    rgb += (int64_t)frame * n * 3;
    gt_rgb += (int64_t)frame * n * 3;
    const int out_cols = p.cols - 2 * kSsimHalf, out_rows = p.rows - 2 * kSsimHalf;
    const int groups = (out_cols + kSsimCols - 1) / kSsimCols;
    const int tasks = groups * strips * 3;
    const int lane = threadIdx.x & 31;
    TwoFloat acc;
    for (int task = blockIdx.x * kEvalWarps + (threadIdx.x >> 5); task < tasks; task += gridDim.x * kEvalWarps) {
        const int ch = task % 3, group = (task / 3) % groups, strip = task / 3 / groups;
        // map pixel (x, y) is image pixel (x + 3, y + 3); its window covers image x .. x + 6
        const int x = group * kSsimCols + 2 * lane, y0 = strip * strip_rows;
        const int rows_in = min(strip_rows, out_rows - y0) + kSsimWin - 1;
        const bool on0 = 2 * lane < kSsimCols && x < out_cols, on1 = 2 * lane < kSsimCols && x + 1 < out_cols;
        const int64_t c0 = 3 * (int64_t)min(x, p.cols - 1) + ch, c1 = 3 * (int64_t)min(x + 1, p.cols - 1) + ch;
        const int64_t pitch = 3 * (int64_t)p.cols;
        const uint8_t* g = gt_rgb + y0 * pitch;
        const uint8_t* e = rgb + y0 * pitch;
        SsimPixel ring[kSsimWin][2];
        int s0[kSums], s1[kSums];
#pragma unroll
        for (int k = 0; k < kSums; ++k) s0[k] = s1[k] = 0;
        uint32_t u0 = __ldg(g + c0), v0 = __ldg(e + c0), u1 = __ldg(g + c1), v1 = __ldg(e + c1);
        for (int r = 0; r < rows_in; r += kSsimWin) {
#pragma unroll
            for (int i = 0; i < kSsimWin; ++i) {
                if (r + i >= rows_in) break;
                SsimPixel a, b;
                a.set(u0, v0, table);
                b.set(u1, v1, table);
                if (r + i + 1 < rows_in) {  // the next row, while this one is summed
                    g += pitch;
                    e += pitch;
                    u0 = __ldg(g + c0), v0 = __ldg(e + c0), u1 = __ldg(g + c1), v1 = __ldg(e + c1);
                }
                a.into<1>(s0);
                b.into<1>(s1);
                if (r > 0) {
                    ring[i][0].into<-1>(s0);
                    ring[i][1].into<-1>(s1);
                }
                ring[i][0] = a;
                ring[i][1] = b;
                if (r + i < kSsimWin - 1) continue;
                int w0[kSums], w1[kSums];
#pragma unroll
                for (int k = 0; k < kSums; ++k) {
                    const int pair = s0[k] + s1[k];
                    const int mid = __shfl_down_sync(0xffffffffu, pair, 1) + __shfl_down_sync(0xffffffffu, pair, 2);
                    w0[k] = pair + mid + __shfl_down_sync(0xffffffffu, s0[k], 3);
                    w1[k] = s1[k] + mid + __shfl_down_sync(0xffffffffu, pair, 3);
                }
                float v, low;
                ssim_value(w0, v, low);
                if (on0) acc.add(v, low);
                ssim_value(w1, v, low);
                if (on1) acc.add(v, low);
            }
        }
    }
    const double s = block_sum(acc.value(), sh);
    if (threadIdx.x == 0) partials[((int64_t)frame * gridDim.x + blockIdx.x) * eval_slots(p) + kSlotSsim] = s;
}

// One block per frame, a warp per slot: the blocks' partial sums in a fixed order, then the metrics.
__global__ void __launch_bounds__(kEvalThreads) eval_finish_kernel(const __grid_constant__ EvalParams p, int blocks,
                                                                   const double* __restrict__ partials,
                                                                   double* __restrict__ out)
{
    const int frame = blockIdx.x, slots = eval_slots(p), lane = threadIdx.x & 31;
    const double n = (double)p.cols * p.rows;
    const double map_n = (double)(p.cols - 2 * kSsimHalf) * (p.rows - 2 * kSsimHalf);
    double* o = out + (int64_t)frame * (SSG_EVAL_FIXED_METRICS + p.thresholds);
    for (int slot = threadIdx.x >> 5; slot < slots; slot += kEvalWarps) {
        double s = 0.0;
        for (int b = lane; b < blocks; b += 32) s += partials[((int64_t)frame * blocks + b) * slots + slot];
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0) {
            if (slot == kSlotSq) o[0] = 10.0 * log10(1.0 / (s / (3.0 * n)));
            else if (slot == kSlotSsim) o[1] = s / (3.0 * map_n);
            else if (slot == kSlotErr) o[2] = s / n;
            else if (slot == kSlotErr2) o[3] = sqrt(s / n);
            else o[SSG_EVAL_FIXED_METRICS + slot - kSlotBad] = 100.0 * s / n;
        }
    }
}

}  // namespace ssg

using namespace ssg;

extern "C" size_t ssg_eval_scratch_bytes(int frames, int threshold_count)
{
    if (frames < 1 || threshold_count < 0 || threshold_count > SSG_EVAL_MAX_THRESHOLDS) return 0;
    return sizeof(double) * (size_t)frames * kEvalBlocks * (kSlotBad + threshold_count);
}

extern "C" int ssg_eval_panoramas(int cols, int rows, int frames, const uint8_t* d_rgb, const uint8_t* d_gt_rgb,
                                  const float* d_inv_distance, const float* d_gt_inv_distance, const float* thresholds,
                                  int threshold_count, void* d_scratch, double* d_metrics, void* stream)
{
    SSG_REQUIRE(d_rgb && d_gt_rgb && d_inv_distance && d_gt_inv_distance && d_scratch && d_metrics, "null pointer");
    SSG_REQUIRE(cols >= 2 * kSsimHalf + 1 && rows >= 2 * kSsimHalf + 1,
                "panoramas of %dx%d are smaller than the 7x7 SSIM window", cols, rows);
    SSG_REQUIRE((int64_t)cols * rows * 3 < ((int64_t)1 << 40), "panoramas of %dx%d are too large", cols, rows);
    SSG_REQUIRE(frames >= 1 && frames <= 65535, "frames %d outside [1, 65535]", frames);
    SSG_REQUIRE(threshold_count >= 0 && threshold_count <= SSG_EVAL_MAX_THRESHOLDS,
                "threshold_count %d outside [0, %d]", threshold_count, SSG_EVAL_MAX_THRESHOLDS);
    SSG_REQUIRE(threshold_count == 0 || thresholds, "null thresholds");
    SSG_REQUIRE(((uintptr_t)d_scratch & 7) == 0 && ((uintptr_t)d_metrics & 7) == 0,
                "scratch and metrics must be 8-byte aligned");
    EvalParams p{};
    p.cols = cols;
    p.rows = rows;
    p.frames = frames;
    p.thresholds = threshold_count;
    for (int k = 0; k < threshold_count; ++k) p.threshold[k] = thresholds[k];
    cudaStream_t st = as_stream(stream);
    double* partials = static_cast<double*>(d_scratch);
    const dim3 grid(kEvalBlocks, frames);
    const int64_t n = (int64_t)cols * rows;
    const bool vec = (((uintptr_t)d_rgb | (uintptr_t)d_gt_rgb | (uintptr_t)d_inv_distance | (uintptr_t)d_gt_inv_distance) & 15) == 0 &&
                     (frames == 1 || n % 16 == 0);
    if (vec)
        eval_pointwise_kernel<true><<<grid, kEvalThreads, 0, st>>>(p, d_rgb, d_gt_rgb, d_inv_distance,
                                                                   d_gt_inv_distance, partials);
    else
        eval_pointwise_kernel<false><<<grid, kEvalThreads, 0, st>>>(p, d_rgb, d_gt_rgb, d_inv_distance,
                                                                    d_gt_inv_distance, partials);
    if (int e = launch_status("eval_pointwise_kernel")) return e;
    // one strip of rows per warp of the grid: every strip reads 6 rows more than it sums, so a strip
    // is at least 8 rows high
    const int out_rows = rows - 2 * kSsimHalf, groups = (cols - 2 * kSsimHalf + kSsimCols - 1) / kSsimCols;
    int strips = std::max(1, std::min(kEvalBlocks * kEvalWarps / (3 * groups), (out_rows + 7) / 8));
    const int strip_rows = (out_rows + strips - 1) / strips;
    strips = (out_rows + strip_rows - 1) / strip_rows;
    eval_ssim_kernel<<<grid, kEvalThreads, 0, st>>>(p, strips, strip_rows, d_rgb, d_gt_rgb, partials);
    if (int e = launch_status("eval_ssim_kernel")) return e;
    eval_finish_kernel<<<frames, kEvalThreads, 0, st>>>(p, kEvalBlocks, partials, d_metrics);
    return launch_status("eval_finish_kernel");
}
