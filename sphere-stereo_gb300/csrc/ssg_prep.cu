// Input preparation on the GPU: the linear resize the reference applies to every decoded image
// before the estimator (python/utils.py:198-201, cv2.resize(image, size, cv2.INTER_AREA) -- the
// third positional argument of cv2.resize is `dst`, so the interpolation in effect is the
// default, INTER_LINEAR).
//
// The taps are ssg_resize.cuh's.  Arithmetic:
//   - float pixels: h = S[sx] * (1 - fx) + S[sx + 1] * fx per row, then h0 * (1 - fy) + h1 * fy,
//     each product and sum rounded separately;
//   - uint8 pixels to uint8 (the ground-truth resize of the evaluation): 11-bit fixed-point
//     weights w0 = round(2048 (1 - f)) (saturated), w1 = 2048 - w0, integer sums, result
//     (v + 2^21) >> 22;
//   - an exact 2x reduction on both axes is an area average (OpenCV switches to INTER_AREA
//     there): floats (a + b + c + d) * 0.25, bytes (a + b + c + d + 2) >> 2.
// cv2 is not available here, so these statements are not pinned against OpenCV's own outputs.
#include <cmath>
#include <type_traits>

#include "ssg_common.cuh"
#include "ssg_resize.cuh"

namespace ssg {

__device__ __forceinline__ int fixed_weight(float f)
{
    const float w = __fmul_rn(__fsub_rn(1.0f, f), 2048.0f);
    return min(max(__float2int_rn(w), -32768), 32767);
}

// A thread takes four consecutive values of a destination row (one 16-byte store of floats) and runs
// down kResizeRows rows; a block takes kResizeThreads of them, whose column taps are formed once (in
// double, as OpenCV forms its tables, and FP64 is slow).  A source row blended for one destination
// row is kept for the next one that reads it, and a row's bytes are asked for while the row before is
// blended.  4 x 1216 x 1216 pixels of 3 bytes to 1024 x 1024 floats, 68 MB read and written (10 us of
// the copy bandwidth): 25.4 us, bound by the latency of its loads, at about a third of the issue rate; 27.5 us
// with 16 rows, 28 us without asking ahead; 41 us with a thread per pixel in blocks of 32 x 8, which
// stored floats 12 bytes apart.
constexpr int kResizeThreads = 192, kResizeRows = 8;
constexpr int kResizeValues = 4 * kResizeThreads;  // of a row, per block: whole pixels of 1, 2, 3 or 4 channels

// four values of one source row, as read: both taps of each
template <typename Tin>
struct RowTaps {
    Tin v0[4], v1[4];
    template <typename I>
    __device__ __forceinline__ void load(const Tin* __restrict__ row, const I (&at)[4], const int (&step)[4])
    {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v0[j] = __ldg(row + at[j]);
            v1[j] = __ldg(row + at[j] + step[j]);
        }
    }
    // blended along the row
    __device__ __forceinline__ void blend(const int (&a0)[4], const int (&a1)[4], int (&h)[4]) const
    {
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = (int)v0[j] * a0[j] + (int)v1[j] * a1[j];
    }
    __device__ __forceinline__ void blend(const float (&a0)[4], const float (&a1)[4], float (&h)[4]) const
    {
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __fadd_rn(__fmul_rn((float)v0[j], a0[j]), __fmul_rn((float)v1[j], a1[j]));
    }
};

template <typename Tout, bool kVector>
__device__ __forceinline__ void store_values(Tout* __restrict__ dst, const Tout (&v)[4], int n)
{
    if constexpr (kVector) {
        if constexpr (sizeof(Tout) == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        else *reinterpret_cast<uchar4*>(dst) = make_uchar4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < n) dst[j] = v[j];
    }
}

// blockIdx.x: kResizeValues values of a row; blockIdx.y: kResizeRows rows; blockIdx.z: image.
// I: holds a source row's values (int below 2^31, else int64_t).
// kVector: rows of a multiple of four values, dst aligned to four of them.
template <typename Tin, typename Tout, typename I, bool kArea, bool kVector>
__global__ void __launch_bounds__(kResizeThreads) resize_linear_kernel(const __grid_constant__ ResizeParams p,
                                                                      const Tin* __restrict__ src,
                                                                      Tout* __restrict__ dst)
{
    using H = std::conditional_t<sizeof(Tout) == 1, int, float>;  // a row's blended value
    __shared__ Tap cols_tap[kResizeValues], rows_tap[kResizeRows];
    const int C = p.channels, pixels = kResizeValues / C;
    const int64_t x0 = (int64_t)blockIdx.x * pixels;  // the block's first pixel
    const int y0 = blockIdx.y * kResizeRows;
    const int64_t values = (int64_t)p.dst_cols * C, pitch = (int64_t)p.src_cols * C;
    src += (int64_t)blockIdx.z * p.src_rows * pitch;
    for (int k = threadIdx.x; k < pixels && x0 + k < p.dst_cols; k += kResizeThreads)
        cols_tap[k] = column_tap(p, (int)(x0 + k));
    if (threadIdx.x < kResizeRows) rows_tap[threadIdx.x] = row_tap(p, min(y0 + (int)threadIdx.x, p.dst_rows - 1));
    __syncthreads();
    const int64_t e = x0 * C + 4 * threadIdx.x;
    if (e >= values) return;
    const int n = (int)(values - e < 4 ? values - e : 4);
    dst += ((int64_t)blockIdx.z * p.dst_rows + y0) * values + e;
    I at[4];
    int step[4];
    H a0[4], a1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int k = 4 * threadIdx.x + min(j, n - 1), px = k / C;
        const Tap t = cols_tap[px];
        at[j] = (I)t.s0 * C + (k - px * C);
        step[j] = (t.s1 - t.s0) * C;
        if constexpr (std::is_same<H, int>::value) {
            a0[j] = fixed_weight(t.f);
            a1[j] = 2048 - a0[j];
        } else {
            a0[j] = __fsub_rn(1.0f, t.f);
            a1[j] = t.f;
        }
    }
    const int rows = min(kResizeRows, p.dst_rows - y0);
    // a row's taps are asked for while the row before is blended
    H h0[4], h1[4];
    RowTaps<Tin> top, bottom, next_top, next_bottom;
    top.load(src + rows_tap[0].s0 * pitch, at, step);
    bottom.load(src + rows_tap[0].s1 * pitch, at, step);
    bool kept = false;  // the row's upper source row is the lower one of the row before: h1
    for (int r = 0; r < rows; ++r, dst += values) {
        bool keep = false;
        if (r + 1 < rows) {
            keep = !kArea && rows_tap[r + 1].s0 == rows_tap[r].s1;
            if (!keep) next_top.load(src + rows_tap[r + 1].s0 * pitch, at, step);
            next_bottom.load(src + rows_tap[r + 1].s1 * pitch, at, step);
        }
        Tout out[4];
        if constexpr (kArea) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const Tin a = top.v0[j], b = top.v1[j], c = bottom.v0[j], d = bottom.v1[j];
                if constexpr (std::is_same<H, int>::value) out[j] = (Tout)(((int)a + b + c + d + 2) >> 2);
                else out[j] = __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn((float)a, (float)b), (float)c), (float)d), 0.25f);
            }
        } else {
            const float f = rows_tap[r].f;
            if (kept) {
#pragma unroll
                for (int j = 0; j < 4; ++j) h0[j] = h1[j];
            } else {
                top.blend(a0, a1, h0);
            }
            bottom.blend(a0, a1, h1);
            if constexpr (std::is_same<H, int>::value) {
                const int b0 = fixed_weight(f), b1 = 2048 - b0;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    out[j] = (Tout)min(max((h0[j] * b0 + h1[j] * b1 + (1 << 21)) >> 22, 0), 255);
            } else {
                const float b0 = __fsub_rn(1.0f, f), b1 = f;
#pragma unroll
                for (int j = 0; j < 4; ++j) out[j] = __fadd_rn(__fmul_rn(h0[j], b0), __fmul_rn(h1[j], b1));
            }
        }
        store_values<Tout, kVector>(dst, out, n);
        kept = keep;
        top = next_top;
        bottom = next_bottom;
    }
}

template <typename Tin, typename Tout>
static int launch_resize(const ResizeParams& p, const void* src, void* dst, int images, cudaStream_t st)
{
    const int pixels = kResizeValues / p.channels;
    const dim3 grid((unsigned)(((int64_t)p.dst_cols + pixels - 1) / pixels),
                    (unsigned)((p.dst_rows + kResizeRows - 1) / kResizeRows), (unsigned)images);
    const bool vector = (int64_t)p.dst_cols * p.channels % 4 == 0 && ((uintptr_t)dst & (4 * sizeof(Tout) - 1)) == 0;
    const bool wide = (int64_t)p.src_cols * p.channels >= ((int64_t)1 << 31) - 4;
    const auto kernel = wide      ? (p.area2 ? resize_linear_kernel<Tin, Tout, int64_t, true, false>
                                             : resize_linear_kernel<Tin, Tout, int64_t, false, false>)
                        : p.area2 ? (vector ? resize_linear_kernel<Tin, Tout, int, true, true>
                                            : resize_linear_kernel<Tin, Tout, int, true, false>)
                                  : (vector ? resize_linear_kernel<Tin, Tout, int, false, true>
                                            : resize_linear_kernel<Tin, Tout, int, false, false>);
    kernel<<<grid, kResizeThreads, 0, st>>>(p, static_cast<const Tin*>(src), static_cast<Tout*>(dst));
    return launch_status("resize_linear_kernel");
}

}  // namespace ssg

using namespace ssg;

extern "C" int ssg_resize_linear(const void* d_src, int src_type, int src_cols, int src_rows, int channels,
                                 void* d_dst, int dst_type, int dst_cols, int dst_rows, int images, void* stream)
{
    SSG_REQUIRE(d_src && d_dst, "null pointer");
    SSG_REQUIRE(src_cols >= 1 && src_rows >= 1 && dst_cols >= 1 && dst_rows >= 1, "empty image");
    SSG_REQUIRE(channels >= 1 && channels <= 4, "channels %d outside [1, 4]", channels);
    SSG_REQUIRE(images >= 1 && images <= 65535, "images %d outside [1, 65535]", images);
    SSG_REQUIRE((int64_t)src_cols * src_rows * channels < ((int64_t)1 << 40) &&
                    (int64_t)dst_cols * dst_rows < ((int64_t)1 << 31) * 256,
                "images too large");
    SSG_REQUIRE((src_type == SSG_PIXEL_U8 || src_type == SSG_PIXEL_F32) &&
                    (dst_type == SSG_PIXEL_F32 || (dst_type == SSG_PIXEL_U8 && src_type == SSG_PIXEL_U8)),
                "unsupported pixel types %d -> %d (u8 -> f32, f32 -> f32, u8 -> u8)", src_type, dst_type);
    const ResizeParams p = make_resize_params(src_cols, src_rows, dst_cols, dst_rows, channels);
    SSG_REQUIRE((dst_rows + 7) / 8 <= 65535, "destination of %d rows is too tall", dst_rows);
    cudaStream_t st = as_stream(stream);
    if (src_type == SSG_PIXEL_F32) return launch_resize<float, float>(p, d_src, d_dst, images, st);
    if (dst_type == SSG_PIXEL_F32) return launch_resize<uint8_t, float>(p, d_src, d_dst, images, st);
    return launch_resize<uint8_t, uint8_t>(p, d_src, d_dst, images, st);
}
