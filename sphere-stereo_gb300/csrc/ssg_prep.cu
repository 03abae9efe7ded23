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

__device__ __forceinline__ float in_value(const float* s, int64_t i) { return __ldg(s + i); }
__device__ __forceinline__ float in_value(const uint8_t* s, int64_t i) { return (float)__ldg(s + i); }

// Small images: one block per kTileX x kTileY destination pixels of one image (blockIdx.z): the tile's column
// and row taps are formed once (in double, as OpenCV forms its tables) into shared memory, then
// one thread per destination pixel (all channels) blends.
constexpr int kTileX = 32, kTileY = 8;

template <typename Tin, typename Tout>
__global__ void __launch_bounds__(kTileX * kTileY) resize_pixels_kernel(const __grid_constant__ ResizeParams p,
                                                                        const Tin* __restrict__ src,
                                                                        Tout* __restrict__ dst)
{
    __shared__ Tap cols_tap[kTileX], rows_tap[kTileY];
    const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kTileY;
    const int C = p.channels;
    src += (int64_t)blockIdx.z * p.src_cols * p.src_rows * C;
    dst += (int64_t)blockIdx.z * p.dst_cols * p.dst_rows * C;
    if (!p.area2) {
        if (threadIdx.x < kTileX) cols_tap[threadIdx.x] = column_tap(p, min(x0 + (int)threadIdx.x, p.dst_cols - 1));
        else if (threadIdx.x < kTileX + kTileY)
            rows_tap[threadIdx.x - kTileX] = row_tap(p, min(y0 + (int)threadIdx.x - kTileX, p.dst_rows - 1));
        __syncthreads();
    }
    const int dx = x0 + (int)(threadIdx.x % kTileX), dy = y0 + (int)(threadIdx.x / kTileX);
    if (dx >= p.dst_cols || dy >= p.dst_rows) return;
    dst += ((int64_t)dy * p.dst_cols + dx) * C;
    if (p.area2) {
        const int64_t r0 = (int64_t)(2 * dy) * p.src_cols, r1 = r0 + p.src_cols;
        for (int c = 0; c < C; ++c) {
            const int64_t a = (r0 + 2 * dx) * C + c, b = a + C, d0 = (r1 + 2 * dx) * C + c, d1 = d0 + C;
            if constexpr (sizeof(Tout) == 1) {
                const int s = (int)__ldg(src + a) + __ldg(src + b) + __ldg(src + d0) + __ldg(src + d1);
                dst[c] = (Tout)((s + 2) >> 2);
            } else {
                const float s = __fadd_rn(__fadd_rn(__fadd_rn(in_value(src, a), in_value(src, b)), in_value(src, d0)),
                                          in_value(src, d1));
                dst[c] = __fmul_rn(s, 0.25f);
            }
        }
        return;
    }
    const Tap tx = cols_tap[threadIdx.x % kTileX], ty = rows_tap[threadIdx.x / kTileX];
    const int64_t r0 = (int64_t)ty.s0 * p.src_cols, r1 = (int64_t)ty.s1 * p.src_cols;
    if constexpr (sizeof(Tout) == 1) {
        const int a0 = fixed_weight(tx.f), a1 = 2048 - a0, b0 = fixed_weight(ty.f), b1 = 2048 - b0;
        for (int c = 0; c < C; ++c) {
            const int h0 = (int)__ldg(src + (r0 + tx.s0) * C + c) * a0 + (int)__ldg(src + (r0 + tx.s1) * C + c) * a1;
            const int h1 = (int)__ldg(src + (r1 + tx.s0) * C + c) * a0 + (int)__ldg(src + (r1 + tx.s1) * C + c) * a1;
            const int v = (h0 * b0 + h1 * b1 + (1 << 21)) >> 22;
            dst[c] = (Tout)min(max(v, 0), 255);
        }
    } else {
        const float a0 = __fsub_rn(1.0f, tx.f), a1 = tx.f, b0 = __fsub_rn(1.0f, ty.f), b1 = ty.f;
        for (int c = 0; c < C; ++c) {
            const float h0 = __fadd_rn(__fmul_rn(in_value(src, (r0 + tx.s0) * C + c), a0),
                                       __fmul_rn(in_value(src, (r0 + tx.s1) * C + c), a1));
            const float h1 = __fadd_rn(__fmul_rn(in_value(src, (r1 + tx.s0) * C + c), a0),
                                       __fmul_rn(in_value(src, (r1 + tx.s1) * C + c), a1));
            dst[c] = __fadd_rn(__fmul_rn(h0, b0), __fmul_rn(h1, b1));
        }
    }
}

// Large images.  A thread takes four consecutive values of a destination row (one 16-byte store of
// floats) and runs down kResizeRows rows; a block takes kResizeThreads of them, whose column taps are
// formed once (in double, as OpenCV forms its tables, and FP64 is slow).  A source row blended for one
// destination row is kept for the next one that reads it, and a row's bytes are asked for while the row
// before is blended.  4 x 1216 x 1216 pixels of 3 bytes to 1024 x 1024 floats, 68 MB read and written (10 us
// of the copy bandwidth), the kernel alone, from cold caches: 25.4 us, bound by the latency of its loads, at
// about a third of the issue rate; 27.5 us with 16 rows, 28 us without asking ahead; 41 us with a thread per
// pixel, which stores floats 12 bytes apart.
constexpr int kResizeThreads = 192, kResizeRows = 8;
constexpr int kResizeValues = 4 * kResizeThreads;  // of a row, per block: whole pixels of 1, 2, 3 or 4 channels

// four values of one source row, as read: both taps of each
template <typename Tin>
struct RowTaps {
    Tin v0[4], v1[4];
    __device__ __forceinline__ void load(const Tin* __restrict__ row, const int (&at)[4], const int (&step)[4])
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
// kVector: rows of a multiple of four values, dst aligned to four of them.
// A source row holds fewer than 2^31 values.
template <typename Tin, typename Tout, bool kArea, bool kVector>
__global__ void __launch_bounds__(kResizeThreads) resize_rows_kernel(const __grid_constant__ ResizeParams p,
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
    int at[4], step[4];
    H a0[4], a1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int k = 4 * threadIdx.x + min(j, n - 1), px = k / C;
        const Tap t = cols_tap[px];
        at[j] = t.s0 * C + (k - px * C);
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
    const Tin* s = static_cast<const Tin*>(src);
    Tout* d = static_cast<Tout*>(dst);
    const int64_t values = (int64_t)p.dst_cols * p.channels;
    const int rows = (p.dst_rows + kResizeRows - 1) / kResizeRows, pixels = kResizeValues / p.channels;
    const int64_t across = ((int64_t)p.dst_cols + pixels - 1) / pixels;  // blocks of a row
    // Small images go by pixels: a thread of the rows kernel takes eight rows one after the other, 4 us and more
    // however little there is to do (64 x 64 to 48 x 48: 4.5 us by rows, 2.3 by pixels; 1001 x 777 to
    // 640 x 333 6.0 and 3.9; 1216 x 1216 to 1024 x 1024, four images, 21 and 37).  The lines, in output pixels,
    // lie where the two are even, measured at 400 K to 4 M pixels of 1 to 4 channels: 3 channels 720 x 720
    // 5.7 by rows and 6.4 by pixels, 640 x 640 5.4 and 5.6; 1 channel 800 x 800 6.8 and 5.9, 900 x 900 6.9 and
    // 7.2; 4 channels (a pixel's load is one access already) 1100 x 1100 12.1 and 11.5, 2000 x 2000 33 and 37;
    // averages of bytes 1000 x 1000 7.9 and 8.1, of floats (no row is read twice) 42 and 39 for four of
    // them.  Rows that leave the last block mostly empty count by the square of its use: sixteen
    // 257 x 257 images of 3 channels take 13.3 by rows, 12.1 by pixels.
    const double pixels_out = (double)p.dst_cols * p.dst_rows * images;
    const double used = (double)values / (across * kResizeValues);
    const double work = p.channels == 1 ? pixels_out : pixels_out * used * used;
    const bool floats = sizeof(Tin) == 4;
    const double least = p.area2 ? (floats || p.channels == 4 ? INFINITY : p.channels == 1 ? 0.95e6 : 1.5e6)
                         : p.channels == 1 ? 0.75e6
                         : p.channels == 4 ? (floats ? 0.7e6 : 1.4e6)
                                           : (floats ? 0.3e6 : 0.42e6);
    const bool by_rows = work >= least && (int64_t)p.src_cols * p.channels < ((int64_t)1 << 31) - 4;
    if (!by_rows) {
        const dim3 grid((unsigned)((p.dst_cols + kTileX - 1) / kTileX), (unsigned)((p.dst_rows + kTileY - 1) / kTileY),
                        (unsigned)images);
        resize_pixels_kernel<Tin, Tout><<<grid, kTileX * kTileY, 0, st>>>(p, s, d);
        return launch_status("resize_pixels_kernel");
    }
    const dim3 grid((unsigned)across, (unsigned)rows, (unsigned)images);
    const bool vector = values % 4 == 0 && ((uintptr_t)dst & (4 * sizeof(Tout) - 1)) == 0;
    if constexpr (sizeof(Tin) == 1) {
        if (p.area2) {
            const auto kernel = vector ? resize_rows_kernel<Tin, Tout, true, true> : resize_rows_kernel<Tin, Tout, true, false>;
            kernel<<<grid, kResizeThreads, 0, st>>>(p, s, d);
            return launch_status("resize_rows_kernel");
        }
    }
    const auto kernel = vector ? resize_rows_kernel<Tin, Tout, false, true> : resize_rows_kernel<Tin, Tout, false, false>;
    kernel<<<grid, kResizeThreads, 0, st>>>(p, s, d);
    return launch_status("resize_rows_kernel");
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
