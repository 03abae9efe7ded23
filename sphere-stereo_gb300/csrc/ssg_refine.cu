// The differentiable sweep of several reference cameras at once: soft-argmin inverse distance and its
// backward pass (ssg_backward.cu documents the mathematics and holds the per-step entry points;
// values, sums and their order are the same here).
//
// What the per-step form spent its time on, and what is done instead:
//   * every transposed filter step evaluated the weights of a cell's neighbours for itself, 200 to 225
//     exponentials per thread in code larger than the instruction cache: 140 us for a step of any
//     size.  The weights of all levels are formed once, by one launch, into a table (38 floats per
//     coarse pixel), and the transposed steps read the 25 values that concern a cell;
//   * the small levels of the transposed filter run in one launch, a block per candidate;
//   * the 64-bit conversions of the image gradient and the pose sums ran on the FP64 pipe, which is 64
//     times slower than the FP32 pipes: conversions are sums with constants or shifts, pose sums are
//     reduced transposed;
//   * the image gradient took 12 atomic adds per sample: neighbouring pixels' samples that land on
//     the same texel are added within the warp first (integers: the sum does not depend on it).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ssg_isb_planar.cuh"
#include "ssg_soft.cuh"
#include "ssg_sweep_packed.cuh"
#include "ssg_uneven.cuh"

namespace ssg {

// ---------------------------------------------------------------------------------------------
// Soft-argmin over the filtered level-0 costs, which are never written.  Blocks of 32 coarse pixels,
// a warp per fine row; a pixel's candidates are taken in order (the online softmax).
// ---------------------------------------------------------------------------------------------
struct SoftSink {
    static constexpr int kAhead = 0;
    float inv_tau;
    const float* inv_cand;
    OnlineSoftmax a, b;
    __device__ __forceinline__ void take(int k, int, float va, float vb)
    {
        a.push(-va * inv_tau, inv_cand[k]);
        b.push(-vb * inv_tau, inv_cand[k]);
    }
};
// the same, keeping the filtered costs in `level` for the second pass
template <bool kPairs>
struct SoftKeepSink {
    static constexpr int kAhead = 0;
    SoftSink soft;
    StoreSink<kPairs> store;
    __device__ __forceinline__ void take(int k, int at, float va, float vb)
    {
        soft.take(k, at, va, vb);
        store.take(k, at, va, vb);
    }
};

template <int FA, int FB, bool kPairs, bool kBackward>
__device__ __forceinline__ void soft_row(const float* __restrict__ cost_in, const float* __restrict__ cost_fine,
                                         const LevelGeom& g, int x, int y, float weight_up, const float (&sw)[kUpRows][32],
                                         const SoftParams& sp, float* __restrict__ q, const float* __restrict__ grad_q,
                                         float* grad_F)
{
    const int px = threadIdx.x & 31, pio = g.rows_out * g.cols_out;
    const int at = (2 * y + (FA & 1)) * g.cols_out + 2 * x;
    const bool second = 2 * x + 1 < g.cols_out;
    const float inv_tau = 1.0f / sp.tau;
    SoftKeepSink<kPairs> sink{{inv_tau, sp.inv_cand}, {grad_F, pio, second}};
    sink.soft.a.init();
    sink.soft.b.init();
    if constexpr (!kBackward) {
        planar_up_row<FA, FB, kPairs>(cost_in, cost_fine, g, x, y, 0, sp.ncand, weight_up, sw, px, sink.soft);
        q[at] = sink.soft.a.t / sink.soft.a.s;
        if (second) q[at + 1] = sink.soft.b.t / sink.soft.b.s;
    } else {
        planar_up_row<FA, FB, kPairs>(cost_in, cost_fine, g, x, y, 0, sp.ncand, weight_up, sw, px, sink);
        const OnlineSoftmax sm[2] = {sink.soft.a, sink.soft.b};
        float qv[2], gq[2];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            qv[f] = sm[f].t / sm[f].s;
            gq[f] = f == 0 || second ? grad_q[at + f] : 0.0f;
        }
        // this thread's own costs, read back
#pragma unroll 4
        for (int z = 0; z < sp.ncand; ++z) {
            float* p = grad_F + (int64_t)z * pio;
            const float2 c2 = load_fine<kPairs>(p, at, second);
            const float c[2] = {c2.x, c2.y};
            float out[2];
#pragma unroll
            for (int f = 0; f < 2; ++f) {
                const float w = expf(-c[f] * inv_tau - sm[f].m) / sm[f].s;
                out[f] = gq[f] * (-inv_tau) * w * (sp.inv_cand[z] - qv[f]);
            }
            if constexpr (kPairs) {
                *reinterpret_cast<float2*>(p + at) = make_float2(out[0], out[1]);
            } else {
                p[at] = out[0];
                if (second) p[at + 1] = out[1];
            }
        }
    }
}

// blockIdx.x: group of 32 coarse pixels; blockIdx.y: instance
template <bool kPairs, bool kBackward>
__global__ void __launch_bounds__(64) isb_soft_kernel(
    const uint8_t* __restrict__ guide_in, const float* __restrict__ cost_in, const uint8_t* __restrict__ guide_fine,
    const float* __restrict__ cost_fine, LevelGeom g, float weight_up, float weight_down, float var_inv_i,
    const float* __restrict__ table, const __grid_constant__ SoftParams sp, float* __restrict__ q,
    const float* __restrict__ grad_q, float* grad_F)
{
    __shared__ float sw[kUpRows][32];
    const int pin = g.rows_in * g.cols_in, pio = g.rows_out * g.cols_out;
    const int64_t inst = blockIdx.y;
    guide_in += inst * pin * G3::bytes;
    guide_fine += inst * pio * G3::bytes;
    cost_in += inst * sp.ncand * pin;
    cost_fine += inst * sp.ncand * pio;
    if constexpr (kBackward) {
        grad_q += inst * pio;
        grad_F += inst * sp.ncand * pio;
    } else {
        q += inst * pio;
    }
    const int o = blockIdx.x * 32 + (threadIdx.x & 31);
    const bool in = o < pin;
    const int y = o / g.cols_in, x = o - y * g.cols_in;
    planar_setup<G3>(guide_in, guide_fine, nullptr, g, x, y, in, weight_up, weight_down, TableRange{table, var_inv_i}, sw);
    __syncthreads();
    if (!in) return;
    if (threadIdx.x < 32)
        soft_row<0, 2, kPairs, kBackward>(cost_in, cost_fine, g, x, y, weight_up, sw, sp, q, grad_q, grad_F);
    else if (2 * y + 1 < g.rows_out)
        soft_row<1, 3, kPairs, kBackward>(cost_in, cost_fine, g, x, y, weight_up, sw, sp, q, grad_q, grad_F);
}

// ---------------------------------------------------------------------------------------------
// The table of the filter's weights: per level pair (fine level s, coarse level s + 1) and coarse pixel
// the 25 weights and 4 reciprocals of its fine pixels in the up step (kUpRows), and the 9 normalised
// weights of its taps in the down step.
// ---------------------------------------------------------------------------------------------
constexpr int kDownRow = kUpRows, kTableRows = kUpRows + 9;

struct TableLevels {
    int levels;
    int rows[SSG_MAX_LEVELS], cols[SSG_MAX_LEVELS];
    const uint8_t* guides[SSG_MAX_LEVELS];    // unfiltered
    const uint8_t* filtered[SSG_MAX_LEVELS];  // filtered (levels >= 1)
    float weight_up[SSG_MAX_LEVELS], weight_down[SSG_MAX_LEVELS];
    int64_t offset[SSG_MAX_LEVELS];  // floats from an instance's table to pair s
    int64_t stride;                  // floats of an instance's table
    int first_group[SSG_MAX_LEVELS + 1];
};

// blockIdx.x: group of 32 coarse pixels of a pair; blockIdx.y: instance.  Warps 0 to 3: the fine
// pixels' weights; warp 4: the down step's.
__global__ void __launch_bounds__(160) isb_table_kernel(const __grid_constant__ TableLevels T, float var_inv_i,
                                                        const float* __restrict__ table, float* __restrict__ tables)
{
    int s = 0;
    while ((int)blockIdx.x >= T.first_group[s + 1]) ++s;
    const LevelGeom g{T.rows[s + 1], T.cols[s + 1], T.rows[s], T.cols[s]};
    const int pin = g.rows_in * g.cols_in, pio = g.rows_out * g.cols_out;
    const int64_t inst = blockIdx.y;
    const int o = ((int)blockIdx.x - T.first_group[s]) * 32 + (threadIdx.x & 31);
    if (o >= pin) return;
    const int y = o / g.cols_in, x = o - y * g.cols_in;
    float* out = tables + inst * T.stride + T.offset[s] + o;
    const TableRange range{table, var_inv_i};
    const uint8_t* fine = T.guides[s] + inst * pio * G3::bytes;
    const auto up = [&](auto tag) {
        constexpr int F = decltype(tag)::value;
        const int fx = 2 * x + (F >= 2 ? 1 : 0), fy = 2 * y + (F & 1);
        if (fx >= g.cols_out || fy >= g.rows_out) return;
        int ci[9];
        G3::Pix gd[9];
        coarse_neighbourhood<int, G3>(T.filtered[s + 1] + inst * pin * G3::bytes, g.rows_in, g.cols_in, x, y, ci, gd);
        float w[UpTaps<F>::n], gs[3];
        const float inv = fine_weights<F, TableRange, G3>(gd, G3::load(fine, fy * g.cols_out + fx), T.weight_up[s],
                                                          T.weight_down[s], range, w, gs);
#pragma unroll
        for (int i = 0; i < UpTaps<F>::n; ++i) out[(int64_t)(up_weight_row<F>() + i) * pin] = w[i];
        out[(int64_t)(kUpInvRow + F) * pin] = inv;
    };
    switch (threadIdx.x >> 5) {
    case 0: up(std::integral_constant<int, 0>{}); return;
    case 1: up(std::integral_constant<int, 1>{}); return;
    case 2: up(std::integral_constant<int, 2>{}); return;
    case 3: up(std::integral_constant<int, 3>{}); return;
    }
    const int x2 = 2 * x, y2 = 2 * y;
    const int xp = min(x2 + 1, g.cols_out - 1), yp = min(y2 + 1, g.rows_out - 1), xm = max(x2 - 1, 0), ym = max(y2 - 1, 0);
    const int rows[8] = {ym, y2, yp, yp, yp, y2, ym, ym}, cols[8] = {xm, xm, xm, x2, xp, xp, xp, x2};
    const G3::Pix cur = G3::load(fine, y2 * g.cols_out + x2);
    float w[9], wsum = 1.0f;
    w[0] = 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        w[i + 1] = fmul(i % 2 ? 0.5f : 0.25f, range(G3::dist(cur, G3::load(fine, rows[i] * g.cols_out + cols[i]))));
        wsum = fadd(wsum, w[i + 1]);
    }
#pragma unroll
    for (int t = 0; t < 9; ++t) out[(int64_t)(kDownRow + t) * pin] = fdiv(w[t], wsum);
}

// ---------------------------------------------------------------------------------------------
// Transposed steps.  A coarse cell (X, Y) is read by 25 fine pixels: those of its 3 x 3 coarse
// neighbours (dx, dy) that hold it in their tap lists, F = 0 of all nine, F = 1 (the row below) of
// those with dy <= 0, F = 2 of those with dx <= 0 and F = 3 of both: the 5 x 5 fine pixels around
// (2 X, 2 Y).  Entries are numbered neighbour by neighbour, then by F, the order of their sum.
// ---------------------------------------------------------------------------------------------
struct TransposeEntry {
    int dx, dy, f;
};
// rows dy = -1, 0, 1 hold 10, 10 and 5 entries; in a row of 10, dx = -1, 0, 1 hold 4, 4 and 2 (F = 0, 1),
// in the row of 5 they hold 2 (F = 0, 2), 2 and 1
__host__ __device__ constexpr TransposeEntry transpose_entry(int e)
{
    return e < 20 ? TransposeEntry{e % 10 / 4 - 1, e / 10 - 1, e % 10 % 4}
                  : TransposeEntry{(e - 20) / 2 - 1, 1, (e - 20) % 2 * 2};
}
constexpr int kEntries = 25;

// weight with which fine pixel F of coarse pixel (x, y) reads cell (X, Y): the sum over its edge-clamped
// taps that are the cell
template <int F>
__device__ __forceinline__ float read_weight(const float* __restrict__ t, const LevelGeom& g, int x, int y, int X, int Y)
{
    if (x < 0 || y < 0 || x >= g.cols_in || y >= g.rows_in) return 0.0f;
    if (((F & 1) && 2 * y + 1 >= g.rows_out) || (F >= 2 && 2 * x + 1 >= g.cols_out)) return 0.0f;
    const int64_t pin = (int64_t)g.rows_in * g.cols_in;
    t += y * g.cols_in + x;
    bool row[3], col[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        row[i] = min(max(y + i - 1, 0), g.rows_in - 1) == Y;
        col[i] = min(max(x + i - 1, 0), g.cols_in - 1) == X;
    }
    const float inv = __ldg(t + (kUpInvRow + F) * pin);
    float k = 0.0f;
#pragma unroll
    for (int i = 0; i < UpTaps<F>::n; ++i)
        if (row[UpTaps<F>::tap(i) / 3] && col[UpTaps<F>::tap(i) % 3])
            k = fmaf(__ldg(t + (up_weight_row<F>() + i) * pin), inv, k);
    return k;
}
__device__ __forceinline__ float read_weight(int f, const float* __restrict__ t, const LevelGeom& g, int x, int y, int X,
                                             int Y)
{
    switch (f) {
    case 0: return read_weight<0>(t, g, x, y, X, Y);
    case 1: return read_weight<1>(t, g, x, y, X, Y);
    case 2: return read_weight<2>(t, g, x, y, X, Y);
    default: return read_weight<3>(t, g, x, y, X, Y);
    }
}

// weight of fine pixel F's own cost in its filtered one
__device__ __forceinline__ float own_weight(int f, const float* __restrict__ t, const LevelGeom& g, int X, int Y,
                                            float weight_up)
{
    if (((f & 1) && 2 * Y + 1 >= g.rows_out) || (f >= 2 && 2 * X + 1 >= g.cols_out)) return 0.0f;
    return weight_up * __ldg(t + (int64_t)(kUpInvRow + f) * g.rows_in * g.cols_in + Y * g.cols_in + X);
}

// weight of fine cell (X, Y) in the down step's coarse pixel (x, y), at most one clamped tap apart
__device__ __forceinline__ float down_read_weight(const float* __restrict__ t, const LevelGeom& g, int x, int y, int X,
                                                  int Y)
{
    const int64_t pin = (int64_t)g.rows_in * g.cols_in;
    const int x2 = 2 * x, y2 = 2 * y;
    const bool cp = min(x2 + 1, g.cols_out - 1) == X, cm = max(x2 - 1, 0) == X, c0 = x2 == X;
    const bool rp = min(y2 + 1, g.rows_out - 1) == Y, rm = max(y2 - 1, 0) == Y, r0 = y2 == Y;
    const bool hit[9] = {r0 && c0, rm && cm, r0 && cm, rp && cm, rp && c0, rp && cp, r0 && cp, rm && cp, rm && c0};
    t += kDownRow * pin + y * g.cols_in + x;
    float k = 0.0f;
#pragma unroll
    for (int i = 0; i < 9; ++i)
        if (hit[i]) k += __ldg(t + i * pin);
    return k;
}
// the coarse pixels that can hold a fine cell: n-th of (X >> 1) + {0, 1} x (Y >> 1) + {0, 1}
__device__ __forceinline__ bool down_reader(const LevelGeom& g, int n, int X, int Y, int& x, int& y)
{
    x = (X >> 1) + (n & 1);
    y = (Y >> 1) + (n >> 1);
    const bool none = ((n & 1) && !(X & 1)) || ((n >> 1) && !(Y & 1));
    return !none && x < g.cols_in && y < g.rows_in;
}

// Threads of a transposed step's block: 8 warps share out the candidates, or 4, which repeat the set-up
// half as often, where the level has enough groups of 32 cells.  48 candidates, 8 and 4 warps: 4096
// groups (level 0 of two 512 x 512 references) up 81 and 72 us, down 69 and 53; 1024 groups up 26.2 and
// 24.8, down 16.4 and 15.5; at 256 groups 4 warps lost 10 and 8 us.
constexpr int kTransposeBlock = 256, kTransposeFull = 1024;

// Up step transposed: g_f(coarse) = sum over the cell's readers.  (A fine pixel's own part, own weight *
// g_f(fine), is formed by the down step's kernel, which reads g_f once more instead of adding to a
// volume written here.)  A block takes 32 coarse cells; its warps share out their weights and then the
// candidates.  blockIdx.y: instance.
template <int kThreads>
__global__ void __launch_bounds__(kThreads) isb_up_transpose_table_kernel(
    const float* __restrict__ tables, int64_t table_stride, LevelGeom g, int ncand,
    const float* __restrict__ grad_f_fine, float* __restrict__ grad_f_coarse)
{
    __shared__ float sk[kEntries][32];
    const int pin = g.rows_in * g.cols_in, pio = g.rows_out * g.cols_out;
    const int64_t inst = blockIdx.y;
    tables += inst * table_stride;
    grad_f_fine += inst * ncand * pio;
    grad_f_coarse += inst * ncand * pin;
    const int px = threadIdx.x & 31, range = threadIdx.x >> 5;
    constexpr int ranges = kThreads / 32;
    const int o = blockIdx.x * 32 + px, oc = min(o, pin - 1);
    const int Y = oc / g.cols_in, X = oc - Y * g.cols_in;
#pragma unroll 1
    for (int e = range; e < kEntries; e += ranges) {
        const TransposeEntry t = transpose_entry(e);
        sk[e][px] = read_weight(t.f, tables, g, X + t.dx, Y + t.dy, X, Y);
    }
    __syncthreads();
    float k[kEntries];
    bool full = true;
#pragma unroll
    for (int e = 0; e < kEntries; ++e) {
        k[e] = sk[e][px];
        full = full && k[e] != 0.0f;
    }
    const int share = (ncand + ranges - 1) / ranges;
    const int z0 = range * share, z1 = min(z0 + share, ncand);
    const int corner = (2 * Y - 2) * g.cols_out + 2 * X - 2;  // of the 5 x 5 fine pixels
    const bool in = o < pin;
    full = __all_sync(0xffffffffu, full) != 0;
#pragma unroll 2
    for (int z = z0; z < z1; ++z) {
        const float* gf = grad_f_fine + (int64_t)z * pio;
        float acc = 0.0f;
        if (full) {
            float v[5][5];
#pragma unroll
            for (int r = 0; r < 5; ++r)
#pragma unroll
                for (int c = 0; c < 5; ++c) v[r][c] = __ldg(gf + corner + r * g.cols_out + c);
#pragma unroll
            for (int e = 0; e < kEntries; ++e) {
                const TransposeEntry t = transpose_entry(e);
                acc = fmaf(k[e], v[2 * t.dy + (t.f & 1) + 2][2 * t.dx + (t.f >= 2) + 2], acc);
            }
        } else {
#pragma unroll
            for (int e = 0; e < kEntries; ++e) {
                const TransposeEntry t = transpose_entry(e);
                if (k[e] != 0.0f)
                    acc = fmaf(k[e], __ldg(gf + corner + (2 * t.dy + (t.f & 1) + 2) * g.cols_out + 2 * t.dx + (t.f >= 2) + 2),
                               acc);
            }
        }
        if (in) grad_f_coarse[(int64_t)z * pin + o] = acc;
    }
}

// Down step transposed: g_c(fine) = own weight * g_f(fine) + sum over the coarse pixels that read the
// cell.  A thread takes the 2 x 2 fine pixels of a coarse one, which are read by it and its right and
// lower neighbours (9 weights); a block takes 32 of them, its warps share out the weights and then the
// candidates.  kPairs: fine rows are read and written in pairs.  absmax (level 0, else nullptr): the
// largest |g_c| of the instance, as float bits.  (A thread per fine pixel that added to the up step's
// volume: 131 us at level 0 of two 512 x 512 references, 48 candidates, for its set-up; 53 now.)
struct QuadEntry {
    int a, b, n;  // fine column and row, reader
};
__host__ __device__ constexpr QuadEntry quad_entry(int e)
{
    return e == 0 ? QuadEntry{0, 0, 0}
         : e < 3  ? QuadEntry{1, 0, e - 1}
         : e < 5  ? QuadEntry{0, 1, (e - 3) * 2}
                  : QuadEntry{1, 1, e - 5};
}
constexpr int kQuadEntries = 9;

template <bool kPairs, int kThreads>
__global__ void __launch_bounds__(kThreads) isb_down_transpose_table_kernel(
    const float* __restrict__ tables, int64_t table_stride, LevelGeom g, int ncand, float weight_up,
    const float* __restrict__ grad_f_fine, const float* __restrict__ grad_c_coarse, float* __restrict__ grad_c_fine,
    uint32_t* __restrict__ absmax)
{
    __shared__ float sk[kQuadEntries + 4][32];
    const int pin = g.rows_in * g.cols_in, pio = g.rows_out * g.cols_out;
    const int64_t inst = blockIdx.y;
    tables += inst * table_stride;
    const int px = threadIdx.x & 31, range = threadIdx.x >> 5;
    constexpr int ranges = kThreads / 32;
    const int o = blockIdx.x * 32 + px, oc = min(o, pin - 1);
    const int y = oc / g.cols_in, x = oc - y * g.cols_in;
    const bool set1 = 2 * y + 1 < g.rows_out, set2 = 2 * x + 1 < g.cols_out;
#pragma unroll 1
    for (int e = range; e < kQuadEntries + 4; e += ranges) {
        if (e < kQuadEntries) {
            const QuadEntry q = quad_entry(e);
            const int X = 2 * x + q.a, Y = 2 * y + q.b;
            int rx, ry;
            sk[e][px] = X < g.cols_out && Y < g.rows_out && down_reader(g, q.n, X, Y, rx, ry)
                            ? down_read_weight(tables, g, rx, ry, X, Y) : 0.0f;
        } else {
            sk[e][px] = own_weight(e - kQuadEntries, tables, g, x, y, weight_up);
        }
    }
    __syncthreads();
    float k[kQuadEntries], own[4];
    bool full = true;
#pragma unroll
    for (int e = 0; e < kQuadEntries; ++e) {
        k[e] = sk[e][px];
        full = full && k[e] != 0.0f;
    }
#pragma unroll
    for (int f = 0; f < 4; ++f) own[f] = sk[kQuadEntries + f][px];
    const int share = (ncand + ranges - 1) / ranges;
    const int z0 = range * share, z1 = o < pin ? min(z0 + share, ncand) : 0;
    const int right = min(x + 1, g.cols_in - 1) - x, below = (min(y + 1, g.rows_in - 1) - y) * g.cols_in;
    const float* gc = grad_c_coarse + (inst * ncand + z0) * pin + oc;
    const int64_t fine = (inst * ncand + z0) * pio + 2 * y * g.cols_out + 2 * x;
    const float* gf = grad_f_fine + fine;
    float* out = grad_c_fine + fine;
    const int down = set1 ? g.cols_out : 0;
    uint32_t largest = 0;
#pragma unroll 2
    for (int z = z0; z < z1; ++z, gc += pin, gf += pio, out += pio) {
        const float v[4] = {__ldg(gc), __ldg(gc + right), __ldg(gc + below), __ldg(gc + below + right)};
        const float2 top = load_fine<kPairs>(gf, 0, set2), bottom = load_fine<kPairs>(gf, down, set2);
        const float mine[4] = {top.x, bottom.x, top.y, bottom.y};  // by f
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int e = 0; e < kQuadEntries; ++e) {
            const QuadEntry q = quad_entry(e);
            const int f = q.b + 2 * q.a;
            if (full || k[e] != 0.0f) acc[f] = fmaf(k[e], v[q.n], acc[f]);
        }
        float r[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            r[f] = fadd(fmul(own[f], mine[f]), acc[f]);
            if (((f & 1) && !set1) || (f >= 2 && !set2)) r[f] = 0.0f;
            largest = max(largest, __float_as_uint(r[f]) & 0x7FFFFFFFu);
        }
        if constexpr (kPairs) {
            *reinterpret_cast<float2*>(out) = make_float2(r[0], r[2]);
            if (set1) *reinterpret_cast<float2*>(out + g.cols_out) = make_float2(r[1], r[3]);
        } else {
            out[0] = r[0];
            if (set2) out[1] = r[2];
            if (set1) out[g.cols_out] = r[1];
            if (set1 && set2) out[g.cols_out + 1] = r[3];
        }
    }
    if (absmax) {
        largest = __reduce_max_sync(0xffffffffu, largest);
        // most warps find a larger value already there
        if (px == 0 && largest > *reinterpret_cast<volatile uint32_t*>(absmax + inst)) atomicMax(absmax + inst, largest);
    }
}

// The small levels in one launch, one block per (candidate, instance): the up steps transposed from
// level `first` to the coarsest level, and the down steps transposed back to level `first`, in shared
// memory.  grad_f: level `first`, in; grad_c: level `first`, out.
struct TransposeTail {
    int levels, first, ncand;
    int rows[SSG_MAX_LEVELS], cols[SSG_MAX_LEVELS];
    float weight_up[SSG_MAX_LEVELS];
    int64_t offset[SSG_MAX_LEVELS], stride;
};
__global__ void __launch_bounds__(kPlanarTailThreads) isb_transpose_tail_kernel(const __grid_constant__ TransposeTail T,
                                                                               const float* __restrict__ tables,
                                                                               const float* __restrict__ grad_f,
                                                                               float* __restrict__ grad_c)
{
    __shared__ float gf[kPlanarTailCells], gc[kPlanarTailCells];
    const int64_t inst = blockIdx.y;
    tables += inst * T.stride;
    int n = T.rows[T.first] * T.cols[T.first];
    const int64_t volume = (inst * T.ncand + blockIdx.x) * n;
    for (int i = threadIdx.x; i < n; i += kPlanarTailThreads) gf[i] = grad_f[volume + i];
    __syncthreads();
    int fine = 0;
    for (int s = T.first; s + 1 < T.levels; ++s) {
        const LevelGeom g{T.rows[s + 1], T.cols[s + 1], T.rows[s], T.cols[s]};
        const float* t = tables + T.offset[s];
        const int coarse = fine + g.rows_out * g.cols_out;
        for (int o = threadIdx.x; o < g.rows_in * g.cols_in; o += kPlanarTailThreads) {
            const int Y = o / g.cols_in, X = o - Y * g.cols_in;
            float acc = 0.0f;
#pragma unroll 1
            for (int e = 0; e < kEntries; ++e) {
                const TransposeEntry q = transpose_entry(e);
                const float k = read_weight(q.f, t, g, X + q.dx, Y + q.dy, X, Y);
                if (k != 0.0f)
                    acc = fmaf(k, gf[fine + (2 * (Y + q.dy) + (q.f & 1)) * g.cols_out + 2 * (X + q.dx) + (q.f >= 2)], acc);
            }
            gf[coarse + o] = acc;
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const int fx = 2 * X + (f >= 2), fy = 2 * Y + (f & 1);
                if (fx < g.cols_out && fy < g.rows_out)
                    gc[fine + fy * g.cols_out + fx] =
                        own_weight(f, t, g, X, Y, T.weight_up[s]) * gf[fine + fy * g.cols_out + fx];
            }
        }
        fine = coarse;
        __syncthreads();
    }
    // f = c at the coarsest level
    for (int i = threadIdx.x; i < T.rows[T.levels - 1] * T.cols[T.levels - 1]; i += kPlanarTailThreads)
        gc[fine + i] = gf[fine + i];
    __syncthreads();
    for (int s = T.levels - 1; s > T.first; --s) {
        const LevelGeom g{T.rows[s], T.cols[s], T.rows[s - 1], T.cols[s - 1]};
        const float* t = tables + T.offset[s - 1];
        const int coarse = fine;
        fine -= g.rows_out * g.cols_out;
        for (int i = threadIdx.x; i < g.rows_out * g.cols_out; i += kPlanarTailThreads) {
            const int Y = i / g.cols_out, X = i - Y * g.cols_out;
            float acc = 0.0f;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                int x, y;
                if (!down_reader(g, m, X, Y, x, y)) continue;
                const float k = down_read_weight(t, g, x, y, X, Y);
                if (k != 0.0f) acc = fmaf(k, gc[coarse + y * g.cols_in + x], acc);
            }
            gc[fine + i] += acc;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += kPlanarTailThreads) grad_c[volume + i] = gc[i];
}

// ---------------------------------------------------------------------------------------------
// Sweep backward
// ---------------------------------------------------------------------------------------------
constexpr int kBwdReferences = 4;  // of one launch (bounds the parameters)
constexpr int kBwdBlock = 256, kBwdTileX = 32, kBwdTileY = 8;

struct SweepBwdReferences {
    int cols, rows, ncam, ncand;
    float colsf, rowsf, inv_cols, inv_rows;
    int reference[kBwdReferences];
    TorchCam cams[SSG_MAX_CAMERAS];
    float rt[kBwdReferences][SSG_MAX_CAMERAS][12];
    float cand[SSG_MAX_CANDIDATES];
};

// v rounded to the nearest integer (__float2ll_rn, without the FP64 pipe), |v| < 2^62: multiples of 2^40
// and of 2^20 are taken off by sums with 1.5 x 2^63 and 1.5 x 2^43, whose last bits they are, and the
// rest is rounded by a sum with 1.5 x 2^23.  The differences are exact, and the parts taken off are
// even, so a tie rounds as v's does.  (inf and NaN give some number.)
__device__ __forceinline__ long long fixed_of(float v)
{
    const float a = fadd(v, 0x1.8p63f), va = fsub(v, fsub(a, 0x1.8p63f));
    const float b = fadd(va, 0x1.8p43f), vb = fsub(va, fsub(b, 0x1.8p43f));
    const float c = fadd(vb, 0x1.8p23f);
    const int ia = __float_as_int(a) - 0x5F400000, ib = __float_as_int(b) - 0x55400000;
    const int ic = __float_as_int(c) - 0x4B400000;
    return ((long long)ia << 40) + (long long)ib * (1 << 20) + ic;
}

// __ll2float_rn without the FP64 pipe: 24 leading bits, rounded to nearest even
__device__ __forceinline__ float float_of(long long q)
{
    const unsigned long long u = q < 0 ? 0ull - (unsigned long long)q : (unsigned long long)q;
    const int drop = 40 - __clzll((long long)u);  // bits below the 24 leading ones
    float f;
    if (drop <= 0) {
        f = (float)(int)u;
    } else {
        const unsigned long long rest = u & ((1ull << drop) - 1), half = 1ull << (drop - 1);
        uint32_t m = (uint32_t)(u >> drop);
        m += rest > half || (rest == half && (m & 1u)) ? 1u : 0u;
        f = (float)(int)m * __uint_as_float((uint32_t)(drop + 127) << 23);  // 2^drop: exact
    }
    return q < 0 ? -f : f;
}

__device__ __forceinline__ long long shfl_up64(long long v, int d)
{
    const int lo = __shfl_up_sync(0xffffffffu, (int)(uint32_t)v, d);
    const int hi = __shfl_up_sync(0xffffffffu, (int)(v >> 32), d);
    return (long long)(((unsigned long long)(uint32_t)hi << 32) | (uint32_t)lo);
}

__device__ __forceinline__ long long signed_part(long long q, int sign, int ch)
{
    const int s = (sign >> (2 * ch)) & 3;
    return s == 1 ? q : s == 2 ? -q : 0;
}

__device__ __forceinline__ void fixed_add(long long* p, long long q)
{
    if (q) atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)q);
}

// One step of a sum over lanes of kCount values each, `off` lanes apart: a lane keeps one half of the
// values and gives the other to its partner
template <int kCount>
__device__ __forceinline__ void halve(double (&v)[8], int off)
{
    const bool upper = (threadIdx.x & off) != 0;
#pragma unroll
    for (int j = 0; j < kCount / 2; ++j) {
        const double give = upper ? v[j] : v[j + kCount / 2], keep = upper ? v[j + kCount / 2] : v[j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
}

// project_jacobian, its quotients by d1 and d2 from their reciprocals
__device__ __forceinline__ void project_jacobian_packed(const float p[3], const TorchCam& k, float ju[3], float jv[3])
{
    const float x = p[0], y = p[1], z = p[2];
    const float d1 = sqrtf(x * x + y * y + z * z);
    const float c = k.xi * d1 + z;
    const float d2 = sqrtf(x * x + y * y + c * c);
    const float nrm = k.alpha * d2 + k.one_minus_alpha * c;
    float q1[3] = {k.xi * x, k.xi * y, k.xi * z}, q2[3], dc[3];
    const bool fine = d1 > 1e-10f && d1 < 1e10f && d2 > 1e-10f && d2 < 1e10f;
    if (fine) {
        const float r1 = __frcp_rn(d1);
#pragma unroll
        for (int j = 0; j < 3; ++j) q1[j] = div_by_reciprocal(q1[j], d1, r1);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j) q1[j] = fdiv(q1[j], d1);
    }
    dc[0] = q1[0];
    dc[1] = q1[1];
    dc[2] = q1[2] + 1.0f;
    q2[0] = k.alpha * (x + c * dc[0]);
    q2[1] = k.alpha * (y + c * dc[1]);
    q2[2] = k.alpha * (c * dc[2]);
    if (fine) {
        const float r2 = __frcp_rn(d2);
#pragma unroll
        for (int j = 0; j < 3; ++j) q2[j] = div_by_reciprocal(q2[j], d2, r2);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j) q2[j] = fdiv(q2[j], d2);
    }
    float dn[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) dn[j] = q2[j] + k.one_minus_alpha * dc[j];
    const float in = 1.0f / nrm, in2 = in * in;
    ju[0] = k.fx * (in - x * dn[0] * in2);
    ju[1] = k.fx * (-x * dn[1] * in2);
    ju[2] = k.fx * (-x * dn[2] * in2);
    jv[0] = k.fy * (-y * dn[0] * in2);
    jv[1] = k.fy * (in - y * dn[1] * in2);
    jv[2] = k.fy * (-y * dn[2] * in2);
}

// A block takes 32 x 8 pixels of one reference (blockIdx.z), a warp 8 x 4 of them: the samples of
// neighbouring pixels land on neighbouring texels, and what two lanes have for one texel is added in
// the warp.  Per pixel the candidates are taken in order (the float32 sums of the pose gradient).
// Bound by instruction issue, some 800 a sample with the warp's sums, and by how many warps hide their
// latency: two references of 512 x 512, 48 candidates, 1016 us with two blocks per SM (117
// registers), 888 with three, 825 with four (64 registers), 872 with five (spills).
__global__ void __launch_bounds__(kBwdBlock, 4) sweep_backward_references_kernel(
    const __grid_constant__ SweepBwdReferences p, const float4* __restrict__ packed, const int8_t* __restrict__ selected,
    const float* __restrict__ grad_cost, const uint32_t* __restrict__ absmax, long long* __restrict__ image_acc,
    double* __restrict__ pose_partial)
{
    const int64_t P = (int64_t)p.cols * p.rows;
    const int slot = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int reference = p.reference[slot];
    const float scale = fixed_scale(absmax[slot], 2.0 * (double)P * p.ncand);
    const int x = blockIdx.x * kBwdTileX + (warp & 3) * 8 + (lane & 7);
    const int y = blockIdx.y * kBwdTileY + (warp >> 2) * 4 + (lane >> 3);
    const bool inside = x < p.cols && y < p.rows;
    const int64_t i = inside ? (int64_t)y * p.cols + x : 0;
    const int sel = inside ? selected[slot * P + i] : -1;
    const bool active = sel >= 0 && sel < p.ncam;
    image_acc += (int64_t)slot * p.ncam * P * 3;
    grad_cost += (int64_t)slot * p.ncand * P + i;
    float gsrc[6] = {0, 0, 0, 0, 0, 0}, gref6[6] = {0, 0, 0, 0, 0, 0};
    float gref[3] = {0.0f, 0.0f, 0.0f};
    float pu[3] = {0.0f, 0.0f, 0.0f}, r[3] = {0.0f, 0.0f, 0.0f};
    const int s = active ? sel : 0;
    const TorchCam cam = p.cams[s];
    float rt[12];
#pragma unroll
    for (int j = 0; j < 12; ++j) rt[j] = p.rt[slot][s][j];
    if (active) {
        unproject_torch((float)x, (float)y, p.cams[reference], pu);
        const float4 t = __ldg(packed + reference * P + i);
        r[0] = t.x, r[1] = t.y, r[2] = t.z;
    }
    const float4* img = packed + s * P;
    long long* gimg = image_acc + s * P * 3;
    float g_next = active && p.ncand > 0 ? __ldg(grad_cost) : 0.0f;
    for (int k = 0; k < p.ncand; ++k) {
        const float g = g_next;
        if (active && k + 1 < p.ncand) g_next = __ldg(grad_cost + (int64_t)(k + 1) * P);
        bool live = active && g != 0.0f;
        if (!__any_sync(0xffffffffu, live)) continue;
        // |contribution| to the texels left / right of the sample in its upper and lower row; a channel's
        // is that, its negative or 0 (sign: 2 bits per channel)
        long long left[2] = {0, 0}, right[2] = {0, 0};
        int sign = 0;
        int tx = 0, ty = 0;
        bool lands = false;  // on a texel of the image
        if (live) {
            const float d = p.cand[k];
            const float pv[3] = {fmul(d, pu[0]), fmul(d, pu[1]), fmul(d, pu[2])};
            float q[3], uv[2];
            transform_torch(rt, pv, q);
            project_packed(q, cam, uv);
            const float ix = packed_sample_coord(uv[0], p.colsf, p.inv_cols);
            const float iy = packed_sample_coord(uv[1], p.rowsf, p.inv_rows);
            const float x0 = floorf(ix), y0 = floorf(iy), x1 = x0 + 1.0f, y1 = y0 + 1.0f;
            const float xs[4] = {x0, x1, x0, x1}, ys[4] = {y0, y0, y1, y1};
            const float w[4] = {(x1 - ix) * (y1 - iy), (ix - x0) * (y1 - iy), (x1 - ix) * (iy - y0),
                                (ix - x0) * (iy - y0)};
            // d w / d ix and d w / d iy
            const float wx[4] = {-(y1 - iy), (y1 - iy), -(iy - y0), (iy - y0)};
            const float wy[4] = {-(x1 - ix), -(ix - x0), (x1 - ix), (ix - x0)};
            float tv[4][3], sx[3] = {0, 0, 0}, sy[3] = {0, 0, 0};
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                in[t] = xs[t] >= 0.0f && xs[t] < p.colsf && ys[t] >= 0.0f && ys[t] < p.rowsf;
                tv[t][0] = tv[t][1] = tv[t][2] = 0.0f;  // zero padding
                if (in[t]) {
                    const float4 v = __ldg(img + ((int64_t)(int)ys[t] * p.cols + (int)xs[t]));
                    tv[t][0] = v.x, tv[t][1] = v.y, tv[t][2] = v.z;
                }
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) {
                    sx[ch] += tv[t][ch] * wx[t];
                    sy[ch] += tv[t][ch] * wy[t];
                }
            }
            // the sample as two horizontal interpolations and a vertical one: four equal taps give
            // exactly their value (a flat region's residual is exactly 0, the L1 kink's subgradient)
            const float fx = ix - x0, fy = iy - y0;
            float res[3];
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                const float top = tv[0][ch] + fx * (tv[1][ch] - tv[0][ch]);
                const float bot = tv[2][ch] + fx * (tv[3][ch] - tv[2][ch]);
                res[ch] = top + fy * (bot - top) - r[ch];
            }
            const float cost = fabsf(res[0]) + fabsf(res[1]) + fabsf(res[2]);
            live = !(cost > 500.0f);  // clamp(max=500) passes no gradient above the bound
            if (live) {
                float gs[3];
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) {
                    const float sg = res[ch] > 0.0f ? 1.0f : (res[ch] < 0.0f ? -1.0f : 0.0f);
                    gs[ch] = g * sg;
                    gref[ch] -= gs[ch];
                    sign |= (res[ch] > 0.0f ? 1 : res[ch] < 0.0f ? 2 : 0) << (2 * ch);
                }
                lands = in[0] || in[1] || in[2] || in[3];
                if (lands) {
                    tx = (int)x0;
                    ty = (int)y0;
                    if (in[0]) left[0] = fixed_of(g * w[0] * scale);
                    if (in[1]) right[0] = fixed_of(g * w[1] * scale);
                    if (in[2]) left[1] = fixed_of(g * w[2] * scale);
                    if (in[3]) right[1] = fixed_of(g * w[3] * scale);
                }
                // d ix / d u = d iy / d v = 1 (the normalisation round trip is the identity)
                const float gu = gs[0] * sx[0] + gs[1] * sx[1] + gs[2] * sx[2];
                const float gv = gs[0] * sy[0] + gs[1] * sy[1] + gs[2] * sy[2];
                float ju[3], jv[3];
                project_jacobian_packed(q, cam, ju, jv);
                const float gp[3] = {gu * ju[0] + gv * jv[0], gu * ju[1] + gv * jv[1], gu * ju[2] + gv * jv[2]};
                // source camera: p' = exp(-delta) p  ->  dL/domega = g x p, dL/dv = -g
                gsrc[0] += gp[1] * q[2] - gp[2] * q[1];
                gsrc[1] += gp[2] * q[0] - gp[0] * q[2];
                gsrc[2] += gp[0] * q[1] - gp[1] * q[0];
                gsrc[3] -= gp[0];
                gsrc[4] -= gp[1];
                gsrc[5] -= gp[2];
                // reference camera: p' = R (exp(delta) p_ref) + t  ->  with h = R^T g:
                // dL/domega = p_ref x h, dL/dv = h
                const float h[3] = {rt[0] * gp[0] + rt[4] * gp[1] + rt[8] * gp[2],
                                    rt[1] * gp[0] + rt[5] * gp[1] + rt[9] * gp[2],
                                    rt[2] * gp[0] + rt[6] * gp[1] + rt[10] * gp[2]};
                gref6[0] += pv[1] * h[2] - pv[2] * h[1];
                gref6[1] += pv[2] * h[0] - pv[0] * h[2];
                gref6[2] += pv[0] * h[1] - pv[1] * h[0];
                gref6[3] += h[0];
                gref6[4] += h[1];
                gref6[5] += h[2];
            }
        }
        // a sample whose left column is its left neighbour's right column takes that column over, and
        // one whose upper row is the upper neighbour's lower row takes its left column's texel
        const int key = lands ? s : -1;
        const int kx = __shfl_up_sync(0xffffffffu, tx, 1), ky = __shfl_up_sync(0xffffffffu, ty, 1);
        const int ks = __shfl_up_sync(0xffffffffu, key, 1);
        const bool from_left = (lane & 7) != 0 && lands && ks == key && ky == ty && kx + 1 == tx;
        const int left_sign = __shfl_up_sync(0xffffffffu, sign, 1);
        long long ql[2][3];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const long long t = shfl_up64(right[a], 1);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                ql[a][ch] = signed_part(left[a], sign, ch);
                if (from_left) ql[a][ch] += signed_part(t, left_sign, ch);
            }
        }
        const int right_took = __shfl_down_sync(0xffffffffu, (int)from_left, 1);  // every lane shuffles
        const bool given = (lane & 7) != 7 && right_took != 0;
        const int vx = __shfl_up_sync(0xffffffffu, tx, 8), vy = __shfl_up_sync(0xffffffffu, ty, 8);
        const int vs = __shfl_up_sync(0xffffffffu, key, 8);
        const bool from_above = lane >= 8 && lands && vs == key && vx == tx && vy + 1 == ty;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            const long long t = shfl_up64(ql[1][ch], 8);
            if (from_above) ql[0][ch] += t;
        }
        const int below_took = __shfl_down_sync(0xffffffffu, (int)from_above, 8);
        const bool given_down = lane < 24 && below_took != 0;
        if (lands) {
            long long* a = gimg + ((int64_t)ty * p.cols + tx);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch, a += P) {
                fixed_add(a, ql[0][ch]);
                if (!given_down) fixed_add(a + p.cols, ql[1][ch]);
                if (!given) {
                    fixed_add(a + 1, signed_part(right[0], sign, ch));
                    fixed_add(a + p.cols + 1, signed_part(right[1], sign, ch));
                }
            }
        }
    }
    if (active) {
        long long* gr = image_acc + (int64_t)reference * 3 * P + i;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) fixed_add(gr + ch * P, fixed_of(gref[ch] * scale));
    }
    // the pose gradient of the block, per camera: a pixel's candidates were summed in float32; pixels
    // are summed in float64 in a fixed order over the lanes of a warp, and the warps in order
    __shared__ double warp_sum[kBwdBlock / 32][6];
    const int64_t block = (int64_t)slot * gridDim.x * gridDim.y + blockIdx.y * gridDim.x + blockIdx.x;
    for (int c = 0; c < p.ncam; ++c) {
        const bool mine = active && (sel == c || c == reference);
        if (__any_sync(0xffffffffu, mine)) {
            double v[8];
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                v[j] = 0.0;
                if (active && sel == c) v[j] += (double)gsrc[j];
                if (active && c == reference) v[j] += (double)gref6[j];
            }
            v[6] = v[7] = 0.0;
            halve<8>(v, 16);
            halve<4>(v, 8);
            halve<2>(v, 4);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            const int j = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
            if ((lane & 3) == 0 && j < 6) warp_sum[warp][j] = v[0];
        } else if (lane < 6) {
            warp_sum[warp][lane] = 0.0;
        }
        __syncthreads();
        if (threadIdx.x < 6) {
            double t = 0.0;
            for (int w = 0; w < kBwdBlock / 32; ++w) t += warp_sum[w][threadIdx.x];
            pose_partial[(block * p.ncam + c) * 6 + threadIdx.x] = t;
        }
        __syncthreads();
    }
}

struct GradTargets {
    float* ptr[SSG_MAX_CAMERAS];
};

// grad_images[c] += the references' sums in order, image_acc * 2^-e each (NaN where a reference's
// incoming gradient was not finite).  image_acc: channels in planes, so that what a warp adds at
// neighbouring texels lies in one sector.  blockIdx.y: camera
__global__ void __launch_bounds__(kBwdBlock) image_grad_references_kernel(const long long* __restrict__ image_acc,
                                                                          int64_t pixels, int cameras, int references,
                                                                          const uint32_t* __restrict__ absmax,
                                                                          double count,
                                                                          const __grid_constant__ GradTargets out)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pixels) return;
    const int c = blockIdx.y;
    float* o = out.ptr[c] + 3 * i;
    float v[3] = {o[0], o[1], o[2]};
    for (int r = 0; r < references; ++r) {
        const float scale = fixed_scale(absmax[r], count);
        const float inv = scale > 0.0f ? 1.0f / scale : 0.0f;  // a power of two: exact
        const bool finite = __uint_as_float(absmax[r]) <= 3.0e38f;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            const long long q = image_acc[(((int64_t)r * cameras + c) * 3 + ch) * pixels + i];
            if (!finite) v[ch] = __int_as_float(0x7FFFFFFF);
            else if (q) v[ch] += float_of(q) * inv;
        }
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) o[ch] = v[ch];
}

// grad_pose[c][j] += the block sums: 256 threads' shares in a fixed order.  blockIdx.x: 6 c + j
__global__ void __launch_bounds__(kBwdBlock) pose_grad_references_kernel(const double* __restrict__ pose_partial,
                                                                         int64_t blocks, int cameras,
                                                                         double* __restrict__ grad_pose)
{
    __shared__ double sh[kBwdBlock / 32];
    double t = 0.0;
    for (int64_t b = threadIdx.x; b < blocks; b += kBwdBlock) t += pose_partial[b * cameras * 6 + blockIdx.x];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < kBwdBlock / 32; ++w) sum += sh[w];
        grad_pose[blockIdx.x] += sum;
    }
}

static int check_pyramid(int level_count, int rows, int cols, int candidate_count, int instances)
{
    SSG_REQUIRE(cols > 0 && rows > 0, "sizes must be positive");
    const int expected = (int)(std::fmin(std::log2((double)cols), std::log2((double)rows)) - 1);
    SSG_REQUIRE(level_count == expected && level_count >= 2 && level_count <= SSG_MAX_LEVELS,
                "level_count %d differs from the pyramid of a %dx%d image (%d, at least 2)", level_count, cols, rows,
                expected);
    SSG_REQUIRE((int64_t)rows * cols < ((int64_t)1 << 31), "a level of %dx%d pixels is too large", rows, cols);
    SSG_REQUIRE(candidate_count >= 1 && candidate_count <= SSG_MAX_CANDIDATES, "candidate_count out of range");
    SSG_REQUIRE(instances >= 1 && instances <= 65535, "instances out of range");
    return SSG_OK;
}

template <bool kBackward>
static int soft_argmin(const uint8_t* guide_in, const float* cost_in, const uint8_t* guide_fine, const float* cost_fine,
                       int rows, int cols, int ncand, int instances, double sigma_i, double sigma_s,
                       const float* candidates, float temperature, float* q, const float* grad_q, float* grad_F,
                       cudaStream_t st)
{
    SSG_REQUIRE(guide_in && cost_in && guide_fine && cost_fine && candidates, "null pointer");
    const int levels = cols > 0 && rows > 0 ? (int)(std::fmin(std::log2((double)cols), std::log2((double)rows)) - 1) : 0;
    if (int e = check_pyramid(levels, rows, cols, ncand, instances)) return e;
    SSG_REQUIRE(temperature > 0.0f && sigma_i > 0 && sigma_s > 0, "temperature and sigmas must be positive");
    const Levels c = isb_constants(2, sigma_i, sigma_s);
    const LevelGeom g{level_rows(rows, 1), level_rows(cols, 1), rows, cols};
    const SoftParams sp = soft_params(candidates, ncand, temperature);
    const dim3 grid(grid_1d((int64_t)g.rows_in * g.cols_in, 32), instances);
    const bool pairs = cols % 2 == 0 && (((uintptr_t)cost_fine | (uintptr_t)grad_F) & 7) == 0;
    const float* table = range_table(c.var_inv_i, st);
    if (pairs)
        isb_soft_kernel<true, kBackward><<<grid, 64, 0, st>>>(guide_in, cost_in, guide_fine, cost_fine, g, c.weight_up[0],
                                                              c.weight_down[0], c.var_inv_i, table, sp, q, grad_q, grad_F);
    else
        isb_soft_kernel<false, kBackward><<<grid, 64, 0, st>>>(guide_in, cost_in, guide_fine, cost_fine, g, c.weight_up[0],
                                                               c.weight_down[0], c.var_inv_i, table, sp, q, grad_q, grad_F);
    return launch_status("isb_soft_kernel");
}

}  // namespace ssg

using namespace ssg;

extern "C" int ssg_soft_argmin(const uint8_t* d_guide_coarse, const float* d_cost_coarse, const uint8_t* d_guide_fine,
                               const float* d_cost_fine, int rows, int cols, int candidate_count, int instances,
                               double sigma_i, double sigma_s, const float* candidates, float temperature,
                               float* d_inverse_distance, void* stream)
{
    SSG_REQUIRE(d_inverse_distance, "null pointer");
    return soft_argmin<false>(d_guide_coarse, d_cost_coarse, d_guide_fine, d_cost_fine, rows, cols, candidate_count,
                              instances, sigma_i, sigma_s, candidates, temperature, d_inverse_distance, nullptr, nullptr,
                              as_stream(stream));
}

extern "C" int ssg_soft_argmin_backward(const uint8_t* d_guide_coarse, const float* d_cost_coarse,
                                        const uint8_t* d_guide_fine, const float* d_cost_fine, int rows, int cols,
                                        int candidate_count, int instances, double sigma_i, double sigma_s,
                                        const float* candidates, float temperature, const float* d_grad_inverse_distance,
                                        float* d_grad_filtered, void* stream)
{
    SSG_REQUIRE(d_grad_inverse_distance && d_grad_filtered, "null pointer");
    return soft_argmin<true>(d_guide_coarse, d_cost_coarse, d_guide_fine, d_cost_fine, rows, cols, candidate_count,
                             instances, sigma_i, sigma_s, candidates, temperature, nullptr, d_grad_inverse_distance,
                             d_grad_filtered, as_stream(stream));
}

extern "C" size_t ssg_isb_table_floats(int rows, int cols, int level_count)
{
    if (rows <= 0 || cols <= 0 || level_count < 2 || level_count > SSG_MAX_LEVELS) return 0;
    size_t n = 0;
    for (int s = 1; s < level_count; ++s) n += (size_t)kTableRows * level_rows(rows, s) * level_rows(cols, s);
    return n;
}

extern "C" int ssg_isb_filter_transpose(uint8_t* const* d_guides, uint8_t* const* d_filtered_guides, int level_count,
                                        int rows, int cols, int candidate_count, int instances, double sigma_i,
                                        double sigma_s, float* const* d_grad_filtered, float* const* d_grad_costs,
                                        float* d_tables, uint32_t* d_absmax, void* stream)
{
    SSG_REQUIRE(d_guides && d_filtered_guides && d_grad_filtered && d_grad_costs && d_tables && d_absmax, "null pointer");
    if (int e = check_pyramid(level_count, rows, cols, candidate_count, instances)) return e;
    SSG_REQUIRE(sigma_i > 0 && sigma_s > 0, "sigmas must be positive");
    cudaStream_t st = as_stream(stream);
    const Levels c = isb_constants(level_count, sigma_i, sigma_s);
    TableLevels T{};
    T.levels = level_count;
    for (int s = 0; s < level_count; ++s) {
        SSG_REQUIRE(d_guides[s] && d_grad_filtered[s] && d_grad_costs[s] && (s == 0 || d_filtered_guides[s]),
                    "level %d is NULL", s);
        T.rows[s] = level_rows(rows, s);
        T.cols[s] = level_rows(cols, s);
        T.guides[s] = d_guides[s];
        T.filtered[s] = d_filtered_guides[s];
        T.weight_up[s] = c.weight_up[s];
        T.weight_down[s] = c.weight_down[s];
    }
    for (int s = 0; s + 1 < level_count; ++s) {
        const int64_t n = (int64_t)T.rows[s + 1] * T.cols[s + 1];
        T.offset[s] = T.stride;
        T.stride += kTableRows * n;
        T.first_group[s + 1] = T.first_group[s] + grid_1d(n, 32);
    }
    const float* table = range_table(c.var_inv_i, st);
    isb_table_kernel<<<dim3(T.first_group[level_count - 1], instances), 160, 0, st>>>(T, c.var_inv_i, table, d_tables);
    if (int e = launch_status("isb_table_kernel")) return e;
    const cudaError_t e = cudaMemsetAsync(d_absmax, 0, sizeof(uint32_t) * instances, st);
    if (e != cudaSuccess) return fail(SSG_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    const int first = planar_tail_first(T.rows, T.cols, level_count, 2);
    const auto pair = [&](int s) { return LevelGeom{T.rows[s + 1], T.cols[s + 1], T.rows[s], T.cols[s]}; };
    for (int s = 0; s + 1 < level_count && s < first; ++s) {
        const LevelGeom g = pair(s);
        const dim3 grid(grid_1d((int64_t)g.rows_in * g.cols_in, 32), instances);
        const bool full = (int64_t)grid.x * instances >= kTransposeFull;
        const auto kernel = full ? isb_up_transpose_table_kernel<kTransposeBlock / 2> : isb_up_transpose_table_kernel<kTransposeBlock>;
        kernel<<<grid, full ? kTransposeBlock / 2 : kTransposeBlock, 0, st>>>(
            d_tables + T.offset[s], T.stride, g, candidate_count, d_grad_filtered[s], d_grad_filtered[s + 1]);
        if (int err = launch_status("isb_up_transpose_table_kernel")) return err;
    }
    if (first < level_count) {
        TransposeTail t{};
        t.levels = level_count;
        t.first = first;
        t.ncand = candidate_count;
        t.stride = T.stride;
        std::memcpy(t.rows, T.rows, sizeof t.rows);
        std::memcpy(t.cols, T.cols, sizeof t.cols);
        std::memcpy(t.weight_up, T.weight_up, sizeof t.weight_up);
        std::memcpy(t.offset, T.offset, sizeof t.offset);
        isb_transpose_tail_kernel<<<dim3(candidate_count, instances), kPlanarTailThreads, 0, st>>>(
            t, d_tables, d_grad_filtered[first], d_grad_costs[first]);
        if (int err = launch_status("isb_transpose_tail_kernel")) return err;
    }
    for (int s = std::min(first, level_count - 1); s > 0; --s) {
        const LevelGeom g = pair(s - 1);
        // f = c at the coarsest level
        const float* coarse = s == level_count - 1 && first == level_count ? d_grad_filtered[s] : d_grad_costs[s];
        const dim3 grid(grid_1d((int64_t)g.rows_in * g.cols_in, 32), instances);
        const bool pairs = g.cols_out % 2 == 0 && (((uintptr_t)d_grad_filtered[s - 1] | (uintptr_t)d_grad_costs[s - 1]) & 7) == 0;
        const bool full = (int64_t)grid.x * instances >= kTransposeFull;
        constexpr int kHalf = kTransposeBlock / 2;
        const auto kernel = full ? (pairs ? isb_down_transpose_table_kernel<true, kHalf> : isb_down_transpose_table_kernel<false, kHalf>)
                                 : (pairs ? isb_down_transpose_table_kernel<true, kTransposeBlock>
                                          : isb_down_transpose_table_kernel<false, kTransposeBlock>);
        kernel<<<grid, full ? kHalf : kTransposeBlock, 0, st>>>(d_tables + T.offset[s - 1], T.stride, g, candidate_count,
                                                 c.weight_up[s - 1], d_grad_filtered[s - 1], coarse, d_grad_costs[s - 1],
                                                 s == 1 ? d_absmax : nullptr);
        if (int err = launch_status("isb_down_transpose_table_kernel")) return err;
    }
    return SSG_OK;
}

// scratch: the fixed-point image sums (reference_count x camera_count x pixels x 3 int64) and the block
// sums of the pose gradient
static int64_t bwd_blocks(int cols, int rows)
{
    return (int64_t)((cols + kBwdTileX - 1) / kBwdTileX) * ((rows + kBwdTileY - 1) / kBwdTileY);
}

extern "C" size_t ssg_sweep_backward_references_scratch_bytes(int cols, int rows, int camera_count, int reference_count)
{
    if (cols <= 0 || rows <= 0 || camera_count < 1 || camera_count > SSG_MAX_CAMERAS || reference_count < 1) return 0;
    return (size_t)reference_count * camera_count *
           ((size_t)cols * rows * 3 * 8 + (size_t)bwd_blocks(cols, rows) * 6 * 8);
}

extern "C" int ssg_sweep_backward_references(int cols, int rows, int camera_count, const ssg_camera* cameras,
                                             int reference_count, const int* references, const float* relative_poses,
                                             const float* d_packed, float* const* d_grad_images,
                                             const int8_t* d_selected, const float* candidates, int candidate_count,
                                             const float* d_grad_cost, const uint32_t* d_absmax, double* d_grad_pose,
                                             void* d_scratch, void* stream)
{
    SSG_REQUIRE(cols > 0 && rows > 0, "resolution must be positive");
    SSG_REQUIRE(cameras && references && relative_poses && d_packed && d_grad_images && d_selected && candidates &&
                    d_grad_cost && d_absmax && d_grad_pose && d_scratch,
                "null pointer");
    SSG_REQUIRE(((uintptr_t)d_packed & 15) == 0 && ((uintptr_t)d_scratch & 255) == 0,
                "d_packed must be 16-byte aligned, d_scratch 256-byte aligned");
    SSG_REQUIRE(camera_count >= 1 && camera_count <= SSG_MAX_CAMERAS, "camera_count out of range");
    SSG_REQUIRE(candidate_count >= 1 && candidate_count <= SSG_MAX_CANDIDATES, "candidate_count out of range");
    SSG_REQUIRE(reference_count >= 1, "reference_count must be positive");
    SweepBwdReferences p{};
    p.cols = cols;
    p.rows = rows;
    p.ncam = camera_count;
    p.ncand = candidate_count;
    p.colsf = (float)cols;
    p.rowsf = (float)rows;
    p.inv_cols = 1.0f / (float)cols;
    p.inv_rows = 1.0f / (float)rows;
    GradTargets out{};
    for (int c = 0; c < camera_count; ++c) {
        SSG_REQUIRE(d_grad_images[c], "gradient of image %d is NULL", c);
        p.cams[c] = make_torch_cam(cameras[c]);
        out.ptr[c] = d_grad_images[c];
    }
    for (int r = 0; r < reference_count; ++r)
        SSG_REQUIRE(references[r] >= 0 && references[r] < camera_count, "reference out of range");
    for (int k = 0; k < candidate_count; ++k) p.cand[k] = candidates[k];
    const int64_t P = (int64_t)cols * rows, blocks = bwd_blocks(cols, rows);
    const size_t acc_bytes = (size_t)reference_count * camera_count * P * 3 * 8;
    long long* image_acc = static_cast<long long*>(d_scratch);
    double* pose_partial = reinterpret_cast<double*>(static_cast<uint8_t*>(d_scratch) + acc_bytes);
    cudaStream_t st = as_stream(stream);
    const cudaError_t e = cudaMemsetAsync(d_scratch, 0, acc_bytes, st);
    if (e != cudaSuccess) return fail(SSG_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    for (int r0 = 0; r0 < reference_count; r0 += kBwdReferences) {
        const int count = std::min(kBwdReferences, reference_count - r0);
        for (int r = 0; r < count; ++r) {
            p.reference[r] = references[r0 + r];
            std::memcpy(p.rt[r], relative_poses + (int64_t)(r0 + r) * camera_count * 12,
                        sizeof(float) * 12 * camera_count);
        }
        const dim3 grid((cols + kBwdTileX - 1) / kBwdTileX, (rows + kBwdTileY - 1) / kBwdTileY, count);
        sweep_backward_references_kernel<<<grid, kBwdBlock, 0, st>>>(
            p, reinterpret_cast<const float4*>(d_packed), d_selected + r0 * P, d_grad_cost + r0 * P * candidate_count,
            d_absmax + r0, image_acc + r0 * camera_count * P * 3, pose_partial + r0 * blocks * camera_count * 6);
        if (int err = launch_status("sweep_backward_references_kernel")) return err;
    }
    image_grad_references_kernel<<<dim3(grid_1d(P, kBwdBlock), camera_count), kBwdBlock, 0, st>>>(
        image_acc, P, camera_count, reference_count, d_absmax, 2.0 * (double)P * candidate_count, out);
    if (int err = launch_status("image_grad_references_kernel")) return err;
    pose_grad_references_kernel<<<camera_count * 6, kBwdBlock, 0, st>>>(pose_partial, blocks * reference_count,
                                                                       camera_count, d_grad_pose);
    return launch_status("pose_grad_references_kernel");
}
