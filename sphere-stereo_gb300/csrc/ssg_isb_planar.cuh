// ISB filter steps on planar volumes of several candidates, [candidates][rows][cols] float32, the
// reference's layout (python/isb_filter.cu:44-329): the fp32 path, ISB_Filter and the
// differentiable sweep.
//
// A block takes consecutive pixels of the coarse level and all their candidates: each pixel's guide
// weights are formed once per block, spread over the warps, and left in shared memory; then
// kRanges groups of threads each take a range of the candidates, every thread keeping its pixel's
// weights in registers, with no barrier between candidates.  Weights, sums and the reference's
// operation order are those of ssg_isb_common.cuh, so the bits do not depend on how the candidates
// are shared out.
//
// What bounds the steps: the latency of the loads in flight, against 34 + 134 MB (down) and 34 + 2 x
// 134 MB (up) to move at 1024^2 x 32 candidates, 25 and 45 us at the measured copy rate.  One block
// of a tile staged per candidate between two barriers, as the steps ran before, took 74 and 132 us
// there, and 26 us on every small level, whose time is one thread's chain over all candidates;
// now 45 and 115 us from cold caches (95 us when the caller has just written the volume), and 5 to 8 us.
#pragma once

#include "ssg_isb_common.cuh"

namespace ssg {

constexpr int kPlanarBlock = 256;

// The range weight of a colour distance from the table in global memory (through L1: a block of 32
// pixels looks up 256 to 800 of the 766 entries, so a copy per block in shared memory would cost
// more than the lookups), or evaluated when there is no table.
struct TableRange {
    const float* __restrict__ table;
    float var_inv_i;
    __device__ __forceinline__ float operator()(int d) const
    {
        return table ? __ldg(table + d) : range_weight((float)d, var_inv_i);
    }
};

// Columns 2x and 2x + 1 of the three rows a coarse pixel reads, and column 2x - 1 where the previous
// lane does not hold it.  kPairs: both columns in one 8-byte access (cols_in even, levels 8-byte
// aligned).
struct DownCells {
    float a[3], b[3], l[3];
};
template <bool kPairs>
__device__ __forceinline__ void load_down(const float* __restrict__ c, const int (&row)[3], int x2, int xp, bool left,
                                          DownCells& d)
{
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        if constexpr (kPairs) {
            const float2 v = __ldg(reinterpret_cast<const float2*>(c + row[r] + x2));
            d.a[r] = v.x;
            d.b[r] = v.y;
        } else {
            d.a[r] = __ldg(c + row[r] + x2);
            d.b[r] = __ldg(c + row[r] + xp);
        }
        if (left) d.l[r] = __ldg(c + row[r] + x2 - 1);
    }
}

// Down step of a level pair.  blockIdx.x: group of kPx coarse pixels; blockIdx.y: instance of
// contiguous volumes.  A lane loads columns 2x and 2x + 1 and takes column 2x - 1 from the lane
// before it, kDownDepth candidates ahead of their use.
constexpr int kDownDepth = 2;

template <int kRanges, bool kPairs, typename GL>
__global__ void __launch_bounds__(kPlanarBlock, 4) isb_down_planar_kernel(
    const uint8_t* __restrict__ guide_in, const float* __restrict__ cost_in, uint8_t* __restrict__ guide_out,
    float* __restrict__ cost_out, LevelGeom g, int ncand, float var_inv_i, const float* __restrict__ table)
{
    constexpr int kPx = kPlanarBlock / kRanges;
    __shared__ float sw[8][kPx];
    const int pin = g.rows_in * g.cols_in, pout = g.rows_out * g.cols_out;  // below 2^31 (check_levels)
    const int64_t inst = blockIdx.y;
    guide_in += inst * pin * GL::bytes;
    guide_out += inst * pout * GL::bytes;
    cost_in += inst * ncand * pin;
    cost_out += inst * ncand * pout;
    const int px = threadIdx.x % kPx, range = threadIdx.x / kPx;
    const int o = blockIdx.x * kPx + px;
    const bool in = o < pout;
    const int oc = min(o, pout - 1);
    const int y = oc / g.cols_out, x = oc - y * g.cols_out;
    const int x2 = 2 * x, y2 = 2 * y;
    const int xp = min(x2 + 1, g.cols_in - 1), xm = max(x2 - 1, 0);
    const int row[3] = {max(y2 - 1, 0) * g.cols_in, y2 * g.cols_in, min(y2 + 1, g.rows_in - 1) * g.cols_in};
    const int share = (ncand + kRanges - 1) / kRanges;
    const int k0 = range * share, k1 = min(k0 + share, ncand);  // uniform over a warp: a range is whole warps
    const bool left = (threadIdx.x & 31) == 0 && x > 0;
    DownCells cell[kDownDepth];
    const float* c = cost_in + (int64_t)k0 * pin;
#pragma unroll
    for (int j = 0; j < kDownDepth; ++j)
        if (k0 + j < k1) load_down<kPairs>(c + (int64_t)j * pin, row, x2, xp, left, cell[j]);
    // the eight neighbours in the reference's order (isb_filter.cu:75-104)
    const int idx[8] = {row[0] + xm, row[1] + xm, row[2] + xm, row[2] + x2, row[2] + xp, row[1] + xp, row[0] + xp,
                        row[0] + x2};
    const TableRange rw{table, var_inv_i};
    const typename GL::Pix cur = GL::load(guide_in, row[1] + x2);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (i % kRanges == range)
            sw[i][px] = fmul(i % 2 ? 0.5f : 0.25f, rw(GL::dist(cur, GL::load(guide_in, idx[i]))));
    __syncthreads();
    float w[8], wsum = 1.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        w[i] = sw[i][px];
        wsum = fadd(wsum, w[i]);
    }
    if (range == 0 && in) {
        float gs[3] = {(float)GL::ch(cur, 0), (float)GL::ch(cur, 1), (float)GL::ch(cur, 2)};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const typename GL::Pix nb = GL::load(guide_in, idx[i]);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) gs[ch] = fadd(gs[ch], fmul((float)GL::ch(nb, ch), w[i]));
        }
        const float den = fdiv(1.0f, wsum);
        uint32_t v[3];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) v[ch] = __float2uint_rz(fmul(gs[ch], den));
        GL::store(guide_out, o, v);
    }
    __syncwarp();
    const bool first = x == 0;
    for (int k = k0; k < k1; k += kDownDepth) {
#pragma unroll
        for (int j = 0; j < kDownDepth; ++j) {
            if (k + j >= k1) break;
            const DownCells d = cell[j];
            if (k + j + kDownDepth < k1)
                load_down<kPairs>(c + (int64_t)kDownDepth * pin, row, x2, xp, left, cell[j]);
            float m[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const float prev = __shfl_up_sync(0xffffffffu, d.b[r], 1);
                m[r] = first ? d.a[r] : left ? d.l[r] : prev;
            }
            const float t[8] = {m[0], m[1], m[2], d.a[2], d.b[2], d.b[1], d.b[0], d.a[0]};
            float acc = d.a[1];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc = fadd(acc, fmul(t[i], w[i]));
            if (in) cost_out[(int64_t)(k + j) * pout + o] = fdiv(acc, wsum);
            c += pin;
        }
    }
}

// Offsets of the fine pixels' weights and of the reciprocals of their sums in a pixel's 29 values
template <int F>
constexpr int up_weight_row()
{
    return F == 0 ? 0 : F == 1 ? 9 : F == 2 ? 15 : 21;
}
constexpr int kUpInvRow = 25, kUpRows = 29;
constexpr int kUpDepth = 2;

// Weights of fine pixel F of coarse pixel (x, y) into column `px` of sw, and its filtered guide
template <int F, int kPx, typename GL>
__device__ __forceinline__ void planar_fine_setup(const uint8_t* __restrict__ guide_in, const uint8_t* guide_fine,
                                                  uint8_t* guide_out, const LevelGeom& g, int x, int y, bool in_level,
                                                  float weight_up, float weight_down, const TableRange& range, int px,
                                                  float (&sw)[kUpRows][kPx])
{
    const int fx = 2 * x + (F >= 2 ? 1 : 0), fy = 2 * y + (F & 1);
    if (!in_level || fx >= g.cols_out || fy >= g.rows_out) return;  // no such pixel: its weights are not read
    int ci[9];
    typename GL::Pix gd[9];
    coarse_neighbourhood<int, GL>(guide_in, g.rows_in, g.cols_in, x, y, ci, gd);  // unused taps are not loaded
    const int index = fy * g.cols_out + fx;
    const typename GL::Pix up = GL::load(guide_fine, index);
    float w[UpTaps<F>::n], gs[3];
    const float inv = fine_weights<F, TableRange, GL>(gd, up, weight_up, weight_down, range, w, gs);
#pragma unroll
    for (int i = 0; i < UpTaps<F>::n; ++i) sw[up_weight_row<F>() + i][px] = w[i];
    sw[kUpInvRow + F][px] = inv;
    if (!guide_out) return;
    uint32_t v[3];
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) v[ch] = __float2uint_rz(fmul(gs[ch], inv));
    GL::store(guide_out, index, v);
}

// What one range of consecutive candidates contributes to a pixel's selection: a Selector that saw
// only its candidates, and its first and last cost for the neighbouring ranges
struct RangeSelection {
    float m, M, L, R, first, last;
    int idx_need;  // 2 x index of the minimum + whether it is the range's last candidate
};

// The two fine pixels' costs of a row of one candidate.  kPairs: in one 8-byte access (cols_out even
// and the levels 8-byte aligned, so every row of every plane is).
template <bool kPairs>
__device__ __forceinline__ float2 load_fine(const float* __restrict__ c, int at, bool second)
{
    if constexpr (kPairs) return *reinterpret_cast<const float2*>(c + at);
    else return make_float2(c[at], second ? c[at + 1] : 0.0f);
}

// How many candidates ahead of its use a step asks for its lines to be brought into L2 (0: not).  Rows
// read value by value (an odd width) gain by it, the selecting step with registers for 10 blocks of 64
// threads: 4 x 637 x 479 x 43, level 1 58 -> 49.5 us, selecting level 204 -> 192 us, the frame 938 -> 925 us.
// Rows read in pairs lose: 1024^2 x 32 filtered 311 -> 316 us, a frame of 2 x 1024^2 x 32 1097 -> 1107 us.
// (Measured at these sizes only, where a block has one range of candidates.)
template <bool kPairs>
constexpr int kUpAhead = kPairs ? 0 : 4;

// blocks per SM the up step's registers are bounded for: 640 threads (odd widths, selecting) or 768 with one
// range, as many as whole blocks hold with more (of 4 ranges 2 and 3 blocks of 256 threads), 1024 with 8
template <int kRanges, bool kSelect, bool kPairs>
constexpr int up_blocks = kRanges == 8 ? 2 : (kSelect && !kPairs ? 10 : 12) / kRanges;

// Candidates [k0, k1) of the two fine pixels FA, FB of one fine row of coarse pixel (x, y) in column
// `px` of sw, filtered; sink.take(k, at, a, b) gets each pair, `at` the pair's place in the level.
template <int FA, int FB, bool kPairs, typename Sink>
__device__ __forceinline__ void planar_up_row(const float* __restrict__ cost_in, const float* cost_fine,
                                              const LevelGeom& g, int x, int y, int k0, int k1, float weight_up,
                                              const float (&sw)[kUpRows][32], int px, Sink& sink)
{
    const int fy = 2 * y + (FA & 1);
    const bool second = 2 * x + 1 < g.cols_out;
    const int pin = g.rows_in * g.cols_in, pio = g.rows_out * g.cols_out;
    const int rr[3] = {max(y - 1, 0) * g.cols_in, y * g.cols_in, min(y + 1, g.rows_in - 1) * g.cols_in};
    const int cc[3] = {max(x - 1, 0), x, min(x + 1, g.cols_in - 1)};
    const int f0 = fy * g.cols_out + 2 * x;
    // fine costs, which come from memory, are loaded kUpDepth candidates ahead of their use; the
    // coarse taps, which neighbouring threads share in the caches, one ahead
    float2 own[kUpDepth];
    const float* c = cost_in + (int64_t)k0 * pin;
    const float* f = cost_fine + (int64_t)k0 * pio;
#pragma unroll
    for (int j = 0; j < kUpDepth; ++j)
        if (k0 + j < k1) own[j] = load_fine<kPairs>(f + (int64_t)j * pio, f0, second);
    float cd[9];
#pragma unroll
    for (int t = 0; t < 9; ++t)
        if (uses_tap<FA>(t) || uses_tap<FB>(t)) cd[t] = __ldg(c + rr[t / 3] + cc[t % 3]);
    float wa[UpTaps<FA>::n], wb[UpTaps<FB>::n];
#pragma unroll
    for (int i = 0; i < UpTaps<FA>::n; ++i) wa[i] = sw[up_weight_row<FA>() + i][px];
#pragma unroll
    for (int i = 0; i < UpTaps<FB>::n; ++i) wb[i] = sw[up_weight_row<FB>() + i][px];
    const float inv_a = sw[kUpInvRow + FA][px], inv_b = sw[kUpInvRow + FB][px];
    for (int k = k0; k < k1; k += kUpDepth) {
#pragma unroll
        for (int j = 0; j < kUpDepth; ++j) {
            if (k + j >= k1) break;
            float nd[9];
            if (k + j + 1 < k1) {
                c += pin;
#pragma unroll
                for (int t = 0; t < 9; ++t)
                    if (uses_tap<FA>(t) || uses_tap<FB>(t)) nd[t] = __ldg(c + rr[t / 3] + cc[t % 3]);
            }
            // isb_filter.cu:270-327
            float va = fmul(weight_up, own[j].x), vb = fmul(weight_up, own[j].y);
#pragma unroll
            for (int i = 0; i < UpTaps<FA>::n; ++i) {
                va = fadd(va, fmul(wa[i], cd[UpTaps<FA>::tap(i)]));
                if (i < UpTaps<FB>::n) vb = fadd(vb, fmul(wb[i < UpTaps<FB>::n ? i : 0], cd[UpTaps<FB>::tap(i)]));
            }
            va = fmul(va, inv_a);
            vb = fmul(vb, inv_b);
            constexpr int kAhead = Sink::kAhead;
            if (kAhead && k + j + kAhead < k1) {
                if ((px & 15) == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(f + (int64_t)kAhead * pio + f0));
                if (px == 8)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(c + (int64_t)(kAhead - 1) * pin + rr[2] + cc[1]));
            }
            if (k + j + kUpDepth < k1) own[j] = load_fine<kPairs>(f + (int64_t)kUpDepth * pio, f0, second);
            sink.take(k + j, f0, va, vb);
            f += pio;
#pragma unroll
            for (int t = 0; t < 9; ++t)
                if (uses_tap<FA>(t) || uses_tap<FB>(t)) cd[t] = nd[t];
        }
    }
}

// writes the pairs to a level
template <bool kPairs>
struct StoreSink {
    static constexpr int kAhead = kUpAhead<kPairs>;
    float* level;
    int pio;
    bool second;
    __device__ __forceinline__ void take(int k, int at, float a, float b)
    {
        float* p = level + (int64_t)k * pio + at;
        if constexpr (kPairs) {
            *reinterpret_cast<float2*>(p) = make_float2(a, b);
        } else {
            p[0] = a;
            if (second) p[1] = b;
        }
    }
};

// selects among the candidates of a range that starts at k0
template <bool kPairs>
struct SelectSink {
    static constexpr int kAhead = kUpAhead<kPairs>;
    int k0;
    Selector a, b;
    float first_a = 0.0f, first_b = 0.0f;
    __device__ __forceinline__ void take(int k, int, float va, float vb)
    {
        if (k == k0) {
            first_a = va;
            first_b = vb;
        }
        a.push(k, va);
        b.push(k, vb);
    }
    __device__ __forceinline__ static RangeSelection range(const Selector& s, float first)
    {
        return RangeSelection{s.m, s.M, s.L, s.R, first, s.prev, 2 * s.idx + (s.need_right ? 1 : 0)};
    }
};

// The weights of a block's 32 coarse pixels into sw, the four fine pixels by four of its warps (the
// caller synchronises the block)
template <typename GL>
__device__ __forceinline__ void planar_setup(const uint8_t* __restrict__ guide_in, const uint8_t* guide_fine,
                                             uint8_t* guide_out, const LevelGeom& g, int x, int y, bool in,
                                             float weight_up, float weight_down, const TableRange& range,
                                             float (&sw)[kUpRows][32])
{
    const int px = threadIdx.x & 31;
    for (int f = threadIdx.x >> 5; f < 4; f += blockDim.x >> 5) {
        switch (f) {
        case 0:
            planar_fine_setup<0, 32, GL>(guide_in, guide_fine, guide_out, g, x, y, in, weight_up, weight_down, range, px, sw);
            break;
        case 1:
            planar_fine_setup<1, 32, GL>(guide_in, guide_fine, guide_out, g, x, y, in, weight_up, weight_down, range, px, sw);
            break;
        case 2:
            planar_fine_setup<2, 32, GL>(guide_in, guide_fine, guide_out, g, x, y, in, weight_up, weight_down, range, px, sw);
            break;
        default:
            planar_fine_setup<3, 32, GL>(guide_in, guide_fine, guide_out, g, x, y, in, weight_up, weight_down, range, px, sw);
        }
    }
}

// Up step of a level pair: coarse filtered level -> fine level in place, or (kSelect) the last
// step fused with the selection, its candidates shared out in consecutive ranges and combined in
// candidate order.  A block takes 32 coarse pixels; a warp filters one of their two fine rows in
// one of kRanges ranges of candidates.  The filtered fine guide goes to guide_out (guide_fine itself,
// another pyramid's level, or none).  blockIdx.x: group of coarse pixels; blockIdx.y: instance.
template <int kRanges, bool kSelect, bool kPairs, typename GL>
__global__ void __launch_bounds__(64 * kRanges, up_blocks<kRanges, kSelect, kPairs>) isb_up_planar_kernel(
    const uint8_t* __restrict__ guide_in, const float* __restrict__ cost_in, const uint8_t* guide_fine,
    uint8_t* guide_out, float* cost_io, LevelGeom g, int ncand, float weight_up, float weight_down, float var_inv_i,
    const float* __restrict__ table, SelectOut so)
{
    constexpr int kPx = 32;
    __shared__ float sw[kUpRows][kPx];
    __shared__ RangeSelection part[kSelect ? kRanges : 1][kSelect ? 4 * kPx : 1];
    const int pin = g.rows_in * g.cols_in, pio = g.rows_out * g.cols_out;  // below 2^31 (check_levels)
    const int64_t inst = blockIdx.y;
    guide_in += inst * pin * GL::bytes;
    guide_fine += inst * pio * GL::bytes;
    if (guide_out) guide_out += inst * pio * GL::bytes;
    cost_in += inst * ncand * pin;
    cost_io += inst * ncand * pio;
    const int px = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int o = blockIdx.x * kPx + px;
    const bool in = o < pin;
    const int y = o / g.cols_in, x = o - y * g.cols_in;
    planar_setup<GL>(guide_in, guide_fine, guide_out, g, x, y, in, weight_up, weight_down, TableRange{table, var_inv_i}, sw);
    __syncthreads();
    const int share = (ncand + kRanges - 1) / kRanges, range = warp >> 1;
    const int k0 = range * share, k1 = min(k0 + share, ncand);
    const bool upper = (warp & 1) == 0;  // the fine row of F = 0, 2, or of F = 1, 3
    if (in && k0 < k1 && (upper || 2 * y + 1 < g.rows_out)) {
        if constexpr (kSelect) {
            using Sink = SelectSink<kPairs>;
            Sink sink{k0};
            if (upper) planar_up_row<0, 2, kPairs>(cost_in, cost_io, g, x, y, k0, k1, weight_up, sw, px, sink);
            else planar_up_row<1, 3, kPairs>(cost_in, cost_io, g, x, y, k0, k1, weight_up, sw, px, sink);
            part[range][(upper ? 0 : kPx) + px] = Sink::range(sink.a, sink.first_a);
            part[range][(upper ? 2 * kPx : 3 * kPx) + px] = Sink::range(sink.b, sink.first_b);
        } else {
            StoreSink<kPairs> sink{cost_io, pio, 2 * x + 1 < g.cols_out};
            if (upper) planar_up_row<0, 2, kPairs>(cost_in, cost_io, g, x, y, k0, k1, weight_up, sw, px, sink);
            else planar_up_row<1, 3, kPairs>(cost_in, cost_io, g, x, y, k0, k1, weight_up, sw, px, sink);
        }
    }
    if constexpr (kSelect) {
        __syncthreads();
        // one thread per fine pixel: the ranges in candidate order, as one Selector would have seen them
        for (int q = warp; q < 4; q += 2 * kRanges) {
            const int fx = 2 * x + (q >= 2 ? 1 : 0), fy = 2 * y + (q & 1);
            if (!in || fx >= g.cols_out || fy >= g.rows_out) continue;
            Selector s;
            for (int r = 0; r * share < ncand; ++r) {
                const RangeSelection p = part[r][q * kPx + px];
                if (s.need_right) s.R = p.first;
                s.need_right = false;
                if (p.m < s.m) {
                    s.m = p.m;
                    s.idx = p.idx_need >> 1;
                    s.L = s.idx == r * share ? s.prev : p.L;
                    s.R = p.R;
                    s.need_right = (p.idx_need & 1) != 0;
                }
                s.M = fmaxf(p.M, s.M);
                s.prev = p.last;
            }
            const int64_t at = inst * pio + fy * g.cols_out + fx;
            const float d = select_from(s, ncand, so.d0, so.dl, so.q);
            so.distance[at] = d;
            if (so.distance2) so.distance2[at] = d;
            if (so.index) so.index[at] = s.idx;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The small levels of the pyramid in one launch: one block per (candidate, instance) takes the down
// step into level `first`, every level below it and the up steps back to level `first`, in shared
// memory.  Every block forms the guides and weights for itself (they are few), the first candidate's
// writes the guides; no other block reads what it writes.  The steps are those of the kernels
// above, value by value (same bits).  A launch per step takes 5 to 8 us on such a level; the
// pyramid of 1024^2 x 32 took seven of them, 48 us, and takes 12.5 us here.
// ---------------------------------------------------------------------------------------------
constexpr int kPlanarTailPixels = 1024;  // of level `first`
constexpr int kPlanarTailCells = 1536;   // of level `first` and below: the next level of an r x c level
                                         // with r, c >= 8 holds at most 81 / 256 of its pixels
constexpr int kPlanarTailThreads = 512;

struct PlanarTail {
    int levels, first, ncand;
    int rows[SSG_MAX_LEVELS], cols[SSG_MAX_LEVELS];
    uint8_t* guides[SSG_MAX_LEVELS];    // unfiltered; level first - 1 is read
    uint8_t* filtered[SSG_MAX_LEVELS];  // filtered (the same arrays, or others)
    float* costs[SSG_MAX_LEVELS];
    float weight_up[SSG_MAX_LEVELS], weight_down[SSG_MAX_LEVELS];
};

// one coarse pixel of a down step, from global (GL) or shared (G4) memory
template <typename GL>
__device__ __forceinline__ void tail_down(const uint8_t* guide_in, const float* cost_in, int rows_in, int cols_in, int x,
                                          int y, const float* lut, uint32_t& guide, float& cost)
{
    const int x2 = 2 * x, y2 = 2 * y;
    const int xp = min(x2 + 1, cols_in - 1), yp = min(y2 + 1, rows_in - 1), xm = max(x2 - 1, 0), ym = max(y2 - 1, 0);
    const int idx[8] = {ym * cols_in + xm, y2 * cols_in + xm, yp * cols_in + xm, yp * cols_in + x2,
                        yp * cols_in + xp, y2 * cols_in + xp, ym * cols_in + xp, ym * cols_in + x2};
    const int centre = y2 * cols_in + x2;
    const typename GL::Pix cur = GL::load(guide_in, centre);
    float gs[3] = {(float)GL::ch(cur, 0), (float)GL::ch(cur, 1), (float)GL::ch(cur, 2)};
    float wsum = 1.0f, acc = cost_in[centre];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const typename GL::Pix nb = GL::load(guide_in, idx[i]);
        const float w = fmul(i % 2 ? 0.5f : 0.25f, lut[GL::dist(cur, nb)]);
        wsum = fadd(wsum, w);
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) gs[ch] = fadd(gs[ch], fmul((float)GL::ch(nb, ch), w));
        acc = fadd(acc, fmul(cost_in[idx[i]], w));
    }
    const float den = fdiv(1.0f, wsum);
    guide = 0;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) guide |= __float2uint_rz(fmul(gs[ch], den)) << (8 * ch);
    cost = fdiv(acc, wsum);
}

// fine pixel F of coarse pixel (x, y) of an up step in shared memory
template <int F>
__device__ __forceinline__ void tail_up(const uint32_t* guide_in, const float* cost_in, uint32_t* guide_io, float* cost_io,
                                        const LevelGeom& g, int x, int y, float weight_up, float weight_down,
                                        const LutRange& range)
{
    const int fx = 2 * x + (F >= 2 ? 1 : 0), fy = 2 * y + (F & 1);
    if (fx >= g.cols_out || fy >= g.rows_out) return;
    const int rr[3] = {max(y - 1, 0) * g.cols_in, y * g.cols_in, min(y + 1, g.rows_in - 1) * g.cols_in};
    const int cc[3] = {max(x - 1, 0), x, min(x + 1, g.cols_in - 1)};
    const int index = fy * g.cols_out + fx;
    G4::Pix gd[9];
    float cd[9];
#pragma unroll
    for (int t = 0; t < 9; ++t)
        if (uses_tap<F>(t)) {
            gd[t] = guide_in[rr[t / 3] + cc[t % 3]];
            cd[t] = cost_in[rr[t / 3] + cc[t % 3]];
        }
    float w[UpTaps<F>::n], gs[3];
    const float inv = fine_weights<F, LutRange, G4>(gd, guide_io[index], weight_up, weight_down, range, w, gs);
    float s = fmul(weight_up, cost_io[index]);
#pragma unroll
    for (int i = 0; i < UpTaps<F>::n; ++i) s = fadd(s, fmul(w[i], cd[UpTaps<F>::tap(i)]));
    cost_io[index] = fmul(s, inv);
    uint32_t v = 0;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) v |= __float2uint_rz(fmul(gs[ch], inv)) << (8 * ch);
    guide_io[index] = v;
}

template <typename GL>
__device__ __forceinline__ void tail_store_guides(const PlanarTail& T, uint8_t* const* to, int64_t inst,
                                                  const uint32_t* guides)
{
    int at = 0;
    for (int s = T.first; s < T.levels; ++s) {
        const int n = T.rows[s] * T.cols[s];
        for (int i = threadIdx.x; i < n; i += kPlanarTailThreads) {
            const uint32_t q = guides[at + i], v[3] = {q & 255u, (q >> 8) & 255u, (q >> 16) & 255u};
            GL::store(to[s] + inst * n * GL::bytes, i, v);
        }
        at += n;
    }
}

// blockIdx.x: candidate; blockIdx.y: instance
template <typename GL>
__global__ void __launch_bounds__(kPlanarTailThreads) isb_planar_tail_kernel(const __grid_constant__ PlanarTail T,
                                                                             float var_inv_i,
                                                                             const float* __restrict__ table)
{
    __shared__ __align__(16) float lut[kRangeLutStride];
    __shared__ uint32_t guides[kPlanarTailCells];
    __shared__ float costs[kPlanarTailCells];
    load_range_lut(lut, table, var_inv_i);
    __syncthreads();
    const int64_t inst = blockIdx.y;
    const int cand = blockIdx.x;
    int begin[2] = {0, 0};  // of the finer and the coarser level of a step
    for (int s = T.first; s < T.levels; ++s) {
        const int n = T.rows[s] * T.cols[s];
        const int rows_in = T.rows[s - 1], cols_in = T.cols[s - 1], nin = rows_in * cols_in;
        for (int i = threadIdx.x; i < n; i += kPlanarTailThreads) {
            const int y = i / T.cols[s], x = i - y * T.cols[s];
            uint32_t g;
            float c;
            if (s == T.first)
                tail_down<GL>(T.guides[s - 1] + inst * nin * GL::bytes, T.costs[s - 1] + (inst * T.ncand + cand) * nin,
                              rows_in, cols_in, x, y, lut, g, c);
            else
                tail_down<G4>(reinterpret_cast<const uint8_t*>(guides + begin[0]), costs + begin[0], rows_in, cols_in, x, y,
                              lut, g, c);
            guides[begin[1] + i] = g;
            costs[begin[1] + i] = c;
        }
        begin[0] = begin[1];
        begin[1] += n;
        __syncthreads();
    }
    const bool writes_guides = cand == 0;
    if (writes_guides && T.filtered[T.first] != T.guides[T.first]) {
        tail_store_guides<GL>(T, T.guides, inst, guides);
        __syncthreads();
    }
    const LutRange range{lut};
    for (int s = T.levels - 2; s >= T.first; --s) {
        const LevelGeom g{T.rows[s + 1], T.cols[s + 1], T.rows[s], T.cols[s]};
        const int coarse = begin[0], fine = coarse - g.rows_out * g.cols_out, n = g.rows_in * g.cols_in;
        // a warp takes one of the four fine pixels of 32 coarse ones
        for (int k = threadIdx.x; k < 4 * ((n + 31) & ~31); k += kPlanarTailThreads) {
            const int i = (k >> 7) * 32 + (k & 31);
            if (i >= n) continue;
            const int y = i / g.cols_in, x = i - y * g.cols_in;
            const uint32_t* gi = guides + coarse;
            const float* ci = costs + coarse;
            switch ((k >> 5) & 3) {
            case 0: tail_up<0>(gi, ci, guides + fine, costs + fine, g, x, y, T.weight_up[s], T.weight_down[s], range); break;
            case 1: tail_up<1>(gi, ci, guides + fine, costs + fine, g, x, y, T.weight_up[s], T.weight_down[s], range); break;
            case 2: tail_up<2>(gi, ci, guides + fine, costs + fine, g, x, y, T.weight_up[s], T.weight_down[s], range); break;
            default: tail_up<3>(gi, ci, guides + fine, costs + fine, g, x, y, T.weight_up[s], T.weight_down[s], range);
            }
        }
        begin[0] = fine;
        __syncthreads();
    }
    int at = 0;
    for (int s = T.first; s < T.levels; ++s) {
        const int n = T.rows[s] * T.cols[s];
        float* out = T.costs[s] + (inst * T.ncand + cand) * n;
        for (int i = threadIdx.x; i < n; i += kPlanarTailThreads) out[i] = costs[at + i];
        at += n;
    }
    if (writes_guides) tail_store_guides<GL>(T, T.filtered, inst, guides);
}

// The first level of a pyramid's tail: the first level s >= 1 of at most kPlanarTailPixels pixels that
// with the levels below it fits the block; `levels` when no level does, or for one candidate.
static int planar_tail_first(const int* rows, const int* cols, int levels, int ncand)
{
    if (ncand < 2) return levels;
    int cells = 0, first = levels;
    for (int s = levels - 1; s >= 1; --s) {
        const int64_t n = (int64_t)rows[s] * cols[s];
        if (n > kPlanarTailPixels || cells + n > kPlanarTailCells) break;
        cells += (int)n;
        first = s;
    }
    return first;
}

// Into how many ranges a step's candidates are shared out: a power of two of at most `ncand`.  Every
// range more repeats the set-up of the pixel's weights, which costs about as much as 10
// candidates, and a level too small to fill the GPU needs the ranges to keep enough loads in
// flight.  Measured at 32 candidates alone (fewer than the ranges only cap them), in microseconds for 1, 2, 4
// and 8 ranges: the down step to
// 262144 pixels 54, 49, 48, 52, to 65536 27, 18, 16, 16, to 16384 24, 14, 9, 7; the up step from
// 262144 pixels (selecting) 116, 128, 152, 192, from 65536 25, 31, 35, 42, from 16384 23, 15, 12, 15,
// from 4096 22, 14, 10, 8.
static int fit_ranges(int ranges, int ncand)
{
    while (ranges > ncand) ranges /= 2;
    return ranges;
}
static int down_ranges(int64_t pixels, int ncand) { return fit_ranges(pixels >= 32768 ? 4 : 8, ncand); }
static int up_ranges(int64_t pixels, int ncand)
{
    return fit_ranges(pixels >= 49152 ? 1 : pixels >= 24576 ? 2 : pixels >= 8192 ? 4 : 8, ncand);
}

template <typename GL>
static int launch_down_planar(const uint8_t* gi, const float* ci, int ri, int cl_i, uint8_t* go, float* co, int ro,
                              int cl_o, int ncand, int instances, float var_inv_i, cudaStream_t st)
{
    const LevelGeom g{ri, cl_i, ro, cl_o};
    const float* table = range_table(var_inv_i, st);
    const int64_t pout = (int64_t)ro * cl_o;
    const int ranges = down_ranges(pout * instances, ncand);
    const dim3 grid(grid_1d(pout, kPlanarBlock / ranges), instances);
    const bool pairs = cl_i % 2 == 0 && ((uintptr_t)ci & 7) == 0;
#define SSG_DOWN_PLANAR(R, P) \
    isb_down_planar_kernel<R, P, GL><<<grid, kPlanarBlock, 0, st>>>(gi, ci, go, co, g, ncand, var_inv_i, table)
#define SSG_DOWN_PLANAR2(R) \
    if (pairs) SSG_DOWN_PLANAR(R, true); \
    else SSG_DOWN_PLANAR(R, false);
    if (ranges == 8) { SSG_DOWN_PLANAR2(8) }
    else if (ranges == 4) { SSG_DOWN_PLANAR2(4) }
    else if (ranges == 2) { SSG_DOWN_PLANAR2(2) }
    else { SSG_DOWN_PLANAR2(1) }
#undef SSG_DOWN_PLANAR2
#undef SSG_DOWN_PLANAR
    return launch_status("isb_down_planar_kernel");
}

template <bool kSelect, typename GL>
static int launch_up_planar(const uint8_t* gi, const float* ci, int rc, int cc, const uint8_t* gf, uint8_t* go,
                            float* cf, int rf, int cf_cols, int ncand, int instances, float wu, float wd, float var_inv_i,
                            const SelectOut& so, cudaStream_t st)
{
    const LevelGeom g{rc, cc, rf, cf_cols};
    const float* table = range_table(var_inv_i, st);
    const int64_t pin = (int64_t)rc * cc;
    const bool pairs = cf_cols % 2 == 0 && ((uintptr_t)cf & 7) == 0;
    const int ranges = up_ranges(pin * instances, ncand);
    const dim3 grid(grid_1d(pin, 32), instances);
#define SSG_UP_PLANAR(R, P) \
    isb_up_planar_kernel<R, kSelect, P, GL><<<grid, 64 * R, 0, st>>>(gi, ci, gf, go, cf, g, ncand, wu, wd, var_inv_i, \
                                                                           table, so)
    if (ranges == 8) {
        if (pairs) SSG_UP_PLANAR(8, true);
        else SSG_UP_PLANAR(8, false);
    } else if (ranges == 4) {
        if (pairs) SSG_UP_PLANAR(4, true);
        else SSG_UP_PLANAR(4, false);
    } else if (ranges == 2) {
        if (pairs) SSG_UP_PLANAR(2, true);
        else SSG_UP_PLANAR(2, false);
    } else {
        if (pairs) SSG_UP_PLANAR(1, true);
        else SSG_UP_PLANAR(1, false);
    }
#undef SSG_UP_PLANAR
    return launch_status(kSelect ? "isb_up_planar_kernel<select>" : "isb_up_planar_kernel");
}

}  // namespace ssg
