// Backprojection of one-row detectors (1D parallel, fan line, fan arc) into 2D images.
//
// A filtered view is one row of sample pairs (row pairs, kernels.hpp): a sample is one 8-byte (FP16
// storage: 4-byte) load and one FMA, where a quad of a one-row view is 16 bytes (8) of which half hold
// zeros. The image is cut into cells of 32 x 32 pixels; 128 threads own a cell, eight pixels each
// along y, and keep the sums in registers over the views. The lanes of a warp cover 8 x 4 pixels per
// step, so that its gathers fall into one to three cache lines whatever the view's direction, and the
// eight pixels of a thread share the x part of the view's forms and run in packed FP32x2 pairs.
//
// Coordinates are evaluated in the same FP32 steps as in the quad kernels (backproject.cu), and FP16
// storage blends in half precision as they do: the rounding of a coordinate of 2000 samples is most of
// an image's error, and it stays what it was.
//
// Bound by instruction issue: 11 (parallel), 16 (FP16 line) and 23 (arc) instructions per update at 58 to 64 % of
// the issue slots (the arc's polynomial also fills the FMA pipe).
// Filter and backprojection, against the quad kernels over one-row views: parallel 1024 x 1024, 900 views
// of 1455: 1.81 -> 0.47 ms; arc 509 x 387, 1151 views of 671: 1.13 -> 0.28 ms; line 512 x 512, 720 views
// of 768, FP16: 0.208 -> 0.161 ms (0.104 with the quarter-turn form below).
// Cells per image are few (1024^2: 1024), so the views of a cell are cut into up to eight chunks, one
// per block of a thread-block cluster; the blocks sum their parts through distributed shared memory
// in chunk order and each writes its share of the cell, so there are no partial images and the
// result does not depend on timing.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/gct_fdk.h"
#include "common.cuh"
#include "geometry.hpp"
#include "kernels.hpp"

namespace gct {
namespace {

namespace cg = cooperative_groups;

constexpr int kCell = 32;              // cell side in pixels
constexpr int kThreads = 128;          // threads of a group, which owns a cell: four warps side by side along x
constexpr int kMaxGroups = 8;          // groups of a block: they share the block's views
constexpr int kPairs = 4;              // pixel pairs per thread: pixels 4 apart along y
constexpr int kStage = 32;             // views staged per barrier
constexpr float kShift = 12582912.0f;  // 1.5 * 2^23: a sum with it holds a whole number in its low bits
constexpr unsigned kShiftBits = 0x4B400000u;

// One view of a cell: a = first form (u, U or A) at pixel (0, 0), per i and j step, and the weight
// scale; b = second form (D or B) and -1 / dgamma; c0 = column of an arc's central ray.
struct CellView {
    float4 a, b;
    float c0;
    int cls;
};
// The cell projects off the row, well inside it, or neither; kNear: neither, and near an arc's axis, where the
// angle's polynomial holds (cells across the row's ends with atan2f: 257 x 257 pixels, 360 views 105 us a
// call, 68 this way)
constexpr int kOff = 0, kInside = 1, kMixed = 2, kNear = 3;

// Where the thread's pixels are evaluated: at themselves, or in quarter-turn plans under the turns
// that take the view to its base view. var: the index that varies over the thread's pixels (j; the
// base view's i after an odd number of turns), c: the other one. Parallel kind: var counts from the
// rows j0 and j0 + 16 of the cell (pairs 0, 1 and 2, 3).
struct Pixels {
    float2 var[kPairs];
    float c, k0;
};

__device__ __forceinline__ float2 two(float x) { return make_float2(x, x); }

// A form at the thread's pixel pair p, in the quad kernels' order: c0 + ci i, then + cj j.
template <bool ODD>
__device__ __forceinline__ float2 form(float4 f, const Pixels &px, int p)
{
    if (ODD) return __ffma2_rn(two(f.z), two(px.c), __ffma2_rn(two(f.y), px.var[p], two(f.x)));
    return __ffma2_rn(two(f.z), px.var[p], two(fmaf(f.y, px.c, f.x)));
}

// Two samples at byte offsets o0, o1. Line and arc kinds: (y, dy) at column fractions f in [0, 1];
// FP16 blends in half precision. Parallel kind (CENTRED): (mean, dy) at centred fractions, in FP32.
struct RowF32 {
    static constexpr unsigned kBytes = 8;
    template <bool CENTRED>
    static __device__ __forceinline__ float2 sample(const char *row, unsigned o0, unsigned o1, float2 f)
    {
        const float2 e0 = __ldg(reinterpret_cast<const float2 *>(row + o0));
        const float2 e1 = __ldg(reinterpret_cast<const float2 *>(row + o1));
        return make_float2(fmaf(f.x, e0.y, e0.x), fmaf(f.y, e1.y, e1.x));
    }
};
struct RowF16 {
    static constexpr unsigned kBytes = 4;
    template <bool CENTRED>
    static __device__ __forceinline__ float2 sample(const char *row, unsigned o0, unsigned o1, float2 f)
    {
        const __half2 h0 = __ldg(reinterpret_cast<const __half2 *>(row + o0));
        const __half2 h1 = __ldg(reinterpret_cast<const __half2 *>(row + o1));
        if (CENTRED) {
            const float2 e0 = __half22float2(h0), e1 = __half22float2(h1);
            return make_float2(fmaf(f.x, e0.y, e0.x), fmaf(f.y, e1.y, e1.x));
        }
        return __half22float2(__hfma2(__floats2half2_rn(f.x, f.y), __highs2half2(h0, h1), __lows2half2(h0, h1)));
    }
};

// One partner of an interleaved stack, for launches over some of the views only.
struct RowF16Partner : RowF16 {
    static constexpr unsigned kBytes = 16;
};

// Adds one view to the thread's pixels. INSIDE: the cell's samples lie well inside the row (and in
// front of an arc's source, near its axis); else pixels that project off the row add nothing.
template <int FAMILY, class R, bool ODD, bool INSIDE>
__device__ __forceinline__ void add_view(const CellView &v, const char *row, float umax, const Pixels &px,
                                         float2 (&acc)[kPairs])
{
    const float4 a = v.a, b = v.b;
    float v0[2] = {0.f, 0.f};
    if (FAMILY == 0) {  // rows j0 and j0 + 16, less the half of the centred split
        const float u = fmaf(a.y, px.c, a.x);
        v0[0] = fmaf(a.z, px.k0, u) - 0.5f;
        v0[1] = fmaf(a.z, px.k0 + 16.f, u) - 0.5f;
    }
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        float2 u, w = two(a.w), t;
        if (FAMILY == 0) {
            u = __ffma2_rn(two(a.z), px.var[p], two(v0[p / 2]));
            if (!INSIDE)  // where the row's zero border is
                u = make_float2(fminf(fmaxf(u.x, -1.5f), umax - 0.5f), fminf(fmaxf(u.y, -1.5f), umax - 0.5f));
            t = __fadd2_rn(u, two(kShift));
        } else {
            u = form<ODD>(a, px, p);
            const float2 d = form<ODD>(b, px, p);
            if (FAMILY == 1) {
                const float2 inv = make_float2(rcp_approx(d.x), rcp_approx(d.y));
                u = __fmul2_rn(u, inv);
                w = __fmul2_rn(__fmul2_rn(w, inv), inv);
            } else {
                const float2 rho2 = __ffma2_rn(u, u, __fmul2_rn(d, d));
                w = __fmul2_rn(w, make_float2(rcp_approx(rho2.x), rcp_approx(rho2.y)));
                const float2 g = INSIDE || v.cls == kNear ? arc_angle_near_neg(u, d)
                                                          : make_float2(-atan2f(u.x, d.x), -atan2f(u.y, d.y));
                u = __ffma2_rn(g, two(b.w), two(v.c0));
            }
        }
        bool on0 = true, on1 = true;
        if (FAMILY != 0) {
            if (!INSIDE) {
                on0 = u.x >= -1.0f && u.x <= umax;
                on1 = u.y >= -1.0f && u.y <= umax;
                u = make_float2(on0 ? u.x : -1.0f, on1 ? u.y : -1.0f);
            }
            t = __fadd2_rd(u, two(kShift));  // floor
        }
        const float2 f = __ffma2_rn(__fadd2_rn(t, two(-kShift)), two(-1.f), u);
        constexpr unsigned kBase = (static_cast<unsigned>(kQuadPad) - kShiftBits) * R::kBytes;  // modulo 2^32
        const float2 val = R::template sample<FAMILY == 0>(row, __float_as_uint(t.x) * R::kBytes + kBase,
                                                           __float_as_uint(t.y) * R::kBytes + kBase, f);
        const float2 r = __ffma2_rn(w, val, acc[p]);
        if (on0) acc[p].x = r.x;
        if (on1) acc[p].y = r.y;
    }
}

// add_view for an arc's kNear and kMixed views as a call: in line they take registers and instruction
// cache from the kInside views, most of them (509 x 387 pixels, 1151 views: 267 us with atan2f for both, 275
// with the kNear form, both in line, 263 this way).
struct Sums {
    float2 s[kPairs];
};
template <class R, bool ODD>
__device__ __noinline__ Sums add_edge_view(CellView v, const char *row, float umax, Pixels px, Sums sums)
{
    add_view<2, R, ODD, false>(v, row, umax, px, sums.s);
    return sums;
}

// Index box of a cell's pixels in the image.
struct Box {
    float i0, i1, j0, j1;
};

// Stages view v (base view b, its pixels in box) for the cell and classifies it: the coordinate is
// linear, or linear-fractional with a positive denominator (arc: its tangent), so that its extremes
// are at the corners; 1/64 of a sample covers the rounding.
template <int FAMILY>
__device__ void stage_view(const BpArgs &a, int v, int b, const Box &box, CellView &out)
{
    const float *c = a.coefs + static_cast<long long>(b) * kCoefPerView;
    constexpr int kD = FAMILY == 1 ? 8 : 4, kW = FAMILY == 0 ? 5 : FAMILY == 1 ? 12 : 16;
    float w = __ldg(a.coefs + static_cast<long long>(v) * kCoefPerView + kW);
    if (a.vinv) w *= __ldg(a.vinv + v);
    out.a = make_float4(__ldg(c), __ldg(c + 1), __ldg(c + 2), w);
    out.b = FAMILY == 0 ? make_float4(0.f, 0.f, 0.f, 0.f)
                        : make_float4(__ldg(c + kD), __ldg(c + kD + 1), __ldg(c + kD + 2), FAMILY == 2 ? -__ldg(c + 12) : 0.f);
    out.c0 = FAMILY == 2 ? __ldg(c + 13) : 0.f;
    float lo = 3.0e38f, hi = -3.0e38f;
    bool plain = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float i = (k & 1) ? box.i1 : box.i0, j = (k & 2) ? box.j1 : box.j0;
        float u = fmaf(out.a.z, j, fmaf(out.a.y, i, out.a.x));
        if (FAMILY != 0) {
            const float d = fmaf(out.b.z, j, fmaf(out.b.y, i, out.b.x));
            if (!(d > 0.f) || (FAMILY == 2 && !(fabsf(u) <= kArcNear * d))) plain = false;
            u = FAMILY == 1 ? u / d : fmaf(-atan2f(u, d), out.b.w, out.c0);
        }
        lo = fminf(lo, u);
        hi = fmaxf(hi, u);
    }
    const float m = 1.0f / 64.0f;
    out.cls = !plain                                   ? kMixed
              : hi < -1.0f - m || lo > a.umax + m      ? kOff
              : lo >= -1.0f + m && hi <= a.umax - m    ? kInside
              : FAMILY == 2                            ? kNear
                                                       : kMixed;
}

// The 128 threads of a group wait for each other. GROUPS: the block has several (barrier 0 is the block's).
template <bool GROUPS>
__device__ __forceinline__ void group_sync(int group)
{
    if (GROUPS) asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kThreads) : "memory");
    else __syncthreads();
}

// Sums of views [a.v_begin, a.v_begin + a.v_count) over the cell at pixel (i0, j0) by one group of 128
// threads (tid counts within it; all of them call it). SYM: quarter-turn plans, whose views take their
// coordinates from the base view at the turned pixel.
template <int FAMILY, class R, bool SYM, bool GROUPS>
__device__ __forceinline__ void cell_sums(const BpArgs &a, int i0, int j0, int tid, int group, CellView *s_view,
                                          float2 (&acc)[kPairs])
{
    const int lane = tid & 31;
    // pixels past the image's last ones repeat them (samples have to lie where the cell's class says)
    // and are not stored
    const float i1 = static_cast<float>(max(min(i0 + kCell, a.nx) - 1, i0));
    const float j1 = static_cast<float>(max(min(j0 + kCell, a.ny) - 1, j0));
    const float fi = fminf(static_cast<float>(i0 + (tid >> 5) * 8 + (lane & 7)), i1);
    const float fj = static_cast<float>(j0 + (lane >> 3));
    Pixels px;
    px.c = fi;
    px.k0 = static_cast<float>(j0);
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        acc[p] = make_float2(0.f, 0.f);
        px.var[p] = make_float2(fminf(fj + 8.f * p, j1), fminf(fj + 8.f * p + 4.f, j1));
        if (FAMILY == 0) {
            const float k = px.k0 + 16.f * (p / 2);
            px.var[p] = make_float2(px.var[p].x - k, px.var[p].y - k);
        }
    }
    const int row_bytes = (static_cast<int>(a.qview)) * static_cast<int>(R::kBytes);
    int v = a.v_begin;
    const int end = a.v_begin + a.v_count;
    while (v < end) {
        // views [v, stop) of one quarter: q turns from their base views
        const int q = SYM ? v / a.quarter : 0, stop = SYM ? min(end, (q + 1) * a.quarter) : end;
        Box box{static_cast<float>(i0), i1, static_cast<float>(j0), j1};
        if (SYM) {
            // R^-q of (i, j): (n-1-i, n-1-j) after two turns, (j, n-1-i) or (n-1-j, i) after one or three
            const float n1 = static_cast<float>(a.nx - 1);
            const bool flip_j = q == 2 || q == (a.sym > 0 ? 3 : 1), flip_i = q == 2 || q == (a.sym > 0 ? 1 : 3);
            px.c = flip_i ? n1 - fi : fi;
#pragma unroll
            for (int p = 0; p < kPairs; ++p) {
                const float y0 = fminf(fj + 8.f * p, j1), y1 = fminf(fj + 8.f * p + 4.f, j1);
                px.var[p] = flip_j ? make_float2(n1 - y0, n1 - y1) : make_float2(y0, y1);
            }
            if (flip_i) box.i0 = n1 - i1, box.i1 = n1 - static_cast<float>(i0);
            if (flip_j) box.j0 = n1 - j1, box.j1 = n1 - static_cast<float>(j0);
            if (q & 1) box = Box{box.j0, box.j1, box.i0, box.i1};
        }
        for (; v < stop; v += kStage) {
            const int nvc = min(kStage, stop - v);
            group_sync<GROUPS>(group);
            if (tid < nvc) stage_view<FAMILY>(a, v + tid, v + tid - q * (SYM ? a.quarter : 0), box, s_view[tid]);
            group_sync<GROUPS>(group);
            const char *row = static_cast<const char *>(a.quads);
            if (R::kBytes == RowF16Partner::kBytes) row += static_cast<long long>(v - q * a.quarter) * row_bytes + 4 * q;
            else row += static_cast<long long>(v) * row_bytes;
            for (int k = 0; k < nvc; ++k, row += row_bytes) {
                const int cls = s_view[k].cls;
                if (cls == kOff) continue;  // every pixel of the cell would add zero
                auto add = [&](auto odd) {
                    constexpr bool ODD = decltype(odd)::value;
                    if (cls == kInside) {
                        add_view<FAMILY, R, ODD, true>(s_view[k], row, a.umax, px, acc);
                    } else if constexpr (FAMILY == 2) {
                        Sums t;
#pragma unroll
                        for (int p = 0; p < kPairs; ++p) t.s[p] = acc[p];
                        t = add_edge_view<R, ODD>(s_view[k], row, a.umax, px, t);
#pragma unroll
                        for (int p = 0; p < kPairs; ++p) acc[p] = t.s[p];
                    } else {
                        add_view<FAMILY, R, ODD, false>(s_view[k], row, a.umax, px, acc);
                    }
                };
                if (SYM && (q & 1)) add(std::true_type());
                else add(std::false_type());
            }
        }
        v = stop;
    }
}

// Shared memory of a group: its sums and its staged views.
constexpr unsigned kRowsSmem = kCell * kCell * sizeof(float) + kStage * sizeof(CellView);

// The block's sums [group][n] into [0], over the groups in order.
__device__ __forceinline__ void sum_groups(float *s_sum, int n, int groups)
{
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        float s = s_sum[e];
        for (int g = 1; g < groups; ++g) s += s_sum[g * n + e];
        s_sum[e] = s;
    }
}

// A cluster of gridDim.z blocks per cell, each with its chunk of the views; the groups of 128 threads of
// a block share its chunk out among themselves.
template <int FAMILY, class R, bool SYM, bool GROUPS>
__global__ void __launch_bounds__(GROUPS ? kThreads * kMaxGroups : kThreads, GROUPS ? 1 : 8)
    rows_kernel(BpArgs a, int chunk, int sub)
{
    extern __shared__ float4 s_mem[];  // GROUPS: kRowsSmem a group
    __shared__ CellView s_view1[GROUPS ? 1 : kStage];
    __shared__ float s_sum1[GROUPS ? 1 : kCell * kCell];
    const int i0 = blockIdx.x * kCell, j0 = blockIdx.y * kCell, tid = GROUPS ? threadIdx.x % kThreads : threadIdx.x;
    const int group = GROUPS ? threadIdx.x / kThreads : 0, groups = GROUPS ? blockDim.x / kThreads : 1;
    float *const s_sum = GROUPS ? reinterpret_cast<float *>(s_mem) : s_sum1;  // [group][pixel][thread]
    CellView *const s_view =
        GROUPS ? reinterpret_cast<CellView *>(s_sum + groups * kCell * kCell) + group * kStage : s_view1;
    const int z = blockIdx.z, chunks = gridDim.z;
    BpArgs la = a;
    const int first = z * chunk + group * sub, end = min((z + 1) * chunk, a.v_count);
    la.v_begin = a.v_begin + first;
    la.v_count = max(0, min(sub, end - first));
    float2 acc[kPairs];
    cell_sums<FAMILY, R, SYM, GROUPS>(la, i0, j0, tid, group, s_view, acc);
    const int i = i0 + (tid >> 5) * 8 + (tid & 7), j = j0 + ((tid >> 3) & 3);
    auto put = [&](int p, float s) {
        const int y = j + 4 * p;
        if (i >= a.nx || y >= a.ny) return;
        float *dst = a.vol + static_cast<long long>(y) * a.nx + i;
        *dst = a.accumulate ? *dst + s : s;
    };
    if (chunks * groups == 1) {
#pragma unroll
        for (int p = 0; p < 2 * kPairs; ++p) put(p, (p & 1) ? acc[p / 2].y : acc[p / 2].x);
        return;
    }
#pragma unroll
    for (int p = 0; p < 2 * kPairs; ++p)
        s_sum[group * kCell * kCell + p * kThreads + tid] = (p & 1) ? acc[p / 2].y : acc[p / 2].x;
    if (GROUPS) sum_groups(s_sum, kCell * kCell, groups);
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    // the block's share of the pixels (the chunks are 1, 2, 4 or 8), over the chunks in order
    for (int p = z + chunks * group; p < 2 * kPairs; p += chunks * groups) {
        float s = 0.f;
        for (int c = 0; c < chunks; ++c) s += cl.map_shared_rank(s_sum, c)[p * kThreads + tid];
        put(p, s);
    }
    cl.sync();  // the sums stay until every block has read them
}

// Work-queue form: the two groups of a block share the views of one cell. (One cell per group made a tile of
// 64 x 32 pixels: a round with a single request, which the server must not split over the views in another
// way than a full one, kept too few blocks busy. Line 512 x 512, 720 views, FP16, a request by itself: 0.90 ms, 0.62
// with a cell per block; 48 at a time the same.)
template <int FAMILY, class R, bool SYM>
__device__ __noinline__ void queue_cell(BpArgs &a, int tx, int ty, int tid, int mode, CellView *s_view, float *s_sum)
{
    const int i0 = tx * kCell, j0 = ty * kCell, group = tid / kThreads, ct = tid % kThreads;
    float2 acc[kPairs];
    cell_sums<FAMILY, R, SYM, true>(a, i0, j0, ct, group, s_view + group * kStage, acc);
    // each group stores half of the pixels: its own sums of the others go through shared memory
    const auto mine = [&](int p) { return (p & 1) ? acc[p / 2].y : acc[p / 2].x; };
#pragma unroll
    for (int p = 0; p < kPairs; ++p) s_sum[(group * kPairs + p) * kThreads + ct] = group ? mine(p) : mine(p + kPairs);
    __syncthreads();
    const int i = i0 + (ct >> 5) * 8 + (ct & 7), j = j0 + ((ct >> 3) & 3);
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const float other = s_sum[((1 - group) * kPairs + p) * kThreads + ct];
        const float s = group ? other + mine(p + kPairs) : mine(p) + other;
        const int y = j + 4 * (group * kPairs + p);
        if (i >= a.nx || y >= a.ny) continue;
        float *dst = a.vol + static_cast<long long>(y) * a.nx + i;
        if (mode == kBpAtomic) atomicAdd(dst, s);
        else *dst = mode == kBpAccumulate ? *dst + s : s;
    }
}

template <class R>
__global__ void __launch_bounds__(kQueueThreads, 4)
    rows_queue_kernel(const BpItem *__restrict__ items, const BpWork *__restrict__ work, int n_work, int *counter)
{
    static_assert(kQueueThreads == 2 * kThreads && kRowsTileX == kCell && kRowsTileY == kCell, "a cell of two groups");
    __shared__ CellView s_view[2 * kStage];
    __shared__ float s_sum[2 * kPairs * kThreads];
    __shared__ BpItem s_item;
    __shared__ BpWork s_work;
    __shared__ int s_next;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_next = atomicAdd(counter, 1);
        __syncthreads();
        const int w = s_next;
        if (w >= n_work) return;
        if (tid == 0) {
            s_work = work[w];
            s_item = items[s_work.item];
        }
        __syncthreads();
        BpArgs a = s_item.a;
        const int count = tid < kThreads ? (s_work.v_count + 1) / 2 : s_work.v_count / 2;  // the first group takes the odd one
        a.v_begin = s_work.v_begin + (tid < kThreads ? 0 : s_work.v_count - count);
        a.v_count = count;
        const int mode = s_work.mode, tx = s_work.tile % s_item.tiles_x, ty = s_work.tile / s_item.tiles_x;
        if (s_item.family == 0) {
            queue_cell<0, R, false>(a, tx, ty, tid, mode, s_view, s_sum);
        } else if (s_item.family == 1) {
            if (a.sym) queue_cell<1, R, true>(a, tx, ty, tid, mode, s_view, s_sum);
            else queue_cell<1, R, false>(a, tx, ty, tid, mode, s_view, s_sum);
        } else if constexpr (R::kBytes == RowF32::kBytes) {  // FP16 arcs keep their quads
            if (a.sym) queue_cell<2, R, true>(a, tx, ty, tid, mode, s_view, s_sum);
            else queue_cell<2, R, false>(a, tx, ty, tid, mode, s_view, s_sum);
        }
        __syncthreads();  // s_item / s_work / s_next are rewritten for the next entry
    }
}

// ---- quarter-turn plans, FP16 lines -------------------------------------------------------------
//
// The rows of the four partner views are interleaved entry by entry (16 bytes). A thread owns the four
// columns R^k(c) of four first-quadrant pixels c and, per base view, evaluates the coordinates at each
// R^k(c) once for the four partners (partner q adds to column R^(k+q)(c)): one 16-byte load and one
// evaluation per four updates. Cells are 32 x 16 pixels of the quadrant.
// Bound by issue at 14 warps per SM (1024 blocks). 512 x 512 pixels, 720 views of 768: 142 us one view at a
// time, 92 us this way (2.05 T updates/s); the call 0.161 -> 0.114 ms (0.104 with the filter's own scales).
constexpr int kSymCellY = 16, kSymPairs = 2, kSymGroups = 4;
constexpr int kSymSums = 4 * 2 * kSymPairs * kThreads;  // a group's sums
constexpr unsigned kSymSmem = kSymSums * sizeof(float) + kStage * (sizeof(float4) + sizeof(int4) + sizeof(CellView));

// Indices of R^K of pixels (i, j): var along the thread's pixels, c the other one (Pixels).
template <int K>
__device__ __forceinline__ void turn_pixels(int sym, float n1, float i, const float2 (&j)[kSymPairs], Pixels &px)
{
    const bool flip_j = K == 2 || K == (sym > 0 ? 1 : 3), flip_i = K == 2 || K == (sym > 0 ? 3 : 1);
    px.c = flip_i ? n1 - i : i;
#pragma unroll
    for (int p = 0; p < kSymPairs; ++p) px.var[p] = flip_j ? make_float2(n1 - j[p].x, n1 - j[p].y) : j[p];
}

// Adds base view v's evaluation at R^K of the thread's pixels, for its four partners (weights w).
template <int K, bool INSIDE>
__device__ __forceinline__ void add_partners(const CellView &v, float4 w, const char *row, float umax,
                                             const Pixels &px, float2 (&acc)[4][kSymPairs])
{
#pragma unroll
    for (int p = 0; p < kSymPairs; ++p) {
        const float2 d = form<(K & 1) != 0>(v.b, px, p);
        const float2 inv = make_float2(rcp_approx(d.x), rcp_approx(d.y));
        float2 u = __fmul2_rn(form<(K & 1) != 0>(v.a, px, p), inv);
        const float2 i2 = __fmul2_rn(inv, inv);
        bool on0 = true, on1 = true;
        if (!INSIDE) {
            on0 = u.x >= -1.0f && u.x <= umax;
            on1 = u.y >= -1.0f && u.y <= umax;
            u = make_float2(on0 ? u.x : -1.0f, on1 ? u.y : -1.0f);
        }
        const float2 t = __fadd2_rd(u, two(kShift));
        const float2 f = __ffma2_rn(__fadd2_rn(t, two(-kShift)), two(-1.f), u);
        constexpr unsigned kBase = (static_cast<unsigned>(kQuadPad) - kShiftBits) * 16u;  // modulo 2^32
        const uint4 e0 = __ldg(reinterpret_cast<const uint4 *>(row + (__float_as_uint(t.x) * 16u + kBase)));
        const uint4 e1 = __ldg(reinterpret_cast<const uint4 *>(row + (__float_as_uint(t.y) * 16u + kBase)));
        const __half2 fh = __floats2half2_rn(f.x, f.y);
        auto blend = [&](unsigned h0, unsigned h1, float wq, float2 &sum) {
            const __half2 a0 = *reinterpret_cast<const __half2 *>(&h0), a1 = *reinterpret_cast<const __half2 *>(&h1);
            const float2 val = __half22float2(__hfma2(fh, __highs2half2(a0, a1), __lows2half2(a0, a1)));
            const float2 r = __ffma2_rn(__fmul2_rn(two(wq), i2), val, sum);
            if (on0) sum.x = r.x;
            if (on1) sum.y = r.y;
        };
        blend(e0.x, e1.x, w.x, acc[K][p]);
        blend(e0.y, e1.y, w.y, acc[(K + 1) & 3][p]);
        blend(e0.z, e1.z, w.z, acc[(K + 2) & 3][p]);
        blend(e0.w, e1.w, w.w, acc[(K + 3) & 3][p]);
    }
}

// A cluster of gridDim.z blocks per cell, each with its chunk of the base views [a.v_begin, + a.v_count),
// which the groups of a block share out among themselves.
template <bool GROUPS>
__global__ void __launch_bounds__(GROUPS ? kThreads * kSymGroups : kThreads, GROUPS ? 1 : 6)
    rows_sym_kernel(BpArgs a, int chunk, int sub)
{
    extern __shared__ float4 s_mem[];  // GROUPS: kSymSmem a group
    __shared__ float4 s_mem1[GROUPS ? 1 : kSymSmem / sizeof(float4)];
    const int tid = GROUPS ? threadIdx.x % kThreads : threadIdx.x;
    const int group = GROUPS ? threadIdx.x / kThreads : 0, groups = GROUPS ? blockDim.x / kThreads : 1;
    float *const s_sum = reinterpret_cast<float *>(GROUPS ? s_mem : s_mem1);  // [group][turn][pixel][thread]
    float4 *const s_w = reinterpret_cast<float4 *>(s_sum + groups * kSymSums) + group * kStage;  // weights of the partners
    int4 *const s_cls = reinterpret_cast<int4 *>(s_w + (groups - group) * kStage) + group * kStage;  // classes of the cell's turns
    CellView *const s_view = reinterpret_cast<CellView *>(s_cls + (groups - group) * kStage) + group * kStage;
    const int i0 = blockIdx.x * kCell, j0 = blockIdx.y * kSymCellY, h = a.nx / 2;
    const int z = blockIdx.z, chunks = gridDim.z;
    const int v_begin = a.v_begin + z * chunk + group * sub;
    const int v_end = min(min(v_begin + sub, a.v_begin + (z + 1) * chunk), a.v_begin + a.v_count);
    const float n1 = static_cast<float>(a.nx - 1);
    const float i1 = static_cast<float>(min(i0 + kCell, h) - 1), j1 = static_cast<float>(min(j0 + kSymCellY, h) - 1);
    const int lane = tid & 31;
    // pixels past the quadrant repeat its last ones and are not stored
    const float fi = fminf(static_cast<float>(i0 + (tid >> 5) * 8 + (lane & 7)), i1);
    const float fy = static_cast<float>(j0 + (lane >> 3));
    float2 fj[kSymPairs], acc[4][kSymPairs];
#pragma unroll
    for (int p = 0; p < kSymPairs; ++p) {
        fj[p] = make_float2(fminf(fy + 8.f * p, j1), fminf(fy + 8.f * p + 4.f, j1));
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k][p] = make_float2(0.f, 0.f);
    }
    for (int vc = v_begin; vc < v_end; vc += kStage) {
        const int nvc = min(kStage, v_end - vc);
        group_sync<GROUPS>(group);
        if (tid / 4 < nvc) {
            const int sv = tid / 4, k = tid & 3, v = vc + sv;
            // the cell's box under k turns
            const bool flip_j = k == 2 || k == (a.sym > 0 ? 1 : 3), flip_i = k == 2 || k == (a.sym > 0 ? 3 : 1);
            Box box{static_cast<float>(i0), i1, static_cast<float>(j0), j1};
            if (flip_i) box.i0 = n1 - i1, box.i1 = n1 - static_cast<float>(i0);
            if (flip_j) box.j0 = n1 - j1, box.j1 = n1 - static_cast<float>(j0);
            if (k & 1) box = Box{box.j0, box.j1, box.i0, box.i1};
            CellView mine;
            stage_view<1>(a, v + k * a.quarter, v, box, mine);
            reinterpret_cast<int *>(&s_cls[sv])[k] = mine.cls;
            reinterpret_cast<float *>(&s_w[sv])[k] = mine.a.w;
            if (k == 0) s_view[sv] = mine;
        }
        group_sync<GROUPS>(group);
        const long long base_bytes = a.qview * 16;
        const char *row = static_cast<const char *>(a.quads) + vc * base_bytes;
        for (int k = 0; k < nvc; ++k, row += base_bytes) {
            const CellView &v = s_view[k];
            const float4 w = s_w[k];
            const int4 cls = s_cls[k];
            Pixels px;
            auto add = [&](auto turn, int c) {
                constexpr int K = decltype(turn)::value;
                if (c == kOff) return;  // every pixel of the image would add zero
                turn_pixels<K>(a.sym, n1, fi, fj, px);
                if (c == kInside) add_partners<K, true>(v, w, row, a.umax, px, acc);
                else add_partners<K, false>(v, w, row, a.umax, px, acc);
            };
            add(std::integral_constant<int, 0>(), cls.x);
            add(std::integral_constant<int, 1>(), cls.y);
            add(std::integral_constant<int, 2>(), cls.z);
            add(std::integral_constant<int, 3>(), cls.w);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int p = 0; p < 2 * kSymPairs; ++p)
            s_sum[((group * 4 + k) * 2 * kSymPairs + p) * kThreads + tid] = (p & 1) ? acc[k][p / 2].y : acc[k][p / 2].x;
    if (GROUPS) sum_groups(s_sum, kSymSums, groups);
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    // the block's share of the pixels, over the chunks in order
    for (int e = z + chunks * group; e < 8 * kSymPairs; e += chunks * groups) {
        const int k = e / (2 * kSymPairs), p = e % (2 * kSymPairs);
        float s = 0.f;
        for (int c = 0; c < chunks; ++c) s += cl.map_shared_rank(s_sum, c)[e * kThreads + tid];
        int x = i0 + (tid >> 5) * 8 + (tid & 7), y = j0 + ((tid >> 3) & 3) + 4 * p;
        if (x >= h || y >= h) continue;
        for (int r = 0; r < k; ++r) {  // the plan's quarter turn
            const int tx = a.sym > 0 ? a.nx - 1 - y : y, ty = a.sym > 0 ? x : a.nx - 1 - x;
            x = tx;
            y = ty;
        }
        float *dst = a.vol + static_cast<long long>(y) * a.nx + x;
        *dst = a.accumulate ? *dst + s : s;
    }
    cl.sync();  // the sums stay until every block has read them
}

// Filtered rows Y (row stride nc, views v0 on) -> row pairs.
template <bool F16>
__global__ void row_pairs_kernel(const float *__restrict__ Y, int v0, int nv, int nc, bool centred,
                                 const float *__restrict__ vscale, void *out)
{
    const int pitch = nc + 2 * kQuadPad;
    const long long n = static_cast<long long>(nv) * pitch;
    for (long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
         e += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int v = static_cast<int>(e / pitch), c = static_cast<int>(e - static_cast<long long>(v) * pitch) - kQuadPad;
        const float *y = Y + static_cast<long long>(v) * nc;
        const float sc = F16 ? __ldg(vscale + v0 + v) : 1.f;
        const float y0 = c >= 0 && c < nc ? sc * __ldg(y + c) : 0.f;
        const float y1 = c + 1 >= 0 && c + 1 < nc ? sc * __ldg(y + c + 1) : 0.f;
        store_row_pair<F16>(out, static_cast<long long>(v0) * pitch + e, y0, y1, centred);
    }
}

// Launches kern over clusters of view chunks per cell; per_sm: its blocks that fit an SM. grouped: its form for
// blocks of up to max_groups groups, with group_smem bytes of shared memory each.
template <class Kern>
void launch_cells(Kern kern, Kern grouped, const BpArgs &a, dim3 cells, int max_groups, int per_sm,
                  unsigned group_smem, int num_sms, cudaStream_t s)
{
    // chunks of at least 8 views until the grid holds six waves of eight blocks per SM: the last wave of
    // a launch of one to two waves runs nearly empty, and chunk counts that just fill whole waves measured
    // slower than finer ones (512 x 512 pixels one view at a time: 4 chunks 173 us, 8 chunks 142 us)
    const long long n = static_cast<long long>(cells.x) * cells.y;
    int chunks = 1;
    while (chunks < 8 && n * chunks < 6LL * 8 * num_sms && a.v_count / (2 * chunks) >= 8) chunks *= 2;
    const int chunk = (a.v_count + chunks - 1) / chunks;
    // An image of few cells leaves most of the SMs' warps idle with eight chunks, and a view costs a group
    // its whole latency (0.6 us): then several groups share a chunk, as long as they fill at most half of the
    // blocks that fit (between that and all of them the rest of the block waits for its slowest group:
    // 257 x 254 pixels, 360 views, line 39.5 us as it is against 43.5 with two groups). Calls of 720
    // views, F32: line 64 x 64 68 -> 25 us, 128 x 128 63 -> 32; arc, with the polynomial in kNear cells,
    // 194 -> 36 and 189 -> 52 (the quad kernels' split launches took 35, 60, 40 and 77).
    int groups = 1;
    while (groups < max_groups && n * chunks * groups * 4 <= static_cast<long long>(per_sm) * num_sms &&
           chunk / (2 * groups) >= 4)
        groups *= 2;
    const int sub = (chunk + groups - 1) / groups;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cells.x, cells.y, chunks);
    cfg.blockDim = dim3(kThreads * groups);
    cfg.dynamicSmemBytes = groups > 1 ? groups * group_smem : 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = static_cast<unsigned>(chunks);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, groups > 1 ? grouped : kern, a, chunk, sub);
}

template <int FAMILY, class R, bool SYM>
void launch_rows_kernel(const BpArgs &a, int num_sms, cudaStream_t s)
{
    launch_cells(rows_kernel<FAMILY, R, SYM, false>, rows_kernel<FAMILY, R, SYM, true>, a,
                 dim3((a.nx + kCell - 1) / kCell, (a.ny + kCell - 1) / kCell), kMaxGroups, 8, kRowsSmem, num_sms, s);
}

template <class R>
void launch_rows(const BpArgs &a, int family, int num_sms, cudaStream_t s)
{
    if (family == 0) {
        launch_rows_kernel<0, R, false>(a, num_sms, s);
    } else if (family == 1) {
        if (a.sym) launch_rows_kernel<1, R, true>(a, num_sms, s);
        else launch_rows_kernel<1, R, false>(a, num_sms, s);
    } else if constexpr (R::kBytes == RowF32::kBytes) {
        if (a.sym) launch_rows_kernel<2, R, true>(a, num_sms, s);
        else launch_rows_kernel<2, R, false>(a, num_sms, s);
    }
}

}  // namespace

void launch_backproject_rows(const BpArgs &a, int family, int storage, int num_sms, cudaStream_t s)
{
    if (a.partners) launch_rows_kernel<1, RowF16Partner, true>(a, num_sms, s);
    else if (storage == 0) launch_rows<RowF32>(a, family, num_sms, s);
    else launch_rows<RowF16>(a, family, num_sms, s);
}

void launch_backproject_rows_sym(const BpArgs &a, int num_sms, cudaStream_t s)
{
    const int h = a.nx / 2;
    launch_cells(rows_sym_kernel<false>, rows_sym_kernel<true>, a,
                 dim3((h + kCell - 1) / kCell, (h + kSymCellY - 1) / kSymCellY), kSymGroups, 6, kSymSmem, num_sms, s);
}

int rows_queue_blocks_per_sm(int storage)
{
    int n = 0;
    const cudaError_t e =
        storage == 0 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rows_queue_kernel<RowF32>, kQueueThreads, 0)
                     : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rows_queue_kernel<RowF16>, kQueueThreads, 0);
    return e == cudaSuccess ? n : 0;
}

void launch_rows_queue(const BpItem *items, const BpWork *work, int n_work, int *counter, int storage, int grid,
                       cudaStream_t s)
{
    if (storage == 0) rows_queue_kernel<RowF32><<<grid, kQueueThreads, 0, s>>>(items, work, n_work, counter);
    else rows_queue_kernel<RowF16><<<grid, kQueueThreads, 0, s>>>(items, work, n_work, counter);
}

void launch_row_pairs(const float *Y, int v0, int nv, int nc, bool centred, const float *vscale, void *out,
                      int num_sms, cudaStream_t s)
{
    long long grid = (static_cast<long long>(nv) * (nc + 2 * kQuadPad) + 255) / 256;
    if (grid > static_cast<long long>(num_sms) * 32) grid = static_cast<long long>(num_sms) * 32;
    const unsigned g = static_cast<unsigned>(grid < 1 ? 1 : grid);
    if (vscale) row_pairs_kernel<true><<<g, 256, 0, s>>>(Y, v0, nv, nc, centred, vscale, out);
    else row_pairs_kernel<false><<<g, 256, 0, s>>>(Y, v0, nv, nc, centred, vscale, out);
}

}  // namespace gct
