// Ray-driven projection kernels: exact line integrals of analytic ellipsoid phantoms (input
// generation) and a ray-marching forward projector through a voxel volume (consistency
// checks). Rays are built per detector pixel from the same per-view geometry the
// backprojector inverts, so a projection followed by backprojection uses one convention:
//   parallel kinds : origin s n + (0,0,z), direction (cos t, sin t, 0), n = (cos(t+pi/2), sin(t+pi/2), 0)
//   line / flat    : origin S, direction SDD e_w + u e_u + v e_v
//   arc / cylinder : origin S, direction cos(g) e_w + sin(g) e_u + (t / SDD) e_v
// with u = (c - c0) du, v = (r - r0) dv (src/cuda/geom/coord_trans_proj.cuh:142-150, the
// inverse of DCSToPCS).
#include <algorithm>
#include <climits>
#include <cmath>

#include "../../include/gct_fdk.h"
#include "project.hpp"

namespace gct {
namespace {

// Grids up to this size (64 KB) are read as they are: their calls take longer to allocate and fill
// the copies than the copies save (25 x 25 x 24 voxels, 36 views of 48 x 40: 0.69 ms a call against
// 0.75 with copies; 32 x 32 x 31, 90 views of 64 x 64: 0.75 against 0.84).
constexpr long long kCopyVoxels = 1 << 14;
// What copies cost a call and save it, in us. Up to 2 MB they come with the driver's smallest allocations and
// cost next to nothing (48^3 voxels, 4 views of 64 x 64 and more: 0 to 15 % less time with them); larger ones cost
// 0.5 ms and 18 us per million voxels, the exchanged grid alone 5 us. A million samples of rays along x, within
// the tenth of a voxel of y per step that keeps the warp from marching in step, take 15 to 24 us longer in the
// grid itself than in either copy (every gather touches 32 lines); others take 0.8 us longer than in the
// pairs. Without / exchanged grid / pairs, ms a call: 2 views of 64 x 64 through 512^3 1.4 / - / 4.9, of
// 256 x 256 5.0 / 3.3 / 5.2, of 512 x 512 10.4 / 3.4 / 5.8; 8 views of 96 x 96 through 96^3 1.0 / - / 1.4, 180 of
// 160 x 160 5.3 / - / 3.3; 192^3, 16 views of 256 x 256, half-voxel steps 2.7 / - / 2.3, whole ones 1.8 / - / 2.0.
constexpr long long kSmallCopies = 2 << 20;
constexpr double kCopyCall = 500.0, kPairsVoxel = 18e-6, kAlongVoxel = 5e-6;
constexpr double kSaveX = 21e-6, kPairsSave = 0.8e-6;

struct Ray {
    double o[3];
    double d[3];
};

__device__ Ray make_ray(const ProjView &pv, int kind, double du, double dv, int c, int r)
{
    Ray ray;
    const double u = (static_cast<double>(c) - pv.c0) * du;
    const double t = (static_cast<double>(r) - pv.r0) * dv;
    if (kind == GCT_GEOM_PARALLEL_1D || kind == GCT_GEOM_PARALLEL_2D || kind == GCT_GEOM_CONE_PARALLEL) {
        const double th = pv.extra;
        double sn, cs;
        sincos(th, &sn, &cs);
        // n = (cos(th + pi/2), sin(th + pi/2)) = (-sin th, cos th)
        double z = 0.0;
        if (kind == GCT_GEOM_PARALLEL_2D) z = -t;
        if (kind == GCT_GEOM_CONE_PARALLEL) z = -t * pv.zscale;
        ray.o[0] = -sn * u;
        ray.o[1] = cs * u;
        ray.o[2] = z;
        ray.d[0] = cs;
        ray.d[1] = sn;
        ray.d[2] = 0.0;
        return ray;
    }
    for (int i = 0; i < 3; ++i) ray.o[i] = pv.src[i];
    if (kind == GCT_GEOM_FAN_LINE || kind == GCT_GEOM_CONE_FLAT) {
        for (int i = 0; i < 3; ++i) ray.d[i] = pv.sdd * pv.ew[i] + u * pv.eu[i] + t * pv.ev[i];
    } else {
        double sg, cg;
        sincos(u, &sg, &cg);
        for (int i = 0; i < 3; ++i) ray.d[i] = cg * pv.ew[i] + sg * pv.eu[i] + (t / pv.sdd) * pv.ev[i];
    }
    return ray;
}

__global__ void phantom_kernel(const ProjView *__restrict__ views, int kind, int nv, int nr,
                               int nc, double du, double dv, const gct_ellipsoid *__restrict__ ell,
                               int ne, bool planar, float *__restrict__ out)
{
    const long long total = static_cast<long long>(nv) * nr * nc;
    for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
         idx += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int c = static_cast<int>(idx % nc);
        const long long vr = idx / nc;
        const int r = static_cast<int>(vr % nr);
        const int v = static_cast<int>(vr / nr);
        const Ray ray = make_ray(views[v], kind, du, dv, c, r);
        const double dn = sqrt(ray.d[0] * ray.d[0] + ray.d[1] * ray.d[1] + ray.d[2] * ray.d[2]);
        double sum = 0.0;
        for (int e = 0; e < ne; ++e) {
            const gct_ellipsoid E = ell[e];
            double sp, cp;
            sincos(E.phi, &sp, &cp);
            double p[3] = {ray.o[0] - E.center[0], ray.o[1] - E.center[1],
                           planar ? 0.0 : ray.o[2] - E.center[2]};
            double q[3] = {ray.d[0], ray.d[1], planar ? 0.0 : ray.d[2]};
            // rotate by -phi about z, then scale by the semi-axes
            const double px = (cp * p[0] + sp * p[1]) / E.semi_axes[0];
            const double py = (-sp * p[0] + cp * p[1]) / E.semi_axes[1];
            const double pz = p[2] / E.semi_axes[2];
            const double qx = (cp * q[0] + sp * q[1]) / E.semi_axes[0];
            const double qy = (-sp * q[0] + cp * q[1]) / E.semi_axes[1];
            const double qz = q[2] / E.semi_axes[2];
            const double A = qx * qx + qy * qy + qz * qz;
            const double B = px * qx + py * qy + pz * qz;
            const double C = px * px + py * py + pz * pz - 1.0;
            const double disc = B * B - A * C;
            if (disc > 0.0) sum += E.mu * 2.0 * sqrt(disc) / A * dn;
        }
        out[idx] = static_cast<float>(sum);
    }
}

// Trilinear sample with zero outside the grid; (x, y, z) in voxel-index units.
__device__ __forceinline__ float trilinear(const float *__restrict__ vol, int nx, int ny, int nz,
                                           float x, float y, float z)
{
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int ix = static_cast<int>(fx), iy = static_cast<int>(fy), iz = static_cast<int>(fz);
    const float ax = x - fx, ay = y - fy, az = z - fz;
    float acc = 0.f;
#pragma unroll
    for (int dz = 0; dz < 2; ++dz) {
        const int zz = iz + dz;
        if (zz < 0 || zz >= nz) continue;
        const float wz = dz ? az : 1.f - az;
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const int yy = iy + dy;
            if (yy < 0 || yy >= ny) continue;
            const float wy = dy ? ay : 1.f - ay;
#pragma unroll
            for (int dx = 0; dx < 2; ++dx) {
                const int xx = ix + dx;
                if (xx < 0 || xx >= nx) continue;
                const float wx = dx ? ax : 1.f - ax;
                acc += wx * wy * wz * __ldg(vol + (static_cast<long long>(zz) * ny + yy) * nx + xx);
            }
        }
    }
    return acc;
}

// Forward projection: midpoint sums of trilinear samples every step_vox voxel lengths between a
// ray's two crossings of the grid's outer faces (half a voxel outside the outermost centres).
//
// Ray setup is FP64 and gives the sample positions as x(s) = x0 + s dx per axis in voxel-index
// units. The samples whose taps all lie in the grid (solved for s per axis, kEdge voxels inside the
// taps' range) run without range checks in chunks of kChunk samples: the chunk's middle is evaluated
// in FP64 and split into a whole voxel, which goes into the chunk's base pointer, and a remainder;
// the samples are FP32 steps from it. A position's rms error against FP64 is 1.3e-7 voxels for steps of half a voxel
// and 2.6e-7 for whole ones (2.5e-7 and 5e-7 with steps from the chunk's start); FP64 positions rounded to FP32
// have 1.7e-7 on 12 voxels, 4.1e-7 on 32 and 7e-7 on 48. Rays that step more than 1/22 of an axis, where
// those are the better ones, take the range-checked path, which has them. The floor is one add that rounds down
// at 1.5 * 2^23 (its bits are the voxel offset). The samples at a ray's two ends take the range-checked
// path too.
//
// The warp marches its rays in step along axis 1: lane l takes sample k + o_l in iteration k, o_l
// chosen so that every lane is at the same plane of axis 1 (rays that enter through different faces
// start at different depths). The 32 lanes' taps then lie in one or two rows of the grid.
//
// Bound by the latency and the L1 wavefronts of the gathers (3.3 lines per request of (z, z + 1)
// pairs), so four blocks per SM (64 registers, the ray setup spills) beat three (80 registers: 20.1 ms)
// and two with twice the loads in flight (18.7 ms). 192^3 grid, 180 views of 384 x 288, half-voxel
// steps (7.7e9 samples): 70.7 ms with FP64 positions and range checks per sample, 54 ms without
// those, 33 ms with the exchanged copy, 19.3 ms marching in step, 16.5 ms with packed pairs and the
// masked ends, 15.6 with only the samples that some lane takes there. Chunks of 64 samples: 18.8 ms (more
// masked samples at the rays' ends).
constexpr int kChunk = 32;
constexpr double kEdge = 1.0 / 1024.0;
constexpr float kFloorShift = 12582912.0f;  // 1.5 * 2^23
constexpr int kFloorBits = 0x4B400000;

// (1 - f) a + f b with g = 1 - f. Infinite taps of either sign stay what the sum of the weighted taps
// makes of them (a + f (b - a) would turn them into NaN).
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 f, float2 g)
{
    return __ffma2_rn(f, b, __fmul2_rn(g, a));
}

// Sum of one ray; every lane of the warp calls it (`on` false: the lane has no ray). `grid` holds the
// box's voxels (PAIRS: each with the voxel of the next plane); the range-checked samples read `vol`,
// in which x and y are the other way round where `swapped`. Off: the type of byte offsets into the
// grid (32 bits below 4 GB: one register, added to a uniform address).
template <bool PLANAR, bool PAIRS, class Off>
__device__ __forceinline__ float forward_ray(const Ray &ray, bool on, const float *__restrict__ vol,
                                             const float *__restrict__ grid, bool swapped, const VolBox &box,
                                             float step_vox)
{
    constexpr int NA = PLANAR ? 2 : 3;
    const int n[3] = {box.nx, box.ny, box.nz};
    const double dn = sqrt(ray.d[0] * ray.d[0] + ray.d[1] * ray.d[1] + ray.d[2] * ray.d[2]);
    double dir[NA];
    // slab intersection with the voxel-centre box extended by half a voxel
    double t0 = -1e300, t1 = 1e300;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        dir[a] = ray.d[a] / dn;
        const double lo = box.lo[a] - 0.5 * box.w[a], hi = box.hi[a] + 0.5 * box.w[a];
        if (fabs(dir[a]) < 1e-15) {
            if (ray.o[a] < lo || ray.o[a] > hi) on = false;
            continue;
        }
        const double ta = (lo - ray.o[a]) / dir[a], tb = (hi - ray.o[a]) / dir[a];
        t0 = fmax(t0, fmin(ta, tb));
        t1 = fmin(t1, fmax(ta, tb));
    }
    const double wmin = PLANAR ? fmin(box.w[0], box.w[1]) : fmin(box.w[0], fmin(box.w[1], box.w[2]));
    const double h = static_cast<double>(step_vox) * wmin;
    const long long ns = on && t1 > t0 ? static_cast<long long>(ceil((t1 - t0) / h)) : 0;
    // x(s) = x0 + s dx; samples [sa, sb) have every tap inside the grid
    double x0[NA], dx[NA], fa = 0.0, fb = static_cast<double>(ns) - 1.0;
    bool fine = true;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        x0[a] = (ray.o[a] + (t0 + 0.5 * h) * dir[a] - box.lo[a]) / box.w[a];
        dx[a] = h * dir[a] / box.w[a];
        fine = fine && fabs(dx[a]) <= fmin(1.0, n[a] * (1.0 / 22.0));
        const double lo = kEdge - x0[a], hi = (n[a] - 1.0 - kEdge) - x0[a];
        if (fabs(dx[a]) * static_cast<double>(ns) < 0.5 * kEdge) {  // stays where it starts
            if (!(lo + 0.5 * kEdge <= 0.0 && hi - 0.5 * kEdge >= 0.0)) fb = -1.0;
        } else {
            fa = fmax(fa, (dx[a] > 0.0 ? lo : hi) / dx[a]);
            fb = fmin(fb, (dx[a] > 0.0 ? hi : lo) / dx[a]);
        }
    }
    long long sa = ns, sb = ns;
    if (fb >= fa && fine && ns < (1LL << 30) && static_cast<long long>(box.nx) * box.ny <= (1LL << 25)) {
        sa = static_cast<long long>(ceil(fa));
        sb = static_cast<long long>(floor(fb)) + 1;
        if (sb <= sa) sa = sb = ns;
    }
    float sum = 0.f;
    auto checked = [&](long long s) {
        const double f = static_cast<double>(s);
        const float x = static_cast<float>(fma(f, dx[0], x0[0])), y = static_cast<float>(fma(f, dx[1], x0[1]));
        const float z = PLANAR ? 0.f : static_cast<float>(fma(f, dx[NA - 1], x0[NA - 1]));
        sum += swapped ? trilinear(vol, box.ny, box.nx, box.nz, y, x, z) : trilinear(vol, box.nx, box.ny, box.nz, x, y, z);
    };
    for (long long s = 0; s < sa; ++s) checked(s);
    // iterations [ka, kb) of this lane in the warp's march
    const bool run = sb > sa;
    const unsigned runners = __ballot_sync(0xffffffffu, run);
    int ka = INT_MAX, kb = INT_MIN, shift = 0;
    if (runners) {
        const double yref = __shfl_sync(0xffffffffu, x0[1], __ffs(runners) - 1);
        if (run) {
            if (fabs(dx[1]) > 0.1) {
                const double o = rint((yref - x0[1]) / dx[1]);
                if (fabs(o) < 1e6) shift = static_cast<int>(o);
            }
            ka = static_cast<int>(sa) - shift;
            kb = static_cast<int>(sb) - shift;
        }
    }
    const int kend = __reduce_max_sync(0xffffffffu, kb);
    const int sy = box.nx, sz = box.nx * box.ny;
    const float d[3] = {static_cast<float>(dx[0]), static_cast<float>(dx[1]), PLANAR ? 0.f : static_cast<float>(dx[NA - 1])};
    // the taps of a voxel offset: row addresses, the same for every lane (offsets in bytes)
    constexpr int kVox = PAIRS ? 8 : 4;
    const char *const b00 = reinterpret_cast<const char *>(grid), *const b01 = b00 + static_cast<long long>(kVox) * sy,
                      *const b10 = b00 + static_cast<long long>(kVox) * sz,
                      *const b11 = b10 + static_cast<long long>(kVox) * sy;
    auto at = [](const char *row, Off o) { return __ldg(reinterpret_cast<const float *>(row + o)); };
    auto at2 = [](const char *row, Off o) { return __ldg(reinterpret_cast<const float2 *>(row + o)); };
    float2 sum2 = make_float2(0.f, 0.f);
    for (int k0 = __reduce_min_sync(0xffffffffu, ka); k0 < kend; k0 += kChunk) {
        const bool here = ka < k0 + kChunk && kb > k0;  // else no sample of this lane in the chunk
        const unsigned lanes = __ballot_sync(0xffffffffu, here);
        if (!here) continue;
        float r[3] = {0.f, 0.f, 0.f};
        long long c[3] = {0, 0, 0};
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const double xb = fma(static_cast<double>(k0 + shift + kChunk / 2), dx[a], x0[a]), fl = floor(xb);
            c[a] = static_cast<int>(fl);
            r[a] = static_cast<float>(xb - fl);
        }
        // byte offset of the chunk's middle voxel, less what the bits of the shifted floors add (both
        // modulo 2^32 in the 32-bit form: the sum is the offset of a voxel of the grid)
        const Off base = static_cast<Off>(kVox * ((c[2] * box.ny + c[1]) * box.nx + c[0] -
                                                  static_cast<long long>(kFloorBits) * (1LL + sy + (PLANAR ? 0 : sz))));
        // samples k and k + 1 as packed pairs at (FP32) steps fk from the chunk's middle
        auto pair = [&](float2 fk) -> float2 {
            float2 f[NA], g[NA];
            Off o0 = base, o1 = base;
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                const float2 x = __ffma2_rn(fk, make_float2(d[a], d[a]), make_float2(r[a], r[a]));
                const float2 t = __fadd2_rd(x, make_float2(kFloorShift, kFloorShift));  // floor(x) in the low bits
                f[a] = __ffma2_rn(__fadd2_rn(t, make_float2(-kFloorShift, -kFloorShift)), make_float2(-1.f, -1.f), x);
                g[a] = __ffma2_rn(f[a], make_float2(-1.f, -1.f), make_float2(1.f, 1.f));
                const Off st = a == 0 ? kVox : static_cast<Off>(static_cast<long long>(kVox) * (a == 1 ? sy : sz));
                o0 += static_cast<Off>(__float_as_int(t.x)) * st;
                o1 += static_cast<Off>(__float_as_int(t.y)) * st;
            }
            if constexpr (PAIRS) {
                // (z, z + 1) pairs of four taps per sample
                const float2 p00 = at2(b00, o0), p01 = at2(b00 + 8, o0), p10 = at2(b01, o0), p11 = at2(b01 + 8, o0);
                const float2 q00 = at2(b00, o1), q01 = at2(b00 + 8, o1), q10 = at2(b01, o1), q11 = at2(b01 + 8, o1);
                const auto two = [](float v) { return make_float2(v, v); };
                const float2 x0 = two(f[0].x), y0 = two(f[1].x), x1 = two(f[0].y), y1 = two(f[1].y);
                const float2 gx0 = two(g[0].x), gy0 = two(g[1].x), gx1 = two(g[0].y), gy1 = two(g[1].y);
                const float2 e0 = lerp2(lerp2(p00, p01, x0, gx0), lerp2(p10, p11, x0, gx0), y0, gy0);
                const float2 e1 = lerp2(lerp2(q00, q01, x1, gx1), lerp2(q10, q11, x1, gx1), y1, gy1);
                return lerp2(make_float2(e0.x, e1.x), make_float2(e0.y, e1.y), f[NA - 1], g[NA - 1]);
            } else {
                const float2 v00 = make_float2(at(b00, o0), at(b00, o1)), v01 = make_float2(at(b00 + 4, o0), at(b00 + 4, o1));
                const float2 v10 = make_float2(at(b01, o0), at(b01, o1)), v11 = make_float2(at(b01 + 4, o0), at(b01 + 4, o1));
                const float2 e = lerp2(lerp2(v00, v01, f[0], g[0]), lerp2(v10, v11, f[0], g[0]), f[1], g[1]);
                if constexpr (PLANAR) return e;
                const float2 w00 = make_float2(at(b10, o0), at(b10, o1)), w01 = make_float2(at(b10 + 4, o0), at(b10 + 4, o1));
                const float2 w10 = make_float2(at(b11, o0), at(b11, o1)), w11 = make_float2(at(b11 + 4, o0), at(b11 + 4, o1));
                return lerp2(e, lerp2(lerp2(w00, w01, f[0], g[0]), lerp2(w10, w11, f[0], g[0]), f[1], g[1]), f[NA - 1],
                             g[NA - 1]);
            }
        };
        const int first = max(ka - k0, 0), last = min(kb - k0, kChunk) - 1;
        if (__all_sync(lanes, first == 0 && last == kChunk - 1)) {
            float2 fk = make_float2(-0.5f * kChunk, 1.f - 0.5f * kChunk);
#pragma unroll 1
            for (int k = 0; k < kChunk; k += 2, fk = __fadd2_rn(fk, make_float2(2.f, 2.f))) sum2 = __fadd2_rn(sum2, pair(fk));
        } else {  // some ray starts or ends in the chunk: its other samples repeat its first or last one, unsummed
            const float lo = static_cast<float>(first - kChunk / 2), hi = static_cast<float>(last - kChunk / 2);
            const int k1 = __reduce_max_sync(lanes, last);
            int k = __reduce_min_sync(lanes, first);
            float2 fk = make_float2(static_cast<float>(k - kChunk / 2), static_cast<float>(k + 1 - kChunk / 2));
#pragma unroll 1
            for (; k <= k1; k += 2, fk = __fadd2_rn(fk, make_float2(2.f, 2.f))) {
                const float2 fc = make_float2(fminf(fmaxf(fk.x, lo), hi), fminf(fmaxf(fk.y, lo), hi));
                const float2 e = pair(fc);
                sum2.x += fc.x == fk.x ? e.x : 0.f;
                sum2.y += fc.y == fk.y ? e.y : 0.f;
            }
        }
    }
    sum += sum2.x + sum2.y;
    for (long long s = sb; s < ns; ++s) checked(s);
    return sum * static_cast<float>(h);
}

// Whether a view's rays run more along x than along y (its central direction, one answer per view).
__device__ __forceinline__ bool along_x(const ProjView &pv, int kind)
{
    double x = pv.ew[0], y = pv.ew[1];
    if (kind == GCT_GEOM_PARALLEL_1D || kind == GCT_GEOM_PARALLEL_2D || kind == GCT_GEOM_CONE_PARALLEL)
        sincos(pv.extra, &y, &x);
    return fabs(x) > fabs(y);
}
template <class T>
__device__ __forceinline__ void swap2(T *a)
{
    const T t = a[0];
    a[0] = a[1];
    a[1] = t;
}

// Blocks take tiles of bx x by detector pixels of one view (bx by = 256, bx >= 32), in turn. The
// rays of a warp lie side by side across their direction, so a warp's taps are neighbours along the
// grid axis that the rays cross. Views whose rays run along x read `along`, the grid with x and y
// exchanged (NULL for none), where those neighbours are contiguous; in the grid itself they are nx
// voxels apart and every gather would touch 32 cache lines.
template <bool PLANAR, bool PAIRS, class Off>
__global__ void __launch_bounds__(256, 4) forward_kernel(const ProjView *__restrict__ views, int kind, int nv, int nr,
                                                         int nc, double du, double dv, const float *__restrict__ vol,
                                                         const float *__restrict__ across,
                                                         const float *__restrict__ along, VolBox box, float step_vox,
                                                         int bx, float *__restrict__ out)
{
    const int by = 256 / bx, tc = (nc + bx - 1) / bx, tr = (nr + by - 1) / by;
    const long long tiles = static_cast<long long>(nv) * tr * tc;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int v = static_cast<int>(tile / (static_cast<long long>(tr) * tc));
        const int rem = static_cast<int>(tile - static_cast<long long>(v) * tr * tc);
        const int r = (rem / tc) * by + threadIdx.x / bx, c = (rem % tc) * bx + threadIdx.x % bx;
        const bool on = r < nr && c < nc;
        Ray ray = make_ray(views[v], kind, du, dv, c, r);
        if (PLANAR) {
            ray.o[2] = box.lo[2];
            ray.d[2] = 0.0;
        }
        VolBox b = box;
        const bool swapped = along && along_x(views[v], kind);
        if (swapped) {  // x and y exchanged throughout
            swap2(ray.o);
            swap2(ray.d);
            swap2(b.lo);
            swap2(b.hi);
            swap2(b.w);
            b.nx = box.ny;
            b.ny = box.nx;
        }
        const float sum = forward_ray<PLANAR, PAIRS, Off>(ray, on, vol, swapped ? along : across, swapped, b, step_vox);
        if (on) out[(static_cast<long long>(v) * nr + r) * nc + c] = sum;
    }
}

// The grid's copies for the rays, in one pass over 32 x 32 tiles (32 x 8 threads): along[z][x][y] =
// vol[z][y][x]; PAIRS: along and across as (z, z + 1) pairs (zero past the last plane).
template <bool PAIRS>
__global__ void arrange_grid_kernel(const float *__restrict__ vol, int nx, int ny, int nz, float *__restrict__ across,
                                    float *__restrict__ along)
{
    __shared__ float tile[2][32][33];
    const int tx = (nx + 31) / 32, ty = (ny + 31) / 32;
    const long long tiles = static_cast<long long>(tx) * ty * nz, plane = static_cast<long long>(nx) * ny;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        const long long z = t / (static_cast<long long>(tx) * ty);
        const int rem = static_cast<int>(t - z * tx * ty), x0 = (rem % tx) * 32, y0 = (rem / tx) * 32;
        for (int k = threadIdx.y; k < 32; k += 8) {
            if (y0 + k >= ny || x0 + threadIdx.x >= nx) continue;
            const long long at = z * plane + static_cast<long long>(y0 + k) * nx + x0 + threadIdx.x;
            const float v = __ldg(vol + at), w = PAIRS && z + 1 < nz ? __ldg(vol + at + plane) : 0.f;
            tile[0][k][threadIdx.x] = v;
            if (PAIRS) {
                tile[1][k][threadIdx.x] = w;
                reinterpret_cast<float2 *>(across)[at] = make_float2(v, w);
            }
        }
        __syncthreads();
        for (int k = threadIdx.y; k < 32; k += 8) {
            if (x0 + k >= nx || y0 + threadIdx.x >= ny) continue;
            const long long at = z * plane + static_cast<long long>(x0 + k) * ny + y0 + threadIdx.x;
            if (PAIRS) reinterpret_cast<float2 *>(along)[at] = make_float2(tile[0][threadIdx.x][k], tile[1][threadIdx.x][k]);
            else along[at] = tile[0][threadIdx.x][k];
        }
        __syncthreads();
    }
}

}  // namespace

void launch_phantom(const ProjView *views, int kind, int nv, int nr, int nc, double du, double dv,
                    const gct_ellipsoid *ell, int ne, bool planar, float *out, int num_sms,
                    cudaStream_t s)
{
    const long long total = static_cast<long long>(nv) * nr * nc;
    long long grid = (total + 255) / 256;
    if (grid > static_cast<long long>(num_sms) * 32) grid = static_cast<long long>(num_sms) * 32;
    if (grid < 1) grid = 1;
    phantom_kernel<<<static_cast<unsigned>(grid), 256, 0, s>>>(views, kind, nv, nr, nc, du, dv, ell, ne,
                                                               planar, out);
}

void launch_forward(const ProjView *views, int kind, int nv, int nr, int nc, double du, double dv,
                    const float *vol, ForwardCopies copies, float *scratch, const VolBox &box, float step_vox, float *out,
                    int num_sms, cudaStream_t s)
{
    const long long voxels = static_cast<long long>(box.nx) * box.ny * box.nz;
    const float *across = vol, *along = nullptr;
    const bool pairs = copies == ForwardCopies::Pairs;
    if (copies != ForwardCopies::None) {
        float *ac = pairs ? scratch : nullptr, *al = pairs ? scratch + 2 * voxels : scratch;
        long long grid = static_cast<long long>((box.nx + 31) / 32) * ((box.ny + 31) / 32) * box.nz;
        if (grid > static_cast<long long>(num_sms) * 64) grid = static_cast<long long>(num_sms) * 64;
        if (!pairs)
            arrange_grid_kernel<false><<<static_cast<unsigned>(grid), dim3(32, 8), 0, s>>>(vol, box.nx, box.ny, box.nz, ac, al);
        else
            arrange_grid_kernel<true><<<static_cast<unsigned>(grid), dim3(32, 8), 0, s>>>(vol, box.nx, box.ny, box.nz, ac, al);
        if (pairs) across = ac;
        along = al;
    }
    const int bx = nr >= 8 ? 32 : nr >= 4 ? 64 : nr >= 2 ? 128 : 256, by = 256 / bx;
    long long grid = static_cast<long long>(nv) * ((nr + by - 1) / by) * ((nc + bx - 1) / bx);
    if (grid > static_cast<long long>(num_sms) * 64) grid = static_cast<long long>(num_sms) * 64;
    if (grid < 1) grid = 1;
    auto go = [&](auto kern) {
        kern<<<static_cast<unsigned>(grid), 256, 0, s>>>(views, kind, nv, nr, nc, du, dv, vol, across, along, box,
                                                         step_vox, bx, out);
    };
    if (box.planar) go(forward_kernel<true, false, long long>);
    else if (!pairs) go(forward_kernel<false, false, long long>);
    else if (8 * voxels < (1LL << 32)) go(forward_kernel<false, true, unsigned>);
    else go(forward_kernel<false, true, long long>);
}

ForwardCopies forward_copies(const VolBox &box, const ProjView *views, int kind, int nv, int nr, int nc,
                             float step_vox)
{
    const long long voxels = static_cast<long long>(box.nx) * box.ny * box.nz;
    if (voxels <= kCopyVoxels) return ForwardCopies::None;
    if (box.planar) return ForwardCopies::Along;
    if (16 * voxels <= kSmallCopies) return ForwardCopies::Pairs;
    const double h = step_vox * std::min(box.w[0], std::min(box.w[1], box.w[2]));
    const double samples = std::max(box.nx * box.w[0], box.ny * box.w[1]) / h * nr * nc;  // of a view
    double along_x = 0.0, others = 0.0;
    for (int v = 0; v < nv; ++v) {
        const bool parallel = kind == GCT_GEOM_PARALLEL_2D || kind == GCT_GEOM_CONE_PARALLEL;
        const double dy = std::fabs(parallel ? std::sin(views[v].extra) : views[v].ew[1]) * h / box.w[1];
        (dy < 0.1 ? along_x : others) += samples;
    }
    const double pairs = kSaveX * along_x + kPairsSave * others - kCopyCall - kPairsVoxel * voxels;
    const double along = kSaveX * along_x - kCopyCall - kAlongVoxel * voxels;
    return std::max(pairs, along) <= 0.0 ? ForwardCopies::None : pairs >= along ? ForwardCopies::Pairs : ForwardCopies::Along;
}

long long forward_copy_floats(const VolBox &box, ForwardCopies copies)
{
    const long long voxels = static_cast<long long>(box.nx) * box.ny * box.nz;
    return copies == ForwardCopies::Pairs ? 4 * voxels : copies == ForwardCopies::Along ? voxels : 0;
}

}  // namespace gct
