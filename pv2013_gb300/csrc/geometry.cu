// GPU voxelization and boundary classification (sm_103a).  Compiled with
// -fmad=false: every FP64 expression below is evaluated operation by
// operation like the reference's C++ (no fused multiply-add), which is what
// makes the node-type field bit-exact.
//
// Reference semantics restated here:
//   grid points        x = min_x + i*spacing        ComplexGeometry.cpp:199-201
//   ray                +z from the point, end z = (z + L) + 0.1, L = max_z-min_z,
//                      x/y nudged 0.01 inward on bbox faces  :334-357, :438-492
//   crossing test      t = ((q-p).n)/((e-s).n) with the file normal,
//                      t in [-1e-7, 1+1e-7], then the inclusive xy inside test
//                      at (p + t(e-s))                          :284-330, :264-281
//   label              odd count -> Fluid                       :495-502
//   boundary points    Fluid with a NotFluid 26-neighbour or on a bbox face,
//                      x-major order                            :509-556
//   lists              plane predicates, then wall = the rest   :559-638
//
// Work decomposition (GB300-first, not the reference's point x triangle loop):
//   1. one thread per triangle enumerates the grid columns (i,j) whose ray can
//      pass its xy-projection (its bounding box, widened; for needle-thin
//      projections also the columns on the supporting line, where rounding can
//      make the inclusive test succeed beyond the segment) and keeps those
//      passing the exact xy test.  Count pass, scan, fill pass -> per-column
//      candidate lists.
//   2. one warp per column, one lane per candidate: the z range in which the
//      exact crossing test counts the candidate, as a parity mask over the
//      column's points; one bit per point is written.
// Because the ray is vertical, the xy inside test is independent of z, so
// the split is exact.
//
// GB300 retires about 2 FP64 operations per clock and SM, so the exact tests
// bound these kernels wherever they run.  They run only where a cheaper bound
// leaves the answer open:
//   xy test    in FP32 cell units relative to the triangle; decided there unless
//              a cross product lies within its error bound of zero
//   needles    a column further from the supporting line than the rounding of
//              the exact test is skipped after one distance; lines along a
//              grid axis are skipped whole
//   crossings  the range's ends come from the plane equation; the exact
//              test (its division included) runs for the one point that lies
//              within the rounding of an end, if any
// Measured on the 4.76 M-triangle vascular tree (512x1024x512): count / fill /
// columns 18.4 / 18.6 / 11.4 ms with the exact tests everywhere, 1.6 / 1.5 / 0.9 ms now.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "bits.cuh"
#include "column_range.h"
#include "device.cuh"
#include "internal.h"
#include "scan.cuh"
#include "nvtx.h"

namespace lbm {

struct VoxGrid {
    double bb[6];      // min_x,max_x,min_y,max_y,min_z,max_z
    double spacing;
    int32_t Nx, Ny, Nz;
};

// ---------------------------------------------------------------------------
// exact helpers (no contraction in this TU)

__device__ __forceinline__ bool inside2d(double x, double y, const double* T) {
    const double x1 = T[0], y1 = T[1], x2 = T[3], y2 = T[4], x3 = T[6], y3 = T[7];
    const double d1 = ((x - x2) * (y1 - y2) - (y - y2) * (x1 - x2));
    const double d2 = ((x - x3) * (y2 - y3) - (y - y3) * (x2 - x3));
    const double d3 = ((x - x1) * (y3 - y1) - (y - y1) * (x3 - x1));
    const bool neg = (d1 < 0) || (d2 < 0) || (d3 < 0);
    const bool pos = (d1 > 0) || (d2 > 0) || (d3 > 0);
    return !(neg && pos);
}

// Ray start x,y of column (i,j) after adjustLineCoordinates case 0.
__device__ __forceinline__ void column_xy(const VoxGrid& g, int i, int j, double& sx, double& sy) {
    sx = g.bb[0] + (double)i * g.spacing;
    sy = g.bb[2] + (double)j * g.spacing;
    const double off = 0.01;
    if (sx == g.bb[0]) sx += off;
    if (sx == g.bb[1]) sx -= off;
    if (sy == g.bb[2]) sy += off;
    if (sy == g.bb[3]) sy -= off;
}

// Candidate columns of triangle T, in two parts.  enum_box calls fn(col) for
// the columns of the projection's bounding box that pass the exact xy test
// and returns kPointLike when the projection is degenerate to a point (such
// a triangle is tested by every column instead), kNeedle when it is so thin
// that the xy test can also pass on its supporting line outside the box, and
// kBoxOnly otherwise.  enum_band covers the needle case: the columns on the
// supporting line of the longest edge across the whole grid, lanes striding
// over the line's major axis (a warp shares one triangle's band).
constexpr int kPointLike = 0, kBoxOnly = 1, kNeedle = 2;

struct BoxRange {
    int i0, i1, j0, j1;
};

// FP64 classification of a thin projection (see enum_box)
__device__ __noinline__ int classify_thin(const double* T) {
    const double xmn = fmin(T[0], fmin(T[3], T[6])), xmx = fmax(T[0], fmax(T[3], T[6]));
    const double ymn = fmin(T[1], fmin(T[4], T[7])), ymx = fmax(T[1], fmax(T[4], T[7]));
    const double ex[3] = {T[3] - T[0], T[6] - T[3], T[0] - T[6]};
    const double ey[3] = {T[4] - T[1], T[7] - T[4], T[1] - T[7]};
    double best = -1.0;
    for (int m = 0; m < 3; ++m) {
        const double l = fabs(ex[m]) + fabs(ey[m]);
        if (l > best) best = l;
    }
    const double scale = 1.0 + fmax(fmax(fabs(xmn), fabs(xmx)), fmax(fabs(ymn), fabs(ymx)));
    if (!(best > 1e-9 * scale)) return kPointLike;    // point-like projection: every column tests it
    // needle-thin projection: the band below is needed as well
    const double area2 = fabs((T[3] - T[0]) * (T[7] - T[1]) - (T[4] - T[1]) * (T[6] - T[0]));
    return area2 > 1e-9 * best * scale ? kBoxOnly : kNeedle;   // height above 1e-9 relative: box is enough
}

template <class F>
__device__ __forceinline__ int enum_box(const VoxGrid& g, double inv_s, const double* __restrict__ T, BoxRange& r, F fn) {
    // projected vertices in cell units from the grid's corner
    double wx[3], wy[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        wx[m] = (T[3 * m] - g.bb[0]) * inv_s;
        wy[m] = (T[3 * m + 1] - g.bb[2]) * inv_s;
    }
    const float fx0 = (float)wx[0], fx1 = (float)wx[1], fx2 = (float)wx[2];
    const float fy0 = (float)wy[0], fy1 = (float)wy[1], fy2 = (float)wy[2];
    const float xmn = fminf(fx0, fminf(fx1, fx2)), xmx = fmaxf(fx0, fmaxf(fx1, fx2));
    const float ymn = fminf(fy0, fminf(fy1, fy2)), ymx = fmaxf(fy0, fmaxf(fy1, fy2));
    const float big = fmaxf(fmaxf(fabsf(xmn), fabsf(xmx)), fmaxf(fabsf(ymn), fabsf(ymx)));
    // columns whose ray (min + i*s, nudged by at most 0.01 at the grid faces)
    // can lie in the projection: its bounding box widened by the nudge and by
    // the rounding of these cell coordinates (a superset; the xy test decides)
    const float nudge = (float)(0.01 * inv_s) * 1.0001f;
    const float mg = nudge + 1e-3f + big * 4e-7f;
    const bool near_ = big < 1e6f;                    // (false for NaN)
    if (near_) {
        r.i0 = (int)ceilf(fmaxf(xmn - mg, 0.f));
        r.i1 = last_column(xmx + mg, g.Nx);
        r.j0 = (int)ceilf(fmaxf(ymn - mg, 0.f));
        r.j1 = last_column(ymx + mg, g.Ny);
    } else {                                          // far from the grid: the same in FP64 (NaN: the whole range)
        const double md = 0.01 * inv_s + 1e-3 + (double)big * 1e-12;
        r.i0 = (int)ceil(fmin(fmax(fmin(wx[0], fmin(wx[1], wx[2])) - md, 0.0), (double)g.Nx));
        r.i1 = (int)floor(fmax(fmin(fmax(wx[0], fmax(wx[1], wx[2])) + md, (double)(g.Nx - 1)), -1.0));
        r.j0 = (int)ceil(fmin(fmax(fmin(wy[0], fmin(wy[1], wy[2])) - md, 0.0), (double)g.Ny));
        r.j1 = (int)floor(fmax(fmin(fmax(wy[0], fmax(wy[1], wy[2])) + md, (double)(g.Ny - 1)), -1.0));
    }
    const bool empty = r.i0 > r.i1 || r.j0 > r.j1;
    // vertices relative to the box's corner (outside the grid too), FP32: small
    // numbers, error below 1e-6 of the extent
    const float rx = floorf(xmn - mg), ry = floorf(ymn - mg);
    float x[3], y[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        x[m] = (float)(wx[m] - (double)rx);
        y[m] = (float)(wy[m] - (double)ry);
    }
    const float ext = fmaxf(fabsf(xmx - xmn), fabsf(ymx - ymn));
    const float area = (x[1] - x[0]) * (y[2] - y[0]) - (y[1] - y[0]) * (x[2] - x[0]);
    // thin (or not a number): the FP64 classification.  The FP32 area's error is
    // below 8.4e-7 vs^2; the second term is above the needle bound, 1e-9 of the
    // longest edge times the coordinates
    const float far_ = big + fabsf((float)(g.bb[0] * inv_s)) + fabsf((float)(g.bb[2] * inv_s)) + (float)inv_s;
    const float vs = ext + 2.f + mg;                  // bounds the vertices' coordinates
    const bool thick = near_ && fabsf(area) > vs * vs * 2e-6f + ext * far_ * 4e-9f;
    const int kind = thick ? kBoxOnly : classify_thin(T);
    if (kind == kPointLike || empty) return kind;
    // error bound of a cross product of FP32 differences: 8.4e-7 span^2, and the
    // columns' own rounding (1e-16 of far_)
    const float span = ext + 2.f + 3.f * mg;          // bounds the columns' coordinates too
    const float err = 2e-6f * span * span;
    const bool fp32 = near_ && ext < 1e3f && far_ < 1e8f;
    for (int i = r.i0; i <= r.i1; ++i)
        for (int j = r.j0; j <= r.j1; ++j) {
            // (a column that may be nudged: the first, and the one at the box's far face)
            const bool face = i == 0 || j == 0 || i >= g.Nx - 2 || j >= g.Ny - 2;
            bool in, open = true;
            if (fp32 && !face) {
                const float px = (float)i - rx, py = (float)j - ry;
                const float d1 = (px - x[1]) * (y[0] - y[1]) - (py - y[1]) * (x[0] - x[1]);
                const float d2 = (px - x[2]) * (y[1] - y[2]) - (py - y[2]) * (x[1] - x[2]);
                const float d3 = (px - x[0]) * (y[2] - y[0]) - (py - y[0]) * (x[2] - x[0]);
                const float lo = fminf(d1, fminf(d2, d3)), hi = fmaxf(d1, fmaxf(d2, d3));
                if (lo < -err && hi > err) { in = false; open = false; }
                else if (lo > err || hi < -err) { in = true; open = false; }
            }
            if (open) {
                double sx, sy;
                column_xy(g, i, j, sx, sy);
                in = inside2d(sx, sy, T);
            }
            if (in) fn(i * (long)g.Ny + j);
        }
    return kind;
}

// A column at distance d from the needle's supporting line fails the exact
// xy test when d exceeds the needle's height (1e-9 of the coordinates, from the
// classification) plus the rounding of the cross products (8 ulp of the
// distance along the line): the longest edge's product then has its true sign, and
// of the two other edges, which run back along the line, at least one has the
// opposite.  The skip uses 1e-7 of (coordinates + grid extent) for both.
template <class F>
__device__ __noinline__ void enum_band(const VoxGrid& g, const double* T, const BoxRange& r, int lane, int nl, F fn) {
    const double s = g.spacing;
    double ex[3] = {T[3] - T[0], T[6] - T[3], T[0] - T[6]};
    double ey[3] = {T[4] - T[1], T[7] - T[4], T[1] - T[7]};
    int e = 0;
    double best = -1.0;
    for (int m = 0; m < 3; ++m) {
        double l = fabs(ex[m]) + fabs(ey[m]);
        if (l > best) { best = l; e = m; }
    }
    const double ox = T[3 * e], oy = T[3 * e + 1];
    const double dx = ex[e], dy = ey[e];
    const bool along_x = fabs(dx) >= fabs(dy);
    // major axis m, minor axis n
    const double slope = along_x ? dy / dx : dx / dy;
    const double om = along_x ? ox : oy, on = along_x ? oy : ox;
    const double base_n = along_x ? g.bb[2] : g.bb[0];
    const int Nm = along_x ? g.Nx : g.Ny, Nn = along_x ? g.Ny : g.Nx;
    const int m0 = along_x ? r.i0 : r.j0, m1 = along_x ? r.i1 : r.j1;
    const double reach = fabs(ox) + fabs(oy) + fabs(g.bb[0]) + fabs(g.bb[1]) + fabs(g.bb[2]) + fabs(g.bb[3]) + best + 1.0;
    const double tol = 1e-7 * reach;
    auto minor_range = [&](double n, long& lo, long& hi) {     // columns within tol of the line, nudged faces included
        lo = max(0L, (long)floor((n - tol - 0.01 - base_n) / s));
        hi = min((long)Nn - 1, (long)ceil((n + tol + 0.01 - base_n) / s));
    };
    auto visit = [&](long m, double n, long lo, long hi) {
        for (long k = lo; k <= hi; ++k) {
            const int i = (int)(along_x ? m : k), j = (int)(along_x ? k : m);
            double sx, sy;
            column_xy(g, i, j, sx, sy);
            if (fabs((along_x ? sy : sx) - n) > tol) continue;
            if (inside2d(sx, sy, T)) fn(i * (long)g.Ny + j);
        }
    };
    if (slope == 0.0) {                                // parallel to a grid axis: one row of columns, or none
        long lo, hi;
        minor_range(on, lo, hi);
        bool any = false;
        for (long k = lo; k <= hi && !any; ++k) {
            double sx, sy;
            column_xy(g, along_x ? 0 : (int)k, along_x ? (int)k : 0, sx, sy);
            any = !(fabs((along_x ? sy : sx) - on) > tol);
        }
        if (!any) return;
    }
    for (long m = lane; m < Nm; m += nl) {
        if (m >= m0 && m <= m1) continue;
        double sx, sy;
        column_xy(g, along_x ? (int)m : 0, along_x ? 0 : (int)m, sx, sy);
        const double n = on + ((along_x ? sx : sy) - om) * slope;
        long lo, hi;
        minor_range(n, lo, hi);
        visit(m, n, lo, hi);
    }
}

// One thread per triangle for the box; the warp's needle triangles then
// take turns, each band scanned by all 32 lanes.  Threads past the end
// stay for the warp-wide vote.
template <class FMake>
__device__ void enumerate_warp(const VoxGrid& g, double inv_s, const double* tris, int64_t t, int64_t ntris, FMake make_fn,
                               int32_t* global_list, int32_t* nglobal) {
    const int lane = threadIdx.x & 31;
    const bool valid = t < ntris;
    int kind = kBoxOnly;
    BoxRange r = {0, -1, 0, -1};
    if (valid) {
        kind = enum_box(g, inv_s, tris + 12 * t, r, make_fn(t));
        if (kind == kPointLike && global_list) {
            const int slot = atomicAdd(nglobal, 1);
            global_list[slot] = (int32_t)t;
        }
    }
    unsigned m = __ballot_sync(0xffffffffu, valid && kind == kNeedle);
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const long long ts = __shfl_sync(0xffffffffu, (long long)t, src);
        BoxRange rs;
        rs.i0 = __shfl_sync(0xffffffffu, r.i0, src);
        rs.i1 = __shfl_sync(0xffffffffu, r.i1, src);
        rs.j0 = __shfl_sync(0xffffffffu, r.j0, src);
        rs.j1 = __shfl_sync(0xffffffffu, r.j1, src);
        enum_band(g, tris + 12 * ts, rs, lane, 32, make_fn((int64_t)ts));
    }
}

__global__ void k_tri_count(VoxGrid g, double inv_s, const double* __restrict__ tris, int64_t ntris,
                            int32_t* __restrict__ colcount, int32_t* __restrict__ global_list, int32_t* __restrict__ nglobal) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    enumerate_warp(g, inv_s, tris, t, ntris,
                   [&](int64_t) { return [colcount](long col) { atomicAdd(&colcount[col], 1); }; }, global_list, nglobal);
}

__global__ void k_tri_fill(VoxGrid g, double inv_s, const double* __restrict__ tris, int64_t ntris,
                           const int64_t* __restrict__ colstart, int32_t* __restrict__ cursor, int32_t* __restrict__ pairs) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    enumerate_warp(g, inv_s, tris, t, ntris, [&](int64_t tt) {
        return [=](long col) {
            int slot = atomicAdd(&cursor[col], 1);
            pairs[colstart[col] + slot] = (int32_t)tt;
        };
    }, nullptr, nullptr);
}

// Plane terms of a candidate in a column.
struct Cand {
    double c;     // (qx - sx)*nx + (qy - sy)*ny
    double qz;
    double nz;
    double d0;    // (ex - sx)*nx + (ey - sy)*ny  (ex == sx, ey == sy)
};

// the exact crossing test of the ray from point z of the column
__device__ __forceinline__ bool crosses(const VoxGrid& g, double L, const Cand& cd, int z) {
    const double pz = g.bb[4] + (double)z * g.spacing;
    double ez = pz + L;
    ez = ez + 0.1;
    const double dzv = ez - pz;
    const double num = cd.c + (cd.qz - pz) * cd.nz;
    const double den = cd.d0 + dzv * cd.nz;
    const double t = num / den;
    return t >= -1e-7 && t <= 1 + 1e-7;
}

// The points z of the column that the candidate's crossing test counts: a range
// [lo, hi], because t falls with z.  With the plane's height zc = qz + c/nz,
// t = (zc - pz) / (L + 0.1), so the ends are where pz passes zc + 1e-7 (L + 0.1)
// and zc - (1 + 1e-7)(L + 0.1).  The computed t and these ends differ from the
// real ones by less than 32 ulp of (|c/nz| + |qz| + |bb| + L) in z: where that is
// below 1e-3 of a spacing, only a point within 4e-3 spacings of an end needs the
// exact test, else the caller tests every point (returns false).  The 32 ulp hold
// where no product with nz under- or overflows: nz within 2^+-800 and a spacing below
// 1e30, whose lengths (within 1.3e11 spacings by the bound above) stay below 1e42.
__device__ __forceinline__ bool cross_range(const VoxGrid& g, double inv_s, double L, const Cand& cd, int& lo, int& hi) {
    lo = 0;
    hi = -1;
    if (cd.nz == 0.0 && cd.d0 == 0.0) return true;     // den 0: t is not finite, nothing counts
    const uint32_t en = ((uint32_t)__double2hiint(cd.nz) >> 20) & 0x7ffu;
    if (en - (1023u - 800u) > 1600u || !(g.spacing < 1e30)) return false;
    const double h = cd.c / cd.nz, zc = cd.qz + h;
    const double slack = 64.0 * 1.2e-16 * (fabs(h) + fabs(cd.qz) + fabs(g.bb[4]) + fabs(g.bb[5]) + L + 1.0);
    if (!(slack < 1e-3 * g.spacing) || cd.d0 != 0.0) return false;   // (NaN too)
    const double up = (zc + 1e-7 * (L + 0.1) - g.bb[4]) * inv_s;
    const double dn = (zc - (1.0 + 1e-7) * (L + 0.1) - g.bb[4]) * inv_s;
    if (!(fabs(up) < 1e9) || !(fabs(dn) < 1e9)) return false;
    const double un = rint(up), dnn = rint(dn);
    int z = (int)un;
    if (fabs(up - un) > 4e-3 || z < 0 || z >= g.Nz) hi = (int)floor(up);
    else hi = crosses(g, L, cd, z) ? z : z - 1;
    z = (int)dnn;
    if (fabs(dn - dnn) > 4e-3 || z < 0 || z >= g.Nz) lo = (int)ceil(dn);
    else lo = crosses(g, L, cd, z) ? z : z + 1;
    lo = max(lo, 0);
    hi = min(hi, g.Nz - 1);
    return true;
}

constexpr int kVoxWarps = 8;

// One warp per column with candidates (the words of the others are zero
// already), one lane per candidate.  Lane w holds the parity of points 32 w ..
// 32 w + 31 and 32 (w + 32) .. (Nz <= 2048).
__global__ void __launch_bounds__(kVoxWarps * 32)
k_columns(VoxGrid g, double inv_s, const double* __restrict__ tris, const int64_t* __restrict__ colstart,
          const int32_t* __restrict__ pairs, const int32_t* __restrict__ global_list, int32_t nglobal,
          uint32_t* __restrict__ fluid) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t col = blockIdx.x * (int64_t)kVoxWarps + w;
    const int64_t ncol = (int64_t)g.Nx * g.Ny;
    if (col >= ncol) return;
    const int64_t c0 = colstart[col], c1 = colstart[col + 1];
    const int64_t total = (c1 - c0) + nglobal;
    if (total == 0) return;
    const int i = (int)(col / g.Ny), j = (int)(col % g.Ny);
    double sx, sy;
    column_xy(g, i, j, sx, sy);
    const double L = g.bb[5] - g.bb[4];
    uint32_t p0 = 0, p1 = 0;
    for (int64_t cb = 0; cb < total; cb += 32) {
        const int64_t idx = cb + lane;
        Cand cd = {0.0, 0.0, 0.0, 0.0};
        bool keep = idx < total;
        if (keep) {
            const bool listed = idx < (c1 - c0);       // passed the xy test when it was listed
            const int32_t t = listed ? pairs[c0 + idx] : global_list[idx - (c1 - c0)];
            const double* T = tris + 12 * (int64_t)t;
            keep = listed || inside2d(sx, sy, T);
            if (keep) {
                const double dxv = sx - sx, dyv = sy - sy;
                cd.c = (T[0] - sx) * T[9] + (T[1] - sy) * T[10];
                cd.qz = T[2];
                cd.nz = T[11];
                cd.d0 = dxv * T[9] + dyv * T[10];
            }
        }
        int lo = 0, hi = -1;
        const bool ranged = !keep || cross_range(g, inv_s, L, cd, lo, hi);
        const unsigned every = __ballot_sync(0xffffffffu, !ranged);
        unsigned live = __ballot_sync(0xffffffffu, ranged && lo <= hi);
        while (live) {
            const int src = __ffs(live) - 1;
            live &= live - 1;
            const int l = __shfl_sync(0xffffffffu, lo, src), h = __shfl_sync(0xffffffffu, hi, src);
            auto mask = [&](int b) -> uint32_t {       // points of [l, h] among b .. b + 31
                const int x = max(l - b, 0), y = min(h - b, 31);
                return x > y ? 0u : (0xffffffffu << x) & (0xffffffffu >> (31 - y));
            };
            p0 ^= mask(32 * lane);
            p1 ^= mask(32 * (lane + 32));
        }
        for (unsigned m = every; m; m &= m - 1) {      // every point: the exact test, lanes over z
            const int src = __ffs(m) - 1;
            Cand d;
            d.c = __shfl_sync(0xffffffffu, cd.c, src);
            d.qz = __shfl_sync(0xffffffffu, cd.qz, src);
            d.nz = __shfl_sync(0xffffffffu, cd.nz, src);
            d.d0 = __shfl_sync(0xffffffffu, cd.d0, src);
            for (int b = 0; b < (g.Nz + 31) / 32; ++b) {
                const int z = 32 * b + lane;
                const uint32_t word = __ballot_sync(0xffffffffu, z < g.Nz && crosses(g, L, d, z));
                if (lane == (b & 31)) { if (b < 32) p0 ^= word; else p1 ^= word; }
            }
        }
    }
    // (no candidate counts a point from Nz on, so the bits past the column are 0)
    const int W = words_for(g.Nz);
    uint32_t* out = fluid + col * W;
    if (lane < W) out[lane] = p0;
    if (lane + 32 < W) out[lane + 32] = p1;
}

// Boundary points, ComplexGeometry.cpp:509-556: fluid with a neighbour of the 26
// that is not (outside the grid counts as not fluid, which makes the points on its
// faces boundary points), one word a thread.
__global__ void k_boundary(VoxGrid g, const uint32_t* __restrict__ fluid, uint32_t* __restrict__ isb) {
    const int W = words_for(g.Nz);
    const int64_t n = (int64_t)g.Nx * g.Ny * W;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t f = fluid[p];
        uint32_t r = 0;
        if (f) {
            const int w = (int)(p % W);
            const int64_t ij = p / W;
            const int j = (int)(ij % g.Ny), i = (int)(ij / g.Ny);
            uint32_t all = f;                        // points whose neighbours are all fluid
            if (i == 0 || i == g.Nx - 1 || j == 0 || j == g.Ny - 1) all = 0u;
            for (int dx = -1; dx <= 1 && all; ++dx)
                for (int dy = -1; dy <= 1; ++dy) {
                    const uint32_t* c = fluid + ((int64_t)(i + dx) * g.Ny + (j + dy)) * W + w;
                    const uint32_t m = c[0], lo = w > 0 ? c[-1] : 0u, hi = w + 1 < W ? c[1] : 0u;
                    all &= m & ((m << 1) | (lo >> 31)) & ((m >> 1) | (hi << 31));
                }
            r = f & ~all;
        }
        isb[p] = r;
    }
}

// x-major grid indices of the set bits, in order
__global__ void k_bit_points(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ prefix, int64_t n, int W, int Nz,
                             int64_t* __restrict__ out) {
    for_each_bit(bits, prefix, n, [&](int64_t wi, uint32_t, int bit, uint32_t set, uint32_t rank) {
        if (set) out[rank] = (wi / W) * Nz + (wi % W) * 32 + bit;
    });
}

// bytes of grid points [first, first + n)
__global__ void k_bit_bytes(const uint32_t* __restrict__ bits, int64_t first, int64_t n, int W, int Nz, uint8_t* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = point_bit(bits, first + i, W, Nz);
}

struct DevPred {
    int32_t list_id, axis;
    double plane_hi, plane_lo, tol;
    double lo[3], hi[3];
};

// getInOutBP predicates, |p - plane| <= tol with plane = hi + lo (double-double).
__global__ void k_predicates(VoxGrid g, const int64_t* __restrict__ bidx, int64_t nb, const DevPred* __restrict__ preds,
                             int np, uint64_t* __restrict__ mask) {
    for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = bidx[b];
        const int k = (int)(p % g.Nz);
        const int64_t ij = p / g.Nz;
        const int j = (int)(ij % g.Ny), i = (int)(ij / g.Ny);
        const double c[3] = {g.bb[0] + (double)i * g.spacing, g.bb[2] + (double)j * g.spacing,
                             g.bb[4] + (double)k * g.spacing};
        uint64_t m = 0;
        for (int q = 0; q < np; ++q) {
            const DevPred& P = preds[q];
            const double d = (c[P.axis] - P.plane_hi) - P.plane_lo;
            bool ok = fabs(d) <= P.tol;
            for (int a = 0; a < 3 && ok; ++a) {
                if (a == P.axis) continue;
                if (!isnan(P.lo[a]) && !(P.lo[a] < c[a])) ok = false;
                if (!isnan(P.hi[a]) && !(c[a] < P.hi[a])) ok = false;
            }
            if (ok) m |= 1ull << P.list_id;
        }
        mask[b] = m;
    }
}

__global__ void k_list_flag(const uint64_t* __restrict__ mask, int64_t nb, int list, uint8_t* __restrict__ fl) {
    for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x)
        fl[b] = list >= 0 ? (uint8_t)((mask[b] >> list) & 1) : (uint8_t)(mask[b] == 0);
}

// list sizes in one pass: points in no list to out[0], points of list l to out[1 + l]
__global__ void k_list_sizes(const uint64_t* __restrict__ mask, int64_t nb, int nl, unsigned long long* __restrict__ out) {
    __shared__ unsigned int cnt[65];
    for (int l = threadIdx.x; l < 65; l += blockDim.x) cnt[l] = 0u;
    __syncthreads();
    for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x) {
        uint64_t m = mask[b];
        if (m == 0u) atomicAdd(&cnt[0], 1u);
        for (; m; m &= m - 1) atomicAdd(&cnt[__ffsll((long long)m)], 1u);
    }
    __syncthreads();
    for (int l = threadIdx.x; l <= nl; l += blockDim.x)
        if (cnt[l]) atomicAdd(out + l, (unsigned long long)cnt[l]);
}

__global__ void k_gather_i64(const int64_t* __restrict__ src, const int64_t* __restrict__ idx, int64_t n,
                             int64_t* __restrict__ out) {
    for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < n; b += (int64_t)gridDim.x * blockDim.x)
        out[b] = src[idx[b]];
}

}  // namespace lbm

// ---------------------------------------------------------------------------
// host side

struct lbm_geometry {
    lbm::VoxGrid grid;
    int dev = 0;
    uint32_t* d_fluid = nullptr;       // fluid points, one bit each: words_for(Nz) words per column (x, y)
    int64_t* d_bidx = nullptr;         // boundary point grid indices
    uint64_t* d_bmask = nullptr;       // predicate mask per boundary point
    int64_t n_fluid = 0, n_boundary = 0;
    std::vector<int64_t> list_sizes;   // per list id (64)
    int64_t n_wall = 0;
    int32_t n_lists = 0;
    double vox_ms = 0, cls_ms = 0;
};

namespace lbm {

static int g_blocks_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b > 152LL * 64) b = 152LL * 64;
    if (b < 1) b = 1;
    return (int)b;
}

// Device buffer that frees itself, from the device's stream-ordered pool
// (dev_alloc): allocated and freed in the order of the stream that uses it.
template <class T>
struct DBuf {
    T* p = nullptr;
    cudaStream_t s = 0;
    ~DBuf() { if (p) dev_free(p, s); }
    lbm_status alloc(size_t n, const char* what, cudaStream_t st) {
        s = st;
        return dev_alloc(reinterpret_cast<void**>(&p), sizeof(T) * (n ? n : 1), st, what);
    }
    void adopt(T* q, cudaStream_t st) { p = q; s = st; }
    T* release() { T* q = p; p = nullptr; return q; }
};

}  // namespace lbm

using namespace lbm;

#define LBM_TRY(x)                      \
    do {                                \
        lbm_status s_ = (x);            \
        if (s_ != LBM_OK) return s_;    \
    } while (0)

static lbm_status geometry_build(lbm_geometry* G, const lbm_tri* tris, size_t ntris, double spacing,
                                 const lbm_grid* grid, const lbm_bc_predicate* preds, size_t npreds, cudaStream_t st) {
    VoxGrid& g = G->grid;
    g.spacing = spacing;
    if (grid) {
        for (int a = 0; a < 3; ++a) {
            if (grid->dims[a] < 1) return fail(LBM_ERR_ARG, "grid dims must be >= 1");
            g.bb[2 * a] = grid->min[a];
            g.bb[2 * a + 1] = grid->min[a] + (grid->dims[a] - 1) * spacing;
        }
        g.Nx = grid->dims[0]; g.Ny = grid->dims[1]; g.Nz = grid->dims[2];
    } else {
        if (ntris == 0) return fail(LBM_ERR_ARG, "tight grid needs at least one triangle");
        double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (size_t t = 0; t < ntris; ++t) {
            const double* T = &tris[t].x1;
            for (int a = 0; a < 3; ++a) {
                mn[a] = std::min(mn[a], std::min(T[a], std::min(T[3 + a], T[6 + a])));
                mx[a] = std::max(mx[a], std::max(T[a], std::max(T[3 + a], T[6 + a])));
            }
        }
        int d[3];
        for (int a = 0; a < 3; ++a) {
            g.bb[2 * a] = mn[a]; g.bb[2 * a + 1] = mx[a];
            double n = std::ceil((mx[a] - mn[a]) / spacing);
            if (!(n >= 0 && n < 1e6)) return fail(LBM_ERR_ARG, "grid extent on axis %d is not finite or too large", a);
            d[a] = (int)n + 1;
        }
        g.Nx = d[0]; g.Ny = d[1]; g.Nz = d[2];
    }
    if (g.Nz > 2048) return fail(LBM_ERR_ARG, "Nz = %d exceeds the voxelizer's 2048-point column limit", g.Nz);
    const int64_t ncol = (int64_t)g.Nx * g.Ny;
    for (size_t p = 0; p < npreds; ++p) {
        if (preds[p].list_id < 0 || preds[p].list_id > 63 || preds[p].axis < 0 || preds[p].axis > 2)
            return fail(LBM_ERR_ARG, "predicate %zu: list id must be 0..63 and axis 0..2", p);
    }
    if (ntris >= (size_t)INT32_MAX) return fail(LBM_ERR_ARG, "too many triangles");

    cudaEvent_t e0, e1, e2;
    LBM_CUDA(cudaEventCreate(&e0));
    LBM_CUDA(cudaEventCreate(&e1));
    LBM_CUDA(cudaEventCreate(&e2));

    DBuf<double> d_tris;
    LBM_TRY(d_tris.alloc(ntris * 12, "triangles", st));
    if (ntris) LBM_CUDA(cudaMemcpyAsync(d_tris.p, tris, sizeof(double) * 12 * ntris, cudaMemcpyHostToDevice, st));
    DBuf<int32_t> colcount, cursor, glist, nglob;
    DBuf<int64_t> colstart;
    DBuf<uint32_t> fluid;
    LBM_TRY(colcount.alloc(ncol, "column counts", st));
    LBM_TRY(cursor.alloc(ncol, "column cursors", st));
    LBM_TRY(colstart.alloc(ncol + 1, "column offsets", st));
    LBM_TRY(glist.alloc(ntris, "global triangle list", st));
    LBM_TRY(nglob.alloc(1, "global count", st));
    const int W = words_for(g.Nz);
    const int64_t nwords = ncol * W;
    LBM_TRY(fluid.alloc(nwords, "node-type field", st));
    LBM_CUDA(cudaEventRecord(e0, st));
    LBM_CUDA(cudaMemsetAsync(colcount.p, 0, sizeof(int32_t) * ncol, st));
    LBM_CUDA(cudaMemsetAsync(cursor.p, 0, sizeof(int32_t) * ncol, st));
    LBM_CUDA(cudaMemsetAsync(nglob.p, 0, sizeof(int32_t), st));
    const int TB = 128;
    const double inv_s = 1.0 / spacing;
    LBM_CUDA(cudaMemsetAsync(fluid.p, 0, sizeof(uint32_t) * nwords, st));
    if (ntris) k_tri_count<<<(unsigned)((ntris + TB - 1) / TB), TB, 0, st>>>(g, inv_s, d_tris.p, (int64_t)ntris, colcount.p, glist.p, nglob.p);
    int64_t npairs = 0;
    LBM_TRY(scan::exclusive_scan(colcount.p, ncol, colstart.p, &npairs, st));
    LBM_CUDA(cudaMemcpyAsync(colstart.p + ncol, &npairs, sizeof(int64_t), cudaMemcpyHostToDevice, st));
    int32_t nglobal = 0;
    LBM_CUDA(cudaMemcpyAsync(&nglobal, nglob.p, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    DBuf<int32_t> pairs;
    LBM_TRY(pairs.alloc(npairs, "column candidate lists", st));
    if (ntris) k_tri_fill<<<(unsigned)((ntris + TB - 1) / TB), TB, 0, st>>>(g, inv_s, d_tris.p, (int64_t)ntris, colstart.p, cursor.p, pairs.p);
    LBM_CUDA(cudaStreamSynchronize(st));
    k_columns<<<(unsigned)((ncol + kVoxWarps - 1) / kVoxWarps), kVoxWarps * 32, 0, st>>>(
        g, inv_s, d_tris.p, colstart.p, pairs.p, glist.p, nglobal, fluid.p);
    LBM_CUDA(cudaGetLastError());
    LBM_CUDA(cudaEventRecord(e1, st));

    // boundary points and predicate lists
    DBuf<uint32_t> isb, rank;
    LBM_TRY(isb.alloc(nwords, "boundary points", st));
    LBM_TRY(rank.alloc(nwords, "boundary ranks", st));
    k_boundary<<<g_blocks_for(nwords, 256), 256, 0, st>>>(g, fluid.p, isb.p);
    LBM_TRY(scan::bit_ranks(fluid.p, nwords, nullptr, &G->n_fluid, st));
    LBM_TRY(scan::bit_ranks(isb.p, nwords, rank.p, &G->n_boundary, st));
    int64_t* bidx = nullptr;
    if (G->n_boundary <= (int64_t)UINT32_MAX) {
        LBM_TRY(dev_alloc(reinterpret_cast<void**>(&bidx), sizeof(int64_t) * std::max<int64_t>(G->n_boundary, 1), st, "boundary points"));
        k_bit_points<<<g_blocks_for(nwords, 256), 256, 0, st>>>(isb.p, rank.p, nwords, W, g.Nz, bidx);
    } else {
        // the ranks are 32-bit: beyond them one byte a point and the 64-bit compaction
        const int64_t npts = ncol * g.Nz;
        DBuf<uint8_t> bytes;
        LBM_TRY(bytes.alloc(npts, "boundary flags", st));
        k_bit_bytes<<<g_blocks_for(npts, 256), 256, 0, st>>>(isb.p, 0, npts, W, g.Nz, bytes.p);
        LBM_TRY(scan::compact(bytes.p, npts, &bidx, &G->n_boundary, st));
    }
    G->d_bidx = bidx;
    DBuf<uint64_t> bmask;
    LBM_TRY(bmask.alloc(G->n_boundary, "boundary masks", st));
    std::vector<DevPred> hp(npreds);
    int32_t nl = 0;
    for (size_t p = 0; p < npreds; ++p) {
        hp[p] = {preds[p].list_id, preds[p].axis, preds[p].plane_hi, preds[p].plane_lo, preds[p].tol,
                 {preds[p].lo[0], preds[p].lo[1], preds[p].lo[2]}, {preds[p].hi[0], preds[p].hi[1], preds[p].hi[2]}};
        nl = std::max(nl, preds[p].list_id + 1);
    }
    DBuf<DevPred> dpred;
    LBM_TRY(dpred.alloc(npreds, "predicates", st));
    if (npreds) LBM_CUDA(cudaMemcpyAsync(dpred.p, hp.data(), sizeof(DevPred) * npreds, cudaMemcpyHostToDevice, st));
    if (G->n_boundary)
        k_predicates<<<g_blocks_for(G->n_boundary, 256), 256, 0, st>>>(g, bidx, G->n_boundary, dpred.p, (int)npreds, bmask.p);
    LBM_CUDA(cudaGetLastError());
    LBM_CUDA(cudaEventRecord(e2, st));
    G->d_bmask = bmask.release();
    G->d_fluid = fluid.release();
    G->n_lists = nl;
    G->list_sizes.assign(64, 0);
    {
        DBuf<unsigned long long> cnt;
        LBM_TRY(cnt.alloc(65, "list sizes", st));
        LBM_CUDA(cudaMemsetAsync(cnt.p, 0, 65 * sizeof(unsigned long long), st));
        if (G->n_boundary)
            k_list_sizes<<<std::min(g_blocks_for(G->n_boundary, 256), 152 * 4), 256, 0, st>>>(G->d_bmask, G->n_boundary, nl, cnt.p);
        unsigned long long h[65];
        LBM_CUDA(cudaMemcpyAsync(h, cnt.p, sizeof h, cudaMemcpyDeviceToHost, st));
        LBM_CUDA(cudaStreamSynchronize(st));
        G->n_wall = (int64_t)h[0];
        for (int l = 0; l < nl; ++l) G->list_sizes[l] = (int64_t)h[1 + l];
    }
    float ms1 = 0, ms2 = 0;
    cudaEventElapsedTime(&ms1, e0, e1);
    cudaEventElapsedTime(&ms2, e1, e2);
    G->vox_ms = ms1;
    G->cls_ms = ms2;
    cudaEventDestroy(e0); cudaEventDestroy(e1); cudaEventDestroy(e2);
    return LBM_OK;
}

extern "C" {

lbm_status lbm_geometry_create(const lbm_tri* tris, size_t ntris, double spacing, const lbm_grid* grid,
                               const lbm_bc_predicate* preds, size_t npreds, void* stream, lbm_geometry** out) {
    const NvtxRange nvtx_range("lbm_geometry_create");
    if (!out || (!tris && ntris) || (!preds && npreds) || !(spacing > 0))
        return fail(LBM_ERR_ARG, "lbm_geometry_create: bad argument");
    clear_error();
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(LBM_ERR_NODEV, "no CUDA device");
    lbm_geometry* G = new lbm_geometry();
    cudaGetDevice(&G->dev);
    lbm_status s = guarded("lbm_geometry_create",
                           [&] { return geometry_build(G, tris, ntris, spacing, grid, preds, npreds, (cudaStream_t)stream); });
    if (s != LBM_OK) { lbm_geometry_destroy(G); return s; }
    *out = G;
    return LBM_OK;
}

lbm_status lbm_predicates_pv2013(lbm_bc_predicate* out, size_t cap, size_t* n) {
    // ComplexGeometry.cpp:587-633; plane constants are long double literals,
    // represented here as double-double (hi + lo).
    struct P { int list, axis; long double plane; double lo[3], hi[3]; };
    const double N = NAN;
    const P tab[7] = {
        {0, 1, -175.275L, {-9.9, N, -129.979}, {-3.3, N, -124.799}},
        {1, 1, -164.075L, {N, N, N}, {N, N, N}},
        {2, 1, -174.475L, {-5.4, N, -101.379}, {-5, N, -100.979}},
        {3, 0, -28.3L, {N, -179.975, -97.2794}, {N, -178.875, -96.2794}},
        {4, 0, -25.5L, {N, -180.675, -100.779}, {N, -179.875, -100.379}},
        {5, 0, -37.0L, {N, N, N}, {N, N, N}},
        {6, 2, -108.379L, {-29.7, -196.375, N}, {-28.1, -194.575, N}},
    };
    if (!n) return fail(LBM_ERR_ARG, "lbm_predicates_pv2013: null n");
    *n = 7;
    if (!out) return LBM_OK;
    if (cap < 7) return fail(LBM_ERR_ARG, "lbm_predicates_pv2013: capacity %zu < 7", cap);
    for (int i = 0; i < 7; ++i) {
        lbm_bc_predicate& p = out[i];
        p.list_id = tab[i].list;
        p.axis = tab[i].axis;
        p.plane_hi = (double)tab[i].plane;
        p.plane_lo = (double)(tab[i].plane - (long double)p.plane_hi);
        p.tol = 1e-2;
        for (int a = 0; a < 3; ++a) { p.lo[a] = tab[i].lo[a]; p.hi[a] = tab[i].hi[a]; }
    }
    return LBM_OK;
}

lbm_status lbm_geometry_info_get(const lbm_geometry* G, lbm_geometry_info* info) {
    if (!G || !info) return fail(LBM_ERR_ARG, "lbm_geometry_info_get: null argument");
    std::memset(info, 0, sizeof *info);
    info->dims[0] = G->grid.Nx; info->dims[1] = G->grid.Ny; info->dims[2] = G->grid.Nz;
    for (int a = 0; a < 6; ++a) info->bbox[a] = G->grid.bb[a];
    info->spacing = G->grid.spacing;
    info->n_points = (int64_t)G->grid.Nx * G->grid.Ny * G->grid.Nz;
    info->n_fluid = G->n_fluid;
    info->n_boundary = G->n_boundary;
    info->n_wall = G->n_wall;
    for (int l = 0; l < 64; ++l) info->list_size[l] = G->list_sizes.empty() ? 0 : G->list_sizes[l];
    info->n_lists = G->n_lists;
    info->voxelize_ms = G->vox_ms;
    info->classify_ms = G->cls_ms;
    return LBM_OK;
}

lbm_status lbm_geometry_flags(const lbm_geometry* G, uint8_t* host_out, size_t cap) {
    if (!G || !host_out) return fail(LBM_ERR_ARG, "lbm_geometry_flags: null argument");
    clear_error();
    size_t n = (size_t)G->grid.Nx * G->grid.Ny * G->grid.Nz;
    if (cap < n) return fail(LBM_ERR_ARG, "lbm_geometry_flags: capacity %zu < %zu", cap, n);
    const int Nz = G->grid.Nz, W = words_for(Nz);
    // bits to bytes through a scratch of at most 32 MB
    const size_t block = std::min<size_t>(n, size_t(32) << 20);
    cudaStream_t st = 0;
    DBuf<uint8_t> bytes;
    if (bytes.alloc(block, "node-type bytes", st) != LBM_OK) {
        // no room for it: whole columns of bits to the host, about 1 MB at a time
        clear_error();
        const int64_t ncol = (int64_t)G->grid.Nx * G->grid.Ny, step = std::max(1, (1 << 18) / W);
        return guarded("lbm_geometry_flags", [&]() -> lbm_status {
            std::vector<uint32_t> words((size_t)(std::min(step, ncol) * W));
            for (int64_t c = 0; c < ncol; c += step) {
                const int64_t m = std::min(step, ncol - c);
                LBM_CUDA(cudaMemcpy(words.data(), G->d_fluid + c * W, sizeof(uint32_t) * m * W, cudaMemcpyDeviceToHost));
                for (int64_t p = 0; p < m * Nz; ++p) host_out[c * Nz + p] = point_bit(words.data(), p, W, Nz);
            }
            return LBM_OK;
        });
    }
    // (launched by a call that returns its own status: an error that someone else's
    // launch left unread is not this call's)
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    for (size_t at = 0; at < n; at += block) {
        const size_t m = std::min(block, n - at);
        cfg.gridDim = dim3((unsigned)g_blocks_for((int64_t)m, 256));
        LBM_CUDA(cudaLaunchKernelEx(&cfg, k_bit_bytes, (const uint32_t*)G->d_fluid, (int64_t)at, (int64_t)m, W, Nz, bytes.p));
        LBM_CUDA(cudaMemcpy(host_out + at, bytes.p, m, cudaMemcpyDeviceToHost));
    }
    return LBM_OK;
}

lbm_status lbm_geometry_list(const lbm_geometry* G, int32_t list, int64_t* host_out, size_t cap, size_t* n) {
    if (!G || !n || list < -2 || list > 63) return fail(LBM_ERR_ARG, "lbm_geometry_list: bad argument");
    clear_error();
    int64_t cnt = list == LBM_LIST_BOUNDARY ? G->n_boundary : (list == LBM_LIST_WALL ? G->n_wall : G->list_sizes[list]);
    *n = (size_t)cnt;
    if (!host_out) return LBM_OK;
    if (cap < (size_t)cnt) return fail(LBM_ERR_ARG, "lbm_geometry_list: capacity %zu < %lld", cap, (long long)cnt);
    if (cnt == 0) return LBM_OK;
    if (list == LBM_LIST_BOUNDARY) {
        LBM_CUDA(cudaMemcpy(host_out, G->d_bidx, sizeof(int64_t) * cnt, cudaMemcpyDeviceToHost));
        return LBM_OK;
    }
    cudaStream_t st = 0;
    DBuf<uint8_t> fl;
    LBM_TRY(fl.alloc(G->n_boundary, "list flags", st));
    k_list_flag<<<g_blocks_for(G->n_boundary, 256), 256, 0, st>>>(G->d_bmask, G->n_boundary,
                                                                  list == LBM_LIST_WALL ? -1 : list, fl.p);
    int64_t* pos = nullptr;
    int64_t c = 0;
    LBM_TRY(scan::compact(fl.p, G->n_boundary, &pos, &c, st));
    DBuf<int64_t> posb; posb.adopt(pos, st);
    DBuf<int64_t> vals;
    LBM_TRY(vals.alloc(c, "list values", st));
    k_gather_i64<<<g_blocks_for(c, 256), 256, 0, st>>>(G->d_bidx, pos, c, vals.p);
    LBM_CUDA(cudaMemcpy(host_out, vals.p, sizeof(int64_t) * c, cudaMemcpyDeviceToHost));
    return LBM_OK;
}

void lbm_geometry_destroy(lbm_geometry* G) {
    if (!G) return;
    cudaDeviceSynchronize();               // pool memory is freed without an implicit wait
    if (G->d_fluid) cudaFree(G->d_fluid);
    if (G->d_bidx) cudaFree(G->d_bidx);
    if (G->d_bmask) cudaFree(G->d_bmask);
    delete G;
}

}  // extern "C"

// accessors for the lattice builder (sim.cu)
namespace lbm {
const uint32_t* geometry_fluid_dev(const lbm_geometry* g) { return g->d_fluid; }
const int64_t* geometry_bidx_dev(const lbm_geometry* g) { return g->d_bidx; }
const uint64_t* geometry_bmask_dev(const lbm_geometry* g) { return g->d_bmask; }
int64_t geometry_nboundary(const lbm_geometry* g) { return g->n_boundary; }
int64_t geometry_nfluid(const lbm_geometry* g) { return g->n_fluid; }
void geometry_dims(const lbm_geometry* g, int dims[3]) { dims[0] = g->grid.Nx; dims[1] = g->grid.Ny; dims[2] = g->grid.Nz; }
int geometry_device(const lbm_geometry* g) { return g->dev; }
const std::vector<int64_t>& geometry_list_sizes(const lbm_geometry* g) { return g->list_sizes; }
}  // namespace lbm
