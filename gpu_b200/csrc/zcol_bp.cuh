// zcol_bp.cuh -- a voxel column's in-plane setup for the z-column
// backprojectors: the detector columns that cross it and their alpha
// intervals, and the constants of its candidate-row bounds.
#pragma once

#include "zcol.cuh"

namespace ctr {

constexpr int ZC_RUN = 4;                  // detector columns of the run kept with the column
constexpr float ZC_ROW_EPS = 1.0f / 32.0f; // margin of the alpha-range row estimate, in rows

// The alpha interval inside voxel column (xlo..xhi, ylo..yhi) of the rays of
// one detector column (its table entry ct): the projector's own alphas.
__device__ __forceinline__ float2 col_interval(const float4& ct, float xlo, float xhi, float ylo, float yhi)
{
    const float ax0 = fm(fs(xlo, ct.x), ct.y), ax1 = fm(fs(xhi, ct.x), ct.y);
    const float ay0 = fm(fs(ylo, ct.z), ct.w), ay1 = fm(fs(yhi, ct.z), ct.w);
    return make_float2(fmaxf(fminf(ax0, ax1), fminf(ay0, ay1)), fminf(fmaxf(ax0, ax1), fmaxf(ay0, ay1)));
}

struct __align__(16) VoxCol {
    float2 r[ZC_RUN];        // the run's alpha intervals ([1, 0] beyond it)
    int ua, nrun;            // first detector column of the run and its length (0: nothing to do)
    float mlo, mhi;          // height z is seen at rows between z + m (z - zs), m = mlo, mhi
    float row_lo, row_hi;    // row offsets of those bounds, margins included
    int ulo, uhi;            // candidate columns of the corner projections
};

// One thread's setup of voxel column (i, j) at view `view` (the x and y part
// of the reference's bounding rectangle, V63/kernel_IterativeRecon_
// universal.cu:639-706, and the run of detector columns whose rays cross the
// column).  The rows of a voxel are those whose ray meets the cell at some
// alpha of the run's range: the row centred at x1z, seen from a source at
// height zs, is at height z at alpha where x1z = z + m (z - zs),
// m = alpha / (1 - alpha), so the rows lie between the lower plane's least
// and the upper plane's largest value over the range's two ends (both are
// monotone in alpha), widened by ZC_ROW_EPS rows for the float rounding
// (below 1e-3 rows).  Without a usable range (parallel rays, or a range that
// touches the detector or the source) the corners' magnifications bound the
// rows, to the nearest row: half a row of margin.
__device__ __forceinline__ VoxCol vox_col(const DevGeom& g, int i, int j, int view, bool live)
{
    VoxCol o;
    const int ic = min(i, g.M - 1), jc = min(j, g.N - 1);
    live = live && i < g.M && j < g.N;
    const float xlo = __ldg(g.px + ic + 1), xhi = __ldg(g.px + ic + 2);
    const float ylo = __ldg(g.py + jc + 1), yhi = __ldg(g.py + jc + 2);
    const float cx = fa(fa(g.bx, fm(g.vx, 0.5f)), fm((float)ic, g.vx));   // :592-594
    const float cy = fa(fa(g.by, fm(g.vy, 0.5f)), fm((float)jc, g.vy));
    const float2 sc = g.trig[view];
    const float s = sc.x, c = sc.y;
    float umin = __int_as_float(0x7f800000), umax = -umin, mlo = umin, mhi = -umin;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        const float pxc = fs(fa(cx, fm((float)(cc & 1), g.vx)), fm(0.5f, g.vx));
        const float pyc = fs(fa(cy, fm((float)(cc >> 1), g.vy)), fm(0.5f, g.vy));
        const float t = fa(fm(pxc, c), fm(pyc, s));
        const float ss = fa(fm(-pxc, s), fm(pyc, c));
        const float mt = g.ct_style == 2 ? 0.0f : fdv(fs(t, g.dod), fs(g.dso, t));   // :655-670
        const float ou = fa(fm(mt, fs(ss, g.srcy)), ss);
        umin = fminf(umin, ou); umax = fmaxf(umax, ou);
        mlo = fminf(mlo, mt); mhi = fmaxf(mhi, mt);
    }
    if (g.ct_style == 1 || g.ct_style == 2) { mlo = 0.0f; mhi = 0.0f; }   // rays parallel to the xy plane
    int ulo = __float2int_rd(fa(fm(fs(umin, g.ymin), g.inv_du), 0.5f));
    int uhi = __float2int_rd(fa(fm(fs(umax, g.ymin), g.inv_du), 0.5f));
    if ((ulo < 0 && uhi < 0) || (ulo > g.R - 1 && uhi > g.R - 1)) live = false;
    ulo = max(ulo, 0);
    uhi = min(uhi, g.R - 1);
    if (!live) { ulo = 1; uhi = 0; }
    const float4* __restrict__ colt = g.colt + (long long)view * g.R;
    int ua = uhi + 1, ub = ulo - 1;
    float amin = 1.0f, bmax = 0.0f;
    for (int uu = ulo; uu <= uhi; ++uu) {
        const float2 a = col_interval(__ldg(colt + uu), xlo, xhi, ylo, yhi);
        if (a.y > a.x) {
            ua = min(ua, uu);
            ub = uu;
            amin = fminf(amin, a.x);
            bmax = fmaxf(bmax, a.y);
        }
    }
    o.ulo = ulo;
    o.uhi = uhi;
    o.ua = ua;
    o.nrun = max(ub - ua + 1, 0);
    float off = 0.5f;
    if ((g.ct_style == 0 || g.ct_style == 3) && o.nrun > 0 && amin > 0.0f && bmax < 1.0f) {
        mlo = __fdividef(amin, fs(1.0f, amin));
        mhi = __fdividef(bmax, fs(1.0f, bmax));
        off = ZC_ROW_EPS;
    }
    o.mlo = mlo;
    o.mhi = mhi;
    const float zrow0 = -fm(g.zmin, g.inv_dv);
    o.row_lo = fs(zrow0, off);
    o.row_hi = fa(zrow0, off);
#pragma unroll
    for (int q = 0; q < ZC_RUN; ++q)
        o.r[q] = q < o.nrun ? col_interval(__ldg(colt + ua + q), xlo, xhi, ylo, yhi) : make_float2(1.0f, 0.0f);
    return o;
}

}  // namespace ctr
