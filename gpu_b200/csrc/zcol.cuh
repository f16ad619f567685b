// zcol.cuh -- device parts shared by the z-column kernels (zcol_fp.cuh,
// zcol_adj.cu).
//
// A z-column is the nz voxels over one (i, j).  For a circular orbit the
// in-plane part of a ray depends only on the view and the detector column, so
// the 32 lanes of a warp take 32 rows of one detector column (projector) or 32
// voxels of one z-column (adjoint): everything in-plane -- which voxel columns a
// ray crosses and at which alphas, which detector columns cross a voxel column
// -- is the same for the whole warp and is worked out once, and the lanes'
// voxels (in a z-fastest copy, for the projector) or ray records lie next to
// each other.
#pragma once

#include "ctr_device.cuh"

namespace ctr {

// floor of the position along an axis at parameter a, as a plane index (the
// projector's pos_floor).
__device__ __forceinline__ float zc_floor(float a, float d, float x1, float b, float inv_v)
{
    return floorf(fm(fs(fa(fm(a, d), x1), b), inv_v));
}

// One axis of a ray: its planes' alphas at the volume's two faces.
struct AxisSpan {
    float lo, hi;
};
__device__ __forceinline__ AxisSpan axis_span(float p0, float p1, float x1, float inv_d)
{
    const float a0 = fm(fs(p0, x1), inv_d), a1 = fm(fs(p1, x1), inv_d);
    return {fminf(a0, a1), fmaxf(a0, a1)};
}

// Start voxel and next plane of one axis at the entry amin (the projector's
// first/last plane index rules, V63/kernel_IterativeRecon_universal.cu:113-284).
struct AxisStart {
    int v;       // voxel index
    int plane;   // index of the next plane crossed
};
__device__ __forceinline__ AxisStart axis_start(float amin, float face, float x1, float x2, float d, float b,
                                                float inv_v, int n)
{
    if (x1 < x2) {
        const int p = (amin == face) ? 1 : __float2int_rz(fa(zc_floor(amin, d, x1, b, inv_v), 1.0f));
        return {p - 1, p};
    }
    const int p = (amin == face) ? n - 1 : __float2int_rz(zc_floor(amin, d, x1, b, inv_v));
    return {p, p};
}

// A ray as the projector starts it (FP32 entry).
struct RayInit {
    RayEnds e;
    float dx, dy, dz, ix, iy, iz;
    float amin, amax;       // entry and exit of the volume
    float a_last;           // exit by the faces of the axes the ray is not parallel to
    bool hit;               // amax > amin
    bool px, py, pz;        // parallel to the axis (the projector keeps its alpha infinite)
    AxisStart sx, sy, sz;   // at amin
    float ax, ay, az;       // alphas of the next planes (infinite when parallel)
};
__device__ __forceinline__ RayInit ray_init(const DevGeom& g, float s, float c, int u, int v)
{
    RayInit r;
    r.e = ray_ends(g, s, c, u, v);
    const RayEnds& e = r.e;
    r.dx = fs(e.x2x, e.x1x); r.dy = fs(e.x2y, e.x1y); r.dz = fs(e.x2z, e.x1z);
    r.ix = fdv(1.0f, r.dx); r.iy = fdv(1.0f, r.dy); r.iz = fdv(1.0f, r.dz);
    const AxisSpan X = axis_span(__ldg(g.px + 1), __ldg(g.px + g.M + 1), e.x1x, r.ix);
    const AxisSpan Y = axis_span(__ldg(g.py + 1), __ldg(g.py + g.N + 1), e.x1y, r.iy);
    const AxisSpan Zs = axis_span(__ldg(g.pz + 1), __ldg(g.pz + g.Z + 1), e.x1z, r.iz);
    r.amin = fmaxf(fmaxf(X.lo, Y.lo), fmaxf(Y.lo, Zs.lo));
    r.amax = fminf(fminf(X.hi, Y.hi), fminf(Y.hi, Zs.hi));
    r.hit = !(r.amax <= r.amin);
    r.px = fabsf(fs(e.x1x, e.x2x)) < fm(g.vx, 1e-6f);
    r.py = fabsf(fs(e.x1y, e.x2y)) < fm(g.vy, 1e-6f);
    r.pz = fabsf(fs(e.x1z, e.x2z)) < fm(g.vz, 1e-6f);
    r.sx = axis_start(r.amin, X.lo, e.x1x, e.x2x, r.dx, g.bx, g.inv_vx, g.M);
    r.sy = axis_start(r.amin, Y.lo, e.x1y, e.x2y, r.dy, g.by, g.inv_vy, g.N);
    if (r.pz && g.zpar_kr) {
        const int f = __float2int_rz(floorf(fm(fs(e.x1z, g.bz), g.inv_vz)));
        r.sz = {f, f};   // never crossed: the plane is not used
    } else {
        r.sz = axis_start(r.amin, Zs.lo, e.x1z, e.x2z, r.dz, g.bz, g.inv_vz, g.Z);
    }
    const float INF = __int_as_float(0x7f800000);
    r.a_last = fminf(fminf(r.px ? INF : X.hi, r.py ? INF : Y.hi), r.pz ? INF : Zs.hi);
    r.ax = r.px ? INF : fm(fs(fa(fm(g.vx, (float)r.sx.plane), g.bx), e.x1x), r.ix);
    r.ay = r.py ? INF : fm(fs(fa(fm(g.vy, (float)r.sy.plane), g.by), e.x1y), r.iy);
    r.az = r.pz ? INF : fm(fs(fa(fm(g.vz, (float)r.sz.plane), g.bz), e.x1z), r.iz);
    return r;
}
// The projector's test before its first step.
__device__ __forceinline__ bool ray_starts(const DevGeom& g, const RayInit& r)
{
    return r.hit && (fs(r.amax, r.amin) > g.loop_eps) && ((unsigned)r.sx.v < (unsigned)g.M) &&
           ((unsigned)r.sy.v < (unsigned)g.N) && ((unsigned)r.sz.v < (unsigned)g.Z);
}

}  // namespace ctr
