// zcol_fp.cuh -- Siddon projector on a z-column volume (the kernel template;
// zcol_<type>.cu hold the instances, zcol.cu the launcher).
//
// The in-plane crossings of a ray -- the alphas of its x and y planes, merged
// in order, and the voxel column between each two -- depend on the view and
// the detector column only.  A block takes a few detector columns; for each it
// builds that merged list once in shared memory, every plane placing itself
// by counting the other axis's planes before it (an estimate from its
// position, settled by comparing the projector's own float alphas; planes of
// both axes at the same alpha share one entry, as the traversal moves both
// axes at once).  Then each lane walks the list for one detector row: per
// entry one shared-memory broadcast, the segment, one voxel and the sums, plus
// the z plane crossings of that row, which are few for a cone of a few
// degrees.  The lanes of a warp read neighbouring voxels of one z-column.
// The list says where a ray goes next, so the z crossings and the voxel loads
// run ZF_AHEAD entries ahead of the sums: an entry's slot holds its voxel, and
// for a row that crosses a z plane in it the crossing's alpha and the voxel
// behind it.
//
// The traversal, the alphas and the order and rounding of every sum are the
// general projector's (fp_kernels.cuh), so are the results, bit for bit.  A
// ray that enters through a z face starts at the entry of the list that holds
// its start voxel; one whose start voxel the list does not hold, or whose
// first crossing does not lie after its entry (the start rules' rounding), is
// walked by the general projector (zf_general).
//
// Bound by issue (80 % of the slots, 446 M instructions a view of 512^3 and
// 1024 x 768 rays): a step takes about 27 instructions, a third of them for the
// z crossing that any of a warp's rows may make; the general kernel takes about
// 40 (three plane alphas re-evaluated each step).  In the cone beam the two
// halves of a warp take rows mirrored about the middle row: mirrored rays cross
// z planes at the same steps.  Per view, copy included, over 32 views at 35 to 46
// degrees: FP32 0.59 ms (general kernel on the linear volume 0.84 ms), BF16 0.59
// (0.92), fused sums 0.54 and 0.55 (0.83 and 0.92).
#pragma once

#include "fp_kernels.cuh"
#include "zcol.cuh"

namespace ctr {

static constexpr int ZF_WARPS = 8;
static constexpr int ZF_AHEAD = 4;   // entries whose voxels are in flight

// Shared memory of a block: the lists of wc detector columns (cap entries
// each), the tie bits of their y planes, the z planes.
__host__ __device__ __forceinline__ int zf_cap(const DevGeom& g) { return (g.M + g.N + 5) & ~1; }   // even: entries are read in pairs
__host__ __device__ __forceinline__ int zf_words(const DevGeom& g) { return (g.N + 2 + 31) / 32; }
__host__ __device__ __forceinline__ size_t zf_smem(const DevGeom& g, int wc)
{
    return (size_t)wc * ((size_t)zf_cap(g) * sizeof(float2) + (size_t)zf_words(g) * 2 * sizeof(unsigned) + 8) +
           sizeof(float) * (size_t)(g.Z + 8);
}

// Elements between z-columns: whole 32-byte sectors.
__host__ __device__ __forceinline__ int zcol_stride(const DevGeom& g, size_t es)
{
    const int q = 32 / (int)es;
    return (g.Z + q - 1) / q * q;
}
constexpr size_t ZF_SMEM = 50 * 1024;   // of a block: four to an SM
// Detector columns of a block: 4 (with 2 groups of 32 rows) while their lists fit
// -- neighbouring columns cross the same voxel columns, and two warps share the
// building of a list --, 2 with longer lists.  One column a block (above 3,060 x
// and y planes) was never the faster path: 1600^2 x 64 voxels, 64 to 512 rows,
// 125 to 14 ms against 27 to 13 ms.
__host__ __forceinline__ int zf_columns(const DevGeom& g) { return zf_smem(g, 4) <= ZF_SMEM ? 4 : 2; }

// The in-plane crossings of one detector column, in traversal order.
struct Axis2 {
    const float* planes;   // g.px / g.py
    float x1, inv, d, b, inv_v;
    int v0, p0, s, n;      // start voxel, first plane, direction, crossings until the volume's last plane
    __device__ __forceinline__ float alpha(int t) const   // alpha of crossing t
    {
        return fm(fs(__ldg(planes + 1 + p0 + s * t), x1), inv);
    }
    // crossings with alpha < a
    __device__ __forceinline__ int before(float a) const
    {
        if (n == 0) return 0;
        const float pos = (a * d + x1 - b) * inv_v;          // plane position, an estimate
        float e = s > 0 ? pos - (float)p0 : (float)p0 - pos;
        int t = __float2int_ru(fminf(fmaxf(e, 0.0f), (float)n));
        while (t > 0 && alpha(t - 1) >= a) --t;
        while (t < n && alpha(t) < a) ++t;
        return t;
    }
};

// The general projector, on the linear volume.
template <typename VT, bool FAST>
__device__ __noinline__ void zf_general(const DevGeom& g, const float* PZ, const float* PINF, const VT* lin, float s,
                                        float c, int u, int v, float& sum, float& len)
{
    const RayResult r = siddon<VT, false, false, true, false, 0, false, false, FAST>(g, g.px, g.py, PZ, PINF, lin, s, c, u, v);
    sum = r.sum;
    len = r.len;
}

// One row's walk.
template <typename VT> struct ZRay {
    const VT* p;          // the voxel of its z index in z-column 0
    float d12, ac, az, x1z, iz, alim, amin;
    float sum, len;
    const float* zn;      // &plane after the current one, for z index vk: advanced with vk
    int sz, n0;
    bool live;            // walked here and not finished
};

template <typename VT, bool FAST>
__global__ void __launch_bounds__(32 * ZF_WARPS, 4)
k_forward_zcol(const __grid_constant__ DevGeom g, const VT* __restrict__ vol, int zs, const VT* __restrict__ lin, int view0,
               void* __restrict__ out, int out_dt, int wc)
{
    extern __shared__ __align__(16) unsigned char zf_raw[];
    const int cap = zf_cap(g), words = zf_words(g);
    float2* const lists = reinterpret_cast<float2*>(zf_raw);
    unsigned* const ties = reinterpret_cast<unsigned*>(lists + (size_t)wc * cap);   // [wc][2][words]: bits, prefix
    int* const counts = reinterpret_cast<int*>(ties + (size_t)wc * 2 * words);      // [wc][2]: entries, any tie
    float* const PZ = reinterpret_cast<float*>(counts + 2 * wc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wr = ZF_WARPS / wc;                    // row groups of the block
    const int cl = warp / wr, rg = warp - cl * wr;   // this warp's column of the block and row group
    const int u = centre_out(blockIdx.x, gridDim.x) * wc + cl;
    const int w = blockIdx.z, view = view0 + w;
    const float2 sc = g.trig[view];
    const float s = sc.x, c = sc.y;
    for (int t = threadIdx.x; t < g.Z + 3; t += blockDim.x) PZ[t] = __ldg(g.pz + t);
    if (threadIdx.x == 0) PZ[g.Z + 7] = __int_as_float(0x7f800000);
    for (int t = threadIdx.x; t < wc * 2 * words; t += blockDim.x) ties[t] = 0u;
    if (threadIdx.x < 2 * wc) counts[threadIdx.x] = 0;
    __syncthreads();

    // ---- the column's list
    float2* const list = lists + (size_t)cl * cap;
    unsigned* const tie = ties + (size_t)cl * 2 * words;
    const bool col = u < g.R;
    bool base_ok = false;
    float amin_b = 0.0f;
    Axis2 X{}, Y{};
    if (col) {
        const RayEnds e = ray_ends(g, s, c, u, 0);   // the in-plane part does not depend on the row
        const float dx = fs(e.x2x, e.x1x), dy = fs(e.x2y, e.x1y);
        const float ix = fdv(1.0f, dx), iy = fdv(1.0f, dy);
        const AxisSpan sx = axis_span(__ldg(g.px + 1), __ldg(g.px + g.M + 1), e.x1x, ix);
        const AxisSpan sy = axis_span(__ldg(g.py + 1), __ldg(g.py + g.N + 1), e.x1y, iy);
        amin_b = fmaxf(sx.lo, sy.lo);
        const bool hit = !(fminf(sx.hi, sy.hi) <= amin_b);
        const bool px = fabsf(fs(e.x1x, e.x2x)) < fm(g.vx, 1e-6f), py = fabsf(fs(e.x1y, e.x2y)) < fm(g.vy, 1e-6f);
        const AxisStart ax = axis_start(amin_b, sx.lo, e.x1x, e.x2x, dx, g.bx, g.inv_vx, g.M);
        const AxisStart ay = axis_start(amin_b, sy.lo, e.x1y, e.x2y, dy, g.by, g.inv_vy, g.N);
        if (hit && (unsigned)ax.v < (unsigned)g.M && (unsigned)ay.v < (unsigned)g.N) {
            X = Axis2{g.px, e.x1x, ix, dx, g.bx, g.inv_vx, ax.v, ax.plane, e.x1x < e.x2x ? 1 : -1, 0};
            Y = Axis2{g.py, e.x1y, iy, dy, g.by, g.inv_vy, ay.v, ay.plane, e.x1y < e.x2y ? 1 : -1, 0};
            if (!px) X.n = X.s > 0 ? g.M - ax.v : ax.v + 1;
            if (!py) Y.n = Y.s > 0 ? g.N - ay.v : ay.v + 1;
            // the first crossings lie after the entry; a list with no crossing cannot end
            base_ok = (X.n + Y.n > 0) && (X.n == 0 || X.alpha(0) > amin_b) && (Y.n == 0 || Y.alpha(0) > amin_b);
        }
    }
    // every list ends where the ray leaves the volume in the plane
    float aend = __int_as_float(0x7f800000);
    const int step = 32 * wr, first = rg * 32 + lane;
    // the entries; with `tied`, shifted by the tied y planes before them
    auto fill = [&](bool tied) {
        auto before = [&](int t) { return tied ? (int)(tie[words + (t >> 5)] + __popc(tie[t >> 5] & ((1u << (t & 31)) - 1u))) : 0; };
        int last = 0;
        bool seen = false;
        for (int t = first; t < X.n; t += step) {
            const float a = X.alpha(t);
            if (a > aend) break;
            const int q = Y.before(a), pos = t + q - before(q);
            seen |= q < Y.n && Y.alpha(q) == a;
            list[pos] = make_float2(a, __int_as_float(((Y.v0 + Y.s * q) * g.M + X.v0 + X.s * t) * zs));
            last = max(last, pos + 1);
        }
        for (int t = first; t < Y.n; t += step) {
            const float a = Y.alpha(t);
            if (a > aend) break;
            if (tied && ((tie[t >> 5] >> (t & 31)) & 1u)) continue;
            const int q = X.before(a), pos = t + q - before(t);
            list[pos] = make_float2(a, __int_as_float(((Y.v0 + Y.s * t) * g.M + X.v0 + X.s * q) * zs));
            last = max(last, pos + 1);
        }
        if (last) atomicMax(&counts[2 * cl], last);
        if (!tied && seen) counts[2 * cl + 1] = 1;
    };
    if (base_ok) {
        if (X.n) aend = fminf(aend, X.alpha(X.n - 1));
        if (Y.n) aend = fminf(aend, Y.alpha(Y.n - 1));
        fill(false);
    }
    __syncthreads();
    bool any = false;
    for (int t = 0; t < wc; ++t) any |= counts[2 * t + 1] != 0;
    if (any) {   // some column of the block has x and y planes at one alpha: its list again
        const bool mine = base_ok && counts[2 * cl + 1] != 0;
        if (mine)
            for (int t = first; t < Y.n; t += step) {
                const float a = Y.alpha(t);
                const int q = X.before(a);
                if (q < X.n && X.alpha(q) == a) atomicOr(tie + (t >> 5), 1u << (t & 31));
            }
        __syncthreads();
        if (mine && rg == 0) {   // ties before each word
            if (lane == 0) counts[2 * cl] = 0;
            unsigned run = 0;
            for (int t = 0; t < words; t += 32) {
                const unsigned n = t + lane < words ? __popc(tie[t + lane]) : 0u;
                unsigned inc = n;
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned up = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += up;
                }
                if (t + lane < words) tie[words + t + lane] = run + inc - n;
                run += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        __syncthreads();
        if (mine) fill(true);
        __syncthreads();
    }
    if (!col) return;
    const int cnt = counts[2 * cl];

    // ---- the row
    ZRay<VT> r;
    bool general = false, ran = false;   // walked by the general projector / here
    int v = -1, ne = cnt;                // the row; the first entry that finishes the ray
    if (g.ct_style == 0) {               // rows t and ZP-1-t in the two halves of the warp
        const int t = (blockIdx.y * wr + rg) * 16 + (lane & 15);
        if (t < (g.ZP + 1) / 2) {
            const int m = g.ZP - 1 - t;
            v = lane < 16 ? t : (m != t ? m : -1);
        }
    } else {
        const int t = (blockIdx.y * wr + rg) * 32 + lane;
        v = t < g.ZP ? t : -1;
    }
    r.sum = r.len = 0.0f;
    r.live = false;
    r.p = vol; r.sz = 0; r.zn = PZ; r.n0 = 0;
    r.d12 = 0.0f; r.x1z = 0.0f; r.iz = 0.0f; r.amin = r.ac = 0.0f;
    r.az = __int_as_float(0x7f800000);
    r.alim = 0.0f;
    if (v >= 0) {
        const RayInit in = ray_init(g, s, c, u, v);
        r.d12 = ray_d12(in.e);
        if (ray_starts(g, in)) {
            const int off = (in.sy.v * g.M + in.sx.v) * zs;
            int n0 = 0;
            bool ok = base_ok && in.ax > in.amin && in.ay > in.amin && in.az > in.amin;
            if (ok && in.amin != amin_b) {   // entered through a z face: the list entry of its start voxel
                int lo = 0, hi = cnt;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (list[mid].x > in.amin) hi = mid;
                    else lo = mid + 1;
                }
                n0 = lo;
            }
            ok = ok && n0 < cnt && __float_as_int(list[n0].y) == off;
            // alpha at which the ray is finished: the last plane of an axis, or where
            // the loop test fails -- the smallest float a with !(amax - a > eps)
            const int sz = (in.pz || in.e.x1z == in.e.x2z) ? 0 : (in.e.x1z < in.e.x2z ? 1 : -1);
            float t = in.amax;
            if (!g.fast_exit) {
                ok = ok && in.amax > 1e-3f;
                t = fs(in.amax, g.loop_eps);
                if (ok) {
                    for (int it = 0; it < 8 && !(fs(in.amax, t) > g.loop_eps); ++it) t = __int_as_float(__float_as_int(t) - 1);
                    for (int it = 0; it < 16 && fs(in.amax, t) > g.loop_eps; ++it) t = __int_as_float(__float_as_int(t) + 1);
                    ok = !(fs(in.amax, t) > g.loop_eps) &&
                         (fs(in.amax, __int_as_float(__float_as_int(t) - 1)) > g.loop_eps);
                }
            }
            r.alim = t;
            if (sz) r.alim = fminf(r.alim, fm(fs(sz > 0 ? PZ[g.Z + 1] : PZ[1], in.e.x1z), in.iz));
            r.alim = fminf(r.alim, aend);
            // At most one z crossing an entry: an entry is no longer than the shorter
            // in-plane step.  2^-20 for the rounding of the four alphas (below 4 x 2^-24
            // each: the plane's subtraction, 1/d and the product, alphas below 1), 0.1 %
            // for that of the planes' positions.
            ok = ok && fminf(g.vx * fabsf(in.ix), g.vy * fabsf(in.iy)) * 1.001f + 9.5367432e-7f < g.vz * fabsf(in.iz);
            if (ok) {
                r.live = ran = true;
                r.n0 = n0;
                r.amin = r.ac = in.amin;
                r.az = in.az;
                r.x1z = in.e.x1z;
                r.iz = in.iz;
                r.sz = sz;
                r.p = vol + in.sz.v;
                // next plane after a move to z index k: k + 1 when increasing, k when decreasing
                r.zn = PZ + 1 + in.sz.v + (sz > 0);
                int lo = n0, hi = cnt;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (list[mid].x >= r.alim) hi = mid;
                    else lo = mid + 1;
                }
                ne = lo;
            } else {
                general = true;
            }
        }
    }
    // The segment [ac, a] of the ray in a voxel of value f.  The length serves the
    // zero rule (a ray shorter than 1e-6 vz) alone: it is not summed over the
    // entries every ray passes, which hold two planes of one axis, a voxel apart.
    auto segment = [&](float a, float f, bool length) {
        const float da = fs(a, r.ac);
        if (FAST) {
            r.sum = __fmaf_rn(da, f, r.sum);
        } else {
            const float seg = fm(r.d12, da);
            if (length) r.len = fa(r.len, seg);
            r.sum = fa(r.sum, fm(seg, f));
        }
        r.ac = a;
    };
    auto ld1 = [&](int off) { return Store<VT>::ld(r.p + off); };
    auto move_z = [&]() {
        r.p += r.sz;
        r.zn += r.sz;
        r.az = fm(fs(*r.zn, r.x1z), r.iz);
    };
    // a step that may start, finish or sit out the ray
    auto careful = [&](int n, float a, int off) {
        if (!r.live || n < r.n0) return;
        while (r.az < a) {
            segment(r.az, ld1(off), true);
            if (!(r.ac < r.alim)) { r.live = false; return; }
            move_z();
        }
        segment(a, ld1(off), true);
        if (!(r.ac < r.alim)) r.live = false;
        else if (r.az == a) move_z();   // both axes at once
    };
    if (__any_sync(0xffffffffu, r.live)) {
        // the first entry of any ray, and the entries [hot0, hot1) that every ray
        // of the warp passes without starting or finishing
        int n = __reduce_min_sync(0xffffffffu, r.live ? r.n0 : cnt);
        const int hot0 = __reduce_max_sync(0xffffffffu, r.live ? r.n0 : 0);
        const int hot1 = __reduce_min_sync(0xffffffffu, r.live ? ne : cnt);
        for (; n < hot0; ++n) {
            const float2 en = list[n];
            careful(n, en.x, __float_as_int(en.y));
        }
        if ((n & 1) && n < hot1) {   // the entries below are read in pairs
            const float2 en = list[n];
            careful(n, en.x, __float_as_int(en.y));
            ++n;
        }
        // a lane without work (not live) walks along on voxel 0 of each z-column;
        // its sums are not used
        if (n + ZF_AHEAD <= hot1) {
            // A slot: the entry's end, the row's next z crossing (inside the entry, at
            // its end, or later), the voxel before the crossing and the one behind it.
            float sa[ZF_AHEAD], sz[ZF_AHEAD], va[ZF_AHEAD], vb[ZF_AHEAD];
            auto fetch = [&](int j, float a, int off) {
                sa[j] = a;
                sz[j] = r.az;
                va[j] = ld1(off);
                if (r.az <= a) {   // (at the end: both axes move at once, no segment behind it)
                    move_z();
                    vb[j] = ld1(off);
                }
            };
            auto fetch2 = [&](int j, int m) {
                const float4 en = *reinterpret_cast<const float4*>(list + m);
                fetch(j, en.x, __float_as_int(en.y));
                fetch(j + 1, en.z, __float_as_int(en.w));
            };
            auto consume = [&](int j) {
                float f = va[j];
                if (sz[j] < sa[j]) {
                    segment(sz[j], f, false);
                    f = vb[j];
                }
                segment(sa[j], f, false);
            };
#pragma unroll
            for (int j = 0; j < ZF_AHEAD; j += 2) fetch2(j, n + j);
            for (; n + 2 * ZF_AHEAD <= hot1; n += ZF_AHEAD) {
#pragma unroll
                for (int j = 0; j < ZF_AHEAD; j += 2) {
                    consume(j);
                    consume(j + 1);
                    fetch2(j, n + ZF_AHEAD + j);
                }
            }
#pragma unroll
            for (int j = 0; j < ZF_AHEAD; ++j) consume(j);
            n += ZF_AHEAD;
            r.len = fmaxf(r.len, g.thr_fp);
        }
        for (; n < cnt; ++n) {
            if (!__any_sync(0xffffffffu, r.live)) break;
            const float2 en = list[n];
            careful(n, en.x, __float_as_int(en.y));
        }
    }

    if (v < 0) return;
    float sum = 0.0f, len = 0.0f;
    if (ran) {
        sum = FAST ? fm(r.sum, r.d12) : r.sum;
        len = FAST ? fm(r.d12, fs(r.ac, r.amin)) : r.len;
    }
    if (general) zf_general<VT, FAST>(g, PZ, PZ + g.Z + 7, lin, s, c, u, v, sum, len);
    st_any(out, ((long long)w * g.ZP + v) * g.R + u, out_dt, len < g.thr_fp ? 0.0f : sum);   // :554
}

// Views [view0, view0 + nview) of the z-column volume vol (lin: the same, linear).
template <typename VT>
cudaError_t launch_zcol_t(const Geometry& G, const void* vol, const void* lin, int view0, int nview, void* out, ctr_dtype out_dt,
                          cudaStream_t st)
{
    const DevGeom& g = G.dg;
    const int zs = zcol_stride(g, sizeof(VT));
    const int wc = zf_columns(g);
    const void* fn = g.fast_sums ? reinterpret_cast<const void*>(&k_forward_zcol<VT, true>)
                                 : reinterpret_cast<const void*>(&k_forward_zcol<VT, false>);
    // one limit for every geometry: the attribute belongs to the function
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ZF_SMEM);
    if (e != cudaSuccess) return e;
    const int per = 32 * (ZF_WARPS / wc);
    const dim3 grid((g.R + wc - 1) / wc, ((g.ct_style == 0 ? 2 * ((g.ZP + 1) / 2) : g.ZP) + per - 1) / per, nview);
    if (g.fast_sums)
        k_forward_zcol<VT, true><<<grid, 32 * ZF_WARPS, zf_smem(g, wc), st>>>(g, (const VT*)vol, zs, (const VT*)lin, view0, out,
                                                                                    out_dt, wc);
    else
        k_forward_zcol<VT, false><<<grid, 32 * ZF_WARPS, zf_smem(g, wc), st>>>(g, (const VT*)vol, zs, (const VT*)lin, view0, out,
                                                                                    out_dt, wc);
    return cudaGetLastError();
}

cudaError_t launch_zcol_f32(const Geometry& G, const void* vol, const void* lin, int view0, int nview, void* out, ctr_dtype out_dt, cudaStream_t st);
cudaError_t launch_zcol_bf16(const Geometry& G, const void* vol, const void* lin, int view0, int nview, void* out, ctr_dtype out_dt, cudaStream_t st);
cudaError_t launch_zcol_f16(const Geometry& G, const void* vol, const void* lin, int view0, int nview, void* out, ctr_dtype out_dt, cudaStream_t st);

}  // namespace ctr
