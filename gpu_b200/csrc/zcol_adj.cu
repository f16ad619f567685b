// zcol_adj.cu -- the matched adjoint (ctr_backproject) as a z-column gather.
//
// A warp owns 32 voxels of each of 8x4 z-columns and keeps their FP64 sums in
// shared memory over a batch of views.  Per view each lane works out one
// column's in-plane setup (vox_col); then the warp goes through its columns
// with a lane per voxel: candidate rows, the two z alphas of a (voxel, row)
// pair, and per detector column of the run one 8-byte record, the overlap
// of two alpha intervals, and one FP64 multiply-add.  Chord = d12 x overlap in
// the projector's own float alphas, so every (voxel, ray) chord is the
// projector's Siddon segment bit for bit.
//
// That holds for a regular ray: one whose traversal starts in the voxel that
// contains its entry point geometrically, so that the traversal visits
// exactly the voxels with a positive overlap.  The reference's start rules
// can miss it by one voxel when the entry lies within float rounding of a
// voxel edge, or for rays nearly parallel to an axis.  Such irregular rays
// (a few in 1e4; at an axis-aligned view often whole rows and columns, whose
// entries all lie on one plane) get a record of length 0 and set their row
// group's bit in their detector column's mark; the warps whose voxel columns see
// a marked detector column then visit those rays, a lane per column, with the
// traversal's own cell intervals (AdjIrr).  Every sum has a fixed order.
//
// Bound by issue and load latency (60 % of the issue slots): a row's records are
// loaded a row ahead.  The form it replaces, which tested every candidate pair
// against the traversal record in 32 bytes, takes 0.60 ms a view of 256^3 voxels
// and 384^2 rays, records included; this one 0.13 ms (0.15 with 16-byte records
// and no load ahead).
#include "fp_kernels.cuh"
#include "zcol_bp.cuh"

namespace ctr {

// A ray's record: the detector value, and its length source - pixel; 0: no
// chord; -0: an irregular ray, its traversal in the AdjIrr array.
struct __align__(8) AdjRec {
    float y, d12;
};
// An irregular ray: its length, the alphas it covers, its start voxel; the top
// bit of i, j, k: parallel to the axis.  With the record 32 bytes a ray, as
// k_adjoint's AdjRay, so that both kernels work on batches of the same views in
// the same workspace.
struct __align__(8) AdjIrr {
    float d12, a_lo, a_hi;
    int i, j, k;
};
static_assert(sizeof(AdjRec) + sizeof(AdjIrr) == sizeof(AdjRay), "one workspace for both adjoints");
__device__ __forceinline__ bool irregular(const AdjRec& r) { return __float_as_uint(r.d12) == 0x80000000u; }

// A detector column's mark: bit b for irregular rays among rows [b << s, (b + 1) << s), s = mark_shift.
typedef unsigned long long AdjMark;
__host__ __device__ __forceinline__ int mark_shift(const DevGeom& g)
{
    int s = 0;
    while (((g.ZP - 1) >> s) > 63) ++s;
    return s;
}
__device__ __forceinline__ AdjMark mark_range(int vlo, int vhi, int s)   // the bits of rows vlo..vhi
{
    return (~0ull << (vlo >> s)) & (~0ull >> (63 - (vhi >> s)));
}

static __device__ __noinline__ float traversal_end(const DevGeom& g, float s, float c, int u, int v)
{
    const float INF = __int_as_float(0x7f800000);
    return siddon<float, false, false, false>(g, g.px, g.py, g.pz, &INF, nullptr, s, c, u, v).a_hi;
}

// Records of views [view0, view0 + gridDim.z), [view][u][v].  A block of 32
// columns x 8 rows; the records leave through shared memory so that the
// transposed store is coalesced.
static constexpr int AP_ROWS = 32, AP_COLS = 8;
__global__ void __launch_bounds__(AP_ROWS * AP_COLS)
k_adj_prep(const __grid_constant__ DevGeom g, const float* __restrict__ y, int view0, AdjRec* __restrict__ recs,
           AdjIrr* __restrict__ full, AdjMark* __restrict__ marks, int ms)
{
    __shared__ float yt[AP_COLS][AP_ROWS + 1];
    const int w = blockIdx.z, u0 = blockIdx.x * AP_COLS, v0 = blockIdx.y * AP_ROWS;
    const long long P = (long long)g.R * g.ZP;
    {   // the values, read along the detector rows
        const int cu = threadIdx.x % AP_COLS, rv = threadIdx.x / AP_COLS;
        if (u0 + cu < g.R && v0 + rv < g.ZP) yt[cu][rv] = y[w * P + (long long)(v0 + rv) * g.R + u0 + cu];
    }
    __syncthreads();
    const int rv = threadIdx.x % AP_ROWS, cu = threadIdx.x / AP_ROWS;
    const int u = u0 + cu, v = v0 + rv;
    if (u >= g.R || v >= g.ZP) return;
    const float2 sc = g.trig[view0 + w];
    const RayInit r = ray_init(g, sc.x, sc.y, u, v);
    AdjRec rec;
    rec.y = yt[cu][rv];
    rec.d12 = 0.0f;
    if (r.hit) {
        // regular: the start voxel holds the entry (its entry planes at or
        // before amin, its exit planes at or after), and a parallel axis
        // keeps the voxel the column and row tables encode
        auto ok = [&](bool par, const float* planes, const AxisStart& st, float x1, float x2, float inv, float next,
                      float b, float inv_v) {
            if (par) return st.v == (int)floorf(fm(fs(x1, b), inv_v));
            const float back = fm(fs(__ldg(planes + 1 + st.v + (x1 < x2 ? 0 : 1)), x1), inv);
            return back <= r.amin && next >= r.amin;
        };
        const bool in = ((unsigned)r.sx.v < (unsigned)g.M) && ((unsigned)r.sy.v < (unsigned)g.N) &&
                        ((unsigned)r.sz.v < (unsigned)g.Z);
        const bool reg = in && ray_starts(g, r) &&
                         ok(r.px, g.px, r.sx, r.e.x1x, r.e.x2x, r.ix, r.ax, g.bx, g.inv_vx) &&
                         ok(r.py, g.py, r.sy, r.e.x1y, r.e.x2y, r.iy, r.ay, g.by, g.inv_vy) &&
                         ok(r.pz, g.pz, r.sz, r.e.x1z, r.e.x2z, r.iz, r.az, g.bz, g.inv_vz);
        if (reg) {
            rec.d12 = ray_d12(r.e);
        } else if (ray_starts(g, r)) {
            // The traversal ends at the first plane alpha not below the exit, which is
            // the exit itself -- the last plane of an axis the ray crosses -- unless a
            // face the ray runs parallel to set it: such a ray is traversed (a view
            // with one such ray waits for it, 0.1 ms at 96^3).
            float a_hi = r.amax;
            if (r.amax != r.a_last) a_hi = traversal_end(g, sc.x, sc.y, u, v);
            auto axis = [&](int n, bool par) { return n | (par ? (int)0x80000000 : 0); };
            full[w * P + (long long)u * g.ZP + v] =
                AdjIrr{ray_d12(r.e), r.amin, a_hi, axis(r.sx.v, r.px), axis(r.sy.v, r.py), axis(r.sz.v, r.pz)};
            rec.d12 = -0.0f;
            atomicOr(marks + (long long)w * g.R + u, 1ull << (v >> ms));
        }
    }
    recs[w * P + (long long)u * g.ZP + v] = rec;
}

static constexpr int AC_X = 8, AC_Y = 4, AC_N = AC_X * AC_Y;   // z-columns of a warp
static constexpr int AC_WARPS = 4;                             // warps (z chunks of 32) of a block, at most

// The chord of an irregular ray in voxel (i, j, k) over the traversal's own
// cells: the start cell opens at -inf, cells behind the start are never
// visited, a parallel axis keeps its start cell.
__device__ __forceinline__ bool irregular_cell(int n, int n0, bool par, float a0, float a1, float dir, float& lo,
                                               float& hi)
{
    const float INF = __int_as_float(0x7f800000);
    lo = -INF;
    hi = INF;
    if (par) return n == n0;
    const int d = n - n0;
    if ((dir > 0.f && d < 0) || (dir < 0.f && d > 0)) return false;
    if (d != 0) lo = fminf(a0, a1);
    hi = fmaxf(a0, a1);
    return true;
}

struct AdjWarp {
    double acc[AC_N][33];    // [column][z], padded
    VoxCol col[AC_N];
};

// The magnifications of a voxel column's corners (the reference's rectangle): an
// irregular ray's rows, to the nearest row.
__device__ __forceinline__ float2 corner_mags(const DevGeom& g, int i, int j, int view)
{
    const float2 sc = g.trig[view];
    const float cx = fa(fa(g.bx, fm(g.vx, 0.5f)), fm((float)i, g.vx));
    const float cy = fa(fa(g.by, fm(g.vy, 0.5f)), fm((float)j, g.vy));
    float mlo = __int_as_float(0x7f800000), mhi = -mlo;
    for (int q = 0; q < 4; ++q) {
        const float px = fs(fa(cx, fm((float)(q & 1), g.vx)), fm(0.5f, g.vx));
        const float py = fs(fa(cy, fm((float)(q >> 1), g.vy)), fm(0.5f, g.vy));
        const float t = fa(fm(px, sc.y), fm(py, sc.x));
        const float mt = g.ct_style == 2 ? 0.0f : fdv(fs(t, g.dod), fs(g.dso, t));
        mlo = fminf(mlo, mt);
        mhi = fmaxf(mhi, mt);
    }
    return g.ct_style != 0 ? make_float2(0.0f, 0.0f) : make_float2(mlo, mhi);
}

// The irregular rays that cross voxels kb .. kb + nk - 1 of the lane's voxel
// column, into their sums acc[k - kb].  Called by the whole warp: every lane
// finds its column's next ray, then those that have one work together.
static __device__ __noinline__ void irregular_columns(const DevGeom& g, bool live, const VoxCol& cc, double* acc, int i, int j,
                                                      int kb, int nk, int view, const AdjRec* __restrict__ rw,
                                                      const AdjIrr* __restrict__ fw, const AdjMark* __restrict__ marks,
                                                      int ms)
{
    const float4* __restrict__ colt = g.colt + (long long)view * g.R;
    float xlo = 0.f, xhi = 0.f, ylo = 0.f, yhi = 0.f;
    int vlo = 0, vhi = -1;
    if (live) {
        xlo = __ldg(g.px + i + 1); xhi = __ldg(g.px + i + 2);
        ylo = __ldg(g.py + j + 1); yhi = __ldg(g.py + j + 2);
        // candidate rows of the voxels together, to the nearest row
        const float2 m = corner_mags(g, i, j, view);
        const float z0 = __ldg(g.pz + kb + 1), z1 = __ldg(g.pz + kb + nk + 1);
        const float zl = fs(z0, g.srcz), zh = fs(z1, g.srcz);
        const float zmn = fminf(fa(fm(m.x, zl), z0), fa(fm(m.y, zl), z0));
        const float zmx = fmaxf(fa(fm(m.x, zh), z1), fa(fm(m.y, zh), z1));
        vlo = max(__float2int_rd(fa(fm(fs(zmn, g.zmin), g.inv_dv), 0.5f)), 0);
        vhi = min(__float2int_rd(fa(fm(fs(zmx, g.zmin), g.inv_dv), 0.5f)), g.ZP - 1);
        live = vlo <= vhi;
    }
    const AdjMark range = live ? mark_range(vlo, vhi, ms) : 0;
    int uu = cc.ulo - 1, vv = 1, vend = 0;   // detector column; its rows of the current group left
    AdjMark mark = 0;                        // its groups left
    for (;;) {
        bool found = false;
        AdjRec rec;
        while (live && !found) {
            if (vv <= vend) {
                rec = rw[(long long)uu * g.ZP + vv];
                found = irregular(rec);
                ++vv;
            } else if (mark) {
                const int g0 = (__ffsll(mark) - 1) << ms;
                mark &= mark - 1;
                vv = max(vlo, g0);
                vend = min(vhi, g0 + (1 << ms) - 1);
            } else if (uu < cc.uhi) {
                mark = __ldg(marks + ++uu) & range;
            } else {
                live = false;
            }
        }
        if (!__any_sync(0xffffffffu, found)) break;
        if (found) {
            const int v = vv - 1;
            const AdjIrr ray = fw[(long long)uu * g.ZP + v];
            const float2 rt = g.rowt[v];
            const float4 ct = __ldg(colt + uu);
            const float ax0 = fm(fs(xlo, ct.x), ct.y), ax1 = fm(fs(xhi, ct.x), ct.y);
            const float ay0 = fm(fs(ylo, ct.z), ct.w), ay1 = fm(fs(yhi, ct.z), ct.w);
            const int ri = ray.i & 0x7fffffff, rj = ray.j & 0x7fffffff, rk = ray.k & 0x7fffffff;
            float xl, xh, yl, yh;
            if (irregular_cell(i, ri, ray.i < 0, ax0, ax1, ct.y, xl, xh) &&
                irregular_cell(j, rj, ray.j < 0, ay0, ay1, ct.w, yl, yh)) {
                const float lo = fmaxf(fmaxf(xl, yl), ray.a_lo), hi = fminf(fminf(xh, yh), ray.a_hi);
                // the voxels at the interval's two ends, a voxel of margin; the start voxel is the traversal's own
                const float ka = ((rt.x + lo / rt.y) - g.bz) * g.inv_vz, kz = ((rt.x + hi / rt.y) - g.bz) * g.inv_vz;
                int k0 = __float2int_rd(fminf(ka, kz)) - 1, k1 = __float2int_rd(fmaxf(ka, kz)) + 1;
                const bool start_col = i == ri && j == rj;
                if (start_col) {
                    k0 = min(k0, rk);
                    k1 = max(k1, rk);
                }
                for (int k = max(k0, kb); k <= min(k1, kb + nk - 1); ++k) {
                    const float az0 = fm(fs(__ldg(g.pz + k + 1), rt.x), rt.y), az1 = fm(fs(__ldg(g.pz + k + 2), rt.x), rt.y);
                    float zl, zh;
                    if (!irregular_cell(k, rk, ray.k < 0, az0, az1, rt.y, zl, zh)) continue;
                    const float temp = fm(ray.d12, fs(fminf(hi, zh), fmaxf(lo, zl)));
                    // the traversal's first segment may be a rounding-size negative length
                    if (temp > 0.0f || (start_col && k == rk && ray.a_lo <= ray.a_hi))
                        acc[k - kb] = __fma_rn((double)temp, (double)rec.y, acc[k - kb]);
                }
            }
        }
        __syncwarp();
    }
}

template <typename VT>
__global__ void __launch_bounds__(32 * AC_WARPS, 5)
k_adj_cols(const __grid_constant__ DevGeom g, VT* __restrict__ vol, const AdjRec* __restrict__ recs,
           const AdjIrr* __restrict__ full, const AdjMark* __restrict__ marks, int ms, int view0, int nview,
           int accumulate)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb = (blockIdx.z * (blockDim.x >> 5) + warp) * 32;
    if (kb >= g.Z) return;   // no block-wide step below
    AdjWarp& W = reinterpret_cast<AdjWarp*>(smem_raw)[warp];
    const int i0 = blockIdx.x * AC_X, j0 = blockIdx.y * AC_Y;
    const int k = kb + lane, kc = min(k, g.Z - 1);
    const float z0 = __ldg(g.pz + kc + 1), z1 = __ldg(g.pz + kc + 2);
    const float zs0 = fs(z0, g.srcz), zs1 = fs(z1, g.srcz);
    const int ZP = g.ZP;
    const long long P = (long long)g.R * ZP;
#pragma unroll 4
    for (int q = 0; q < AC_N; ++q) W.acc[q][lane] = 0.0;
    const int ci = i0 + (lane % AC_X), cj = j0 + lane / AC_X;   // this lane's column in the setup
    for (int w = 0; w < nview; ++w) {
        const int view = view0 + w;
        const AdjRec* __restrict__ rw = recs + w * P;
        const AdjMark* __restrict__ mw = marks + (long long)w * g.R;
        __syncwarp();
        bool marked = false;
        {
            const VoxCol c = vox_col(g, ci, cj, view, true);
            W.col[lane] = c;
            for (int uu = c.ulo; uu <= c.uhi; ++uu) marked |= __ldg(mw + uu) != 0;
        }
        const unsigned any_irr = __ballot_sync(0xffffffffu, marked);
        __syncwarp();
        for (int q = 0; q < AC_N; ++q) {
            const VoxCol& c = W.col[q];
            const int nrun = c.nrun;
            if (nrun == 0) continue;
            const float a0 = __fmaf_rn(c.mlo, zs0, z0), a1 = __fmaf_rn(c.mhi, zs0, z0);
            const float b0 = __fmaf_rn(c.mlo, zs1, z1), b1 = __fmaf_rn(c.mhi, zs1, z1);
            const int vlo = min(max(__float2int_ru(__fmaf_rn(fminf(a0, a1), g.inv_dv, c.row_lo)), 0), ZP);
            const int vhi = min(__float2int_rd(__fmaf_rn(fmaxf(b0, b1), g.inv_dv, c.row_hi)), ZP - 1);
            const int nrows = k < g.Z ? max(vhi - vlo + 1, 0) : 0;
            const int wrows = __reduce_max_sync(0xffffffffu, nrows);
            if (wrows == 0) continue;
            double acc = W.acc[q][lane];
            const AdjRec* __restrict__ rc = rw + (long long)c.ua * ZP;
            auto rows = [&](auto nq_c) {
                constexpr int NQ = decltype(nq_c)::value;
                float2 iv[NQ];
#pragma unroll
                for (int t = 0; t < NQ; ++t) iv[t] = c.r[t];
                // a row's records and row constants, loaded one row ahead
                float2 rec[NQ], rt;
                auto load = [&](int r) {
                    const int vv = min(vlo + r, ZP - 1);
                    const float2* __restrict__ pr = reinterpret_cast<const float2*>(rc + vv);
#pragma unroll
                    for (int t = 0; t < NQ; ++t) rec[t] = __ldg(pr + (long long)t * ZP);
                    rt = __ldg(g.rowt + vv);
                };
                load(0);
                for (int r = 0; r < wrows; ++r) {
                    float2 now[NQ];
#pragma unroll
                    for (int t = 0; t < NQ; ++t) now[t] = rec[t];
                    const float az0 = fm(fs(z0, rt.x), rt.y), az1 = fm(fs(z1, rt.x), rt.y);
                    load(r + 1);
                    const float zl = fminf(az0, az1), zh = r < nrows ? fmaxf(az0, az1) : -1.0f;
                    auto pair = [&](const float2& a, const float2& w2) {
                        const float temp = fm(w2.y, fs(fminf(a.y, zh), fmaxf(a.x, zl)));
                        if (temp > 0.0f) acc = __fma_rn((double)temp, (double)w2.x, acc);
                    };
#pragma unroll
                    for (int t = 0; t < NQ; ++t) pair(iv[t], now[t]);
                    if (NQ == ZC_RUN) {   // runs longer than the column keeps
                        const int ii = i0 + (q % AC_X), jj = j0 + q / AC_X;
                        const float2* __restrict__ pr = reinterpret_cast<const float2*>(rc + min(vlo + r, ZP - 1));
                        for (int t = ZC_RUN; t < nrun; ++t)
                            pair(col_interval(__ldg(g.colt + (long long)view * g.R + c.ua + t), __ldg(g.px + ii + 1),
                                              __ldg(g.px + ii + 2), __ldg(g.py + jj + 1), __ldg(g.py + jj + 2)),
                                 __ldg(pr + (long long)t * ZP));
                    }
                }
            };
            if (nrun <= 2) {
                if (nrun == 1) rows(std::integral_constant<int, 1>());
                else rows(std::integral_constant<int, 2>());
            } else if (nrun == 3) {
                rows(std::integral_constant<int, 3>());
            } else {
                rows(std::integral_constant<int, ZC_RUN>());
            }
            W.acc[q][lane] = acc;
        }
        if (any_irr) {   // a lane per column again
            __syncwarp();
            irregular_columns(g, marked, W.col[lane], W.acc[lane], ci, cj, kb, min(32, g.Z - kb), view, rw, full + w * P, mw,
                              ms);
        }
    }
    __syncwarp();
    // the sums leave with a lane per column: 8 voxels of a row side by side
    if (ci < g.M && cj < g.N) {
        const long long MN = (long long)g.M * g.N;
        const int n = min(32, g.Z - kb);
        VT* p = vol + (long long)kb * MN + (long long)cj * g.M + ci;
        for (int t = 0; t < n; ++t, p += MN) {
            const double a = W.acc[lane][t];
            Store<VT>::st(p, (float)(accumulate ? (double)Store<VT>::ldw(p) + a : a));
        }
    }
}

size_t adj_record_bytes(const DevGeom& g, int views)
{
    const size_t n = (size_t)g.R * g.ZP * views;
    return n * (sizeof(AdjRec) + sizeof(AdjIrr)) + (size_t)g.R * views * sizeof(AdjMark);
}

// The gather reproduces the traversal of every scanner whose loop test is one
// comparison (no chord is cut short at the exit) with FP32 entry, the tetrahedron
// beam excepted; the others keep k_adjoint.  Its lanes are voxels of a z-column:
// with few slices they idle, and k_adjoint, whose lanes run along x, is faster.
// k_adjoint / here, ms, 32 views, 512^2 x nz voxels: cone beam (1.5 rows a voxel) nz = 1
// 0.33 / 1.46, 4 1.30 / 1.97, 8 2.49 / 2.08, 16 4.60 / 2.13, 32 9.06 / 2.27; fan beam (1
// row a voxel) nz = 1 0.33 / 1.45, 8 1.72 / 2.29, 16 3.11 / 2.34; parallel beam 8 1.45 /
// 1.91, 16 2.65 / 1.93; the same lines at 192^2 to 1024^2.  (k_adjoint's tables are
// in 48 KB of shared memory; without room for them the gather stays.)
bool adjoint_cols_fits(const Geometry& G)
{
    const DevGeom& g = G.dg;
    if (!g.fast_exit || g.entry64 || g.ct_style == 3) return false;
    return g.Z >= (g.ct_style == 0 ? 8 : 12) || !adjoint_tables_fit(g);
}

ctr_status launch_adjoint_cols(const Geometry& G, const float* y, int view0, int nview, void* ws, void* vol,
                               ctr_dtype vdt, bool accumulate, cudaStream_t st)
{
    const DevGeom& g = G.dg;
    if (nview <= 0) return CTR_OK;
    const size_t n = (size_t)g.R * g.ZP * nview;
    AdjIrr* full = (AdjIrr*)ws;
    AdjRec* recs = (AdjRec*)(full + n);   // 8-byte aligned for any number of rays
    AdjMark* marks = (AdjMark*)(recs + n);
    const int ms = mark_shift(g);
    CTR_CUDA_TRY(cudaMemsetAsync(marks, 0, (size_t)g.R * nview * sizeof(AdjMark), st));
    k_adj_prep<<<dim3((g.R + AP_COLS - 1) / AP_COLS, (g.ZP + AP_ROWS - 1) / AP_ROWS, nview), AP_ROWS * AP_COLS, 0, st>>>(
        g, y, view0, recs, full, marks, ms);
    CTR_CUDA_TRY(cudaGetLastError());
    // no more warps a block than there are z chunks for: an SM's 20 places go to
    // working warps (512^2 x 32, 32 views: 2.27 ms; 5.27 with blocks of 4 warps)
    const int zc = (g.Z + 31) / 32, gz = (zc + AC_WARPS - 1) / AC_WARPS, warps = (zc + gz - 1) / gz;
    const size_t smem = sizeof(AdjWarp) * warps;
    const dim3 grid((g.M + AC_X - 1) / AC_X, (g.N + AC_Y - 1) / AC_Y, gz);
    CTR_DISPATCH_DTYPE(vdt, VT, {
        CTR_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(&k_adj_cols<VT>),
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)(sizeof(AdjWarp) * AC_WARPS)));
        k_adj_cols<VT><<<grid, 32 * warps, smem, st>>>(g, (VT*)vol, recs, full, marks, ms, view0, nview,
                                                      accumulate ? 1 : 0);
    });
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

}  // namespace ctr
