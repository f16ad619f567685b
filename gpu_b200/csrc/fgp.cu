// fgp.cu -- FGP total-variation prox, FISTA momentum, objective reductions.
//
// FGP restates FGP_denoise_GPUx7_exact (V63/host_FGP_Denoise_GPUx7.c:1-111)
// and its kernels FGP_operator_L_Pc / FGP_operator_LT_Pp
// (V63/kernel_FGP_Denoise_GPUx7.cu:2-88) with the same float operations.  The
// duals are stored in the volume's storage type; L is FP32.
//
// Dual layout: volume-sized arrays; r[p] belongs to the edge (x, x+1) and is 0
// at x = nx-1 (the reference's zero-padded d_r[x+1], V63/host_FGP_Denoise_
// GPUx7.c:8-38); likewise s along y and t along z.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "ctr_device.cuh"

namespace ctr {

static constexpr int FG_BX = 32, FG_BY = 8;

// f may be stored in another type than the duals (the refinement solver's
// FP32 sum y_k + d against 16-bit duals).
template <typename T, typename TF = T>
__device__ __forceinline__ float fgp_L(const TF* __restrict__ f, const T* __restrict__ r, const T* __restrict__ s,
                                       const T* __restrict__ t, int x, int y, int z, long long p, int M, long long MN,
                                       float lambda)
{
    const float rv = Store<T>::ld(r + p), rm = x > 0 ? Store<T>::ld(r + p - 1) : 0.0f;
    const float sv = Store<T>::ld(s + p), sm = y > 0 ? Store<T>::ld(s + p - M) : 0.0f;
    const float tv = Store<T>::ld(t + p), tm = z > 0 ? Store<T>::ld(t + p - MN) : 0.0f;
    const float tl = fa(fa(fs(rv, rm), fs(sv, sm)), fs(tv, tm));       // L_Pc :14
    return fs(Store<TF>::ld(f + p), fm(lambda, tl));                   // :17
}

// x / d correctly rounded from r = 1/d correctly rounded (Markstein's division;
// Brisebarre, Muller and Raina, IEEE Trans. Computers 53(8), 2004), where the
// remainder cannot underflow and the quotient is finite; the plain division
// elsewhere.  1 <= d.
__device__ __forceinline__ float div_exact(float x, float d, float r)
{
    const float q = fm(x, r);
    const float y = __fmaf_rn(__fmaf_rn(-d, q, x), r, q);
    const float m = fabsf(x);
    return (m > 1e-30f && m < 1e30f && d < 1e30f) ? y : fdv(x, d);
}

// One inner iteration in one pass: L = f - lambda*div(r,s,t) (L_Pc,
// V63/kernel_FGP_Denoise_GPUx7.cu:2-24) and the dual step from L at the voxel
// and its +x, +y, +z neighbours (LT_Pp, :52-86).  A block marches a 32x8 tile
// through a run of z planes; L of the next plane goes to shared memory (never
// to HBM), L of this plane and the duals read for it stay in registers.  Warp
// 8 computes the tile's two edges (the row below and the column to the right)
// while the others update their voxels.  What the next plane reads is loaded
// before the barrier of this one.  Neighbours' duals are read, so the
// new ones go to another set of arrays.
//
// Bound by HBM bandwidth and latency in FP32 (4.3 TB/s of 6.5), by issue and
// latency with 16-bit duals (66 % of the issue slots).  FP32 duals: the extrapolated r_k = o_k + g (o_k - o_(k-1)) is
// formed from the two stored projections with the operations that stored it,
// so r, s, t are never written: f and six arrays in, three out, 40 bytes a
// voxel.  16-bit duals keep r, s, t as stored (their rounding differs from
// one formed from the rounded o): 24 bytes a voxel and f.  The two-pass form (L
// through HBM) moves 72 and 40 bytes.  An iteration: 512^3 FP32 1.25 ms
// (2.15 ms in two passes), 333x257x190 BF16 0.176 ms (0.245 ms).
template <typename T> struct FgpSet {
    static constexpr bool REC = std::is_same<T, float>::value;
    const T* r[3];    // REC: o_k, p_k, q_k;         else r, s, t
    const T* r0[3];   // REC: o_(k-1), ...;          else unused
    T* rn[3];         // REC: o_(k+1), ...;          else the next r, s, t
    T* o[3];          // else: o, p, q, updated in place
};

template <typename T, typename TF, bool FIRST>
__global__ void __launch_bounds__(32 * (FG_BY + 1), 4)
k_fgp_step(int M, int N, int Z, int zrun, const TF* __restrict__ f, const FgpSet<T> d, float lambda, float alpha12,
           float gam, float gam_prev)
{
    constexpr bool REC = FgpSet<T>::REC;
    __shared__ float sL[2][FG_BY + 1][33];   // [plane parity][row][column]
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * FG_BX, y0 = blockIdx.y * FG_BY;
    const int zb = blockIdx.z * zrun, ze = min(Z, zb + zrun);
    const unsigned MN = (unsigned)M * (unsigned)N;   // voxel indices are below 2^31
    // what L at a voxel reads, loaded a plane ahead: f, the voxel's duals, r at
    // x-1 and s at y-1 (REC: o_k in a, o_(k-1) in b)
    struct Raw { float f, a[5], b[5]; };
    auto load = [&](Raw& w, bool on, int x, int y, unsigned p) {
        const unsigned q[5] = {p, p, p, p - 1u, p - (unsigned)M};
        const bool has[5] = {on, on, on, on && x > 0, on && y > 0};
        w.f = on ? Store<TF>::ld(f + p) : 0.0f;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const int a = i < 3 ? i : i - 3;
            w.a[i] = w.b[i] = 0.0f;
            if (!FIRST && has[i]) {
                w.a[i] = Store<T>::ld(d.r[a] + q[i]);
                if (REC) w.b[i] = Store<T>::ld(d.r0[a] + q[i]);
            }
        }
    };
    // the dual a step reads: as stored, or extrapolated from o_k and o_(k-1)
    auto extrap = [&](float o1, float o0) { return REC ? fa(o1, fm(gam_prev, fs(o1, o0))) : o1; };
    // L (L_Pc :14-17); the voxel's duals to rst, t of the plane below in tm
    auto L_of = [&](const Raw& w, float tm, float rst[3]) -> float {
#pragma unroll
        for (int i = 0; i < 3; ++i) rst[i] = extrap(w.a[i], w.b[i]);
        const float tl = fa(fa(fs(rst[0], extrap(w.a[3], w.b[3])), fs(rst[1], extrap(w.a[4], w.b[4]))), fs(rst[2], tm));
        return fs(w.f, fm(lambda, tl));
    };
    auto t_below = [&](bool on, unsigned p) -> float {   // t at (x, y, zb - 1)
        if (FIRST || !on || zb == 0) return 0.0f;
        return extrap(Store<T>::ld(d.r[2] + p - MN), REC ? Store<T>::ld(d.r0[2] + p - MN) : 0.0f);
    };
    if (ty == FG_BY) {   // the edges: row y0+8 (32 columns), then column x0+32 (8 rows)
        const int xe = x0 + tx, ye = y0 + FG_BY, xc = x0 + FG_BX, yc = y0 + tx;
        const bool row = xe < M && ye < N, colm = tx < FG_BY && xc < M && yc < N;
        unsigned pr = (unsigned)zb * MN + (unsigned)ye * M + xe, pc = (unsigned)zb * MN + (unsigned)yc * M + xc;
        float tr = t_below(row, pr), tc = t_below(colm, pc), u[3];
        Raw wr, wc;
        load(wr, row, xe, ye, pr);
        load(wc, colm, xc, yc, pc);
        for (int z = zb; z < ze; ++z) {
            const float Lr = L_of(wr, tr, u);
            tr = u[2];
            const float Lk = L_of(wc, tc, u);
            tc = u[2];
            pr += MN;
            pc += MN;
            load(wr, row && z + 1 < ze, xe, ye, pr);
            load(wc, colm && z + 1 < ze, xc, yc, pc);
            if (row) sL[z & 1][FG_BY][tx] = Lr;
            if (colm) sL[z & 1][tx][32] = Lk;
            __syncthreads();
        }
        return;
    }
    const int x = x0 + tx, y = y0 + ty;
    const bool in = x < M && y < N;
    const bool ex = x < M - 1, ey = y < N - 1;
    unsigned p = (unsigned)zb * MN + (unsigned)y * M + x;
    float cur[3], nxt[3] = {0.f, 0.f, 0.f}, Ln = 0.0f;
    Raw w;
    load(w, in, x, y, p);
    float Lc = L_of(w, t_below(in, p), cur);
    load(w, in && zb + 1 < Z, x, y, p + MN);
    float ahead[3] = {0.f, 0.f, 0.f};   // not REC: o, p, q of the plane to come
    auto load_o = [&](bool on, unsigned q) {
        if (!REC && !FIRST && on)
#pragma unroll
            for (int a = 0; a < 3; ++a) ahead[a] = Store<T>::ldw(d.o[a] + q);
    };
    load_o(in, p);
    for (int z = zb; z < ze; ++z, p += MN) {
        sL[z & 1][ty][tx] = Lc;
        const bool ez = z < Z - 1;
        const float old[3] = {ahead[0], ahead[1], ahead[2]};
        load_o(in && z + 1 < ze, p + MN);
        Ln = L_of(w, cur[2], nxt);
        load(w, in && z + 1 < ze && z + 2 < Z, x, y, p + 2u * MN);   // (the run's last plane needs L one plane up)
        __syncthreads();   // the other parity's plane is not written before the next barrier
        if (in) {
            float tr = cur[0], ts = cur[1], tt = cur[2];
            if (ex) tr = fa(tr, fm(alpha12, fs(Lc, sL[z & 1][ty][tx + 1])));
            if (ey) ts = fa(ts, fm(alpha12, fs(Lc, sL[z & 1][ty + 1][tx])));
            if (ez) tt = fa(tt, fm(alpha12, fs(Lc, Ln)));
            // :78-86.  The divisor max(1, sqrt(n)) is 1 unless n > 1; otherwise one
            // reciprocal serves the three divisions
            const float n = fa(fa(fm(tr, tr), fm(ts, ts)), fm(tt, tt));
            float v[3] = {tr, ts, tt};
            if (n > 1.0f) {
                const float den = __fsqrt_rn(n), rcp = __frcp_rn(den);
#pragma unroll
                for (int a = 0; a < 3; ++a) v[a] = div_exact(v[a], den, rcp);
            }
            const bool e[3] = {ex, ey, ez};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float on = e[a] ? v[a] : 0.0f;   // an edge that leaves the volume has no dual
                if (REC) {
                    Store<T>::st(d.rn[a] + p, on);
                } else {
                    Store<T>::st(d.rn[a] + p, e[a] ? fa(on, fm(gam, fs(on, old[a]))) : 0.0f);
                    Store<T>::st(d.o[a] + p, on);
                }
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) cur[a] = nxt[a];
        Lc = Ln;
    }
}

// One inner iteration in two passes, for volumes whose tiles k_fgp_step cannot
// fill, and where its nine dual arrays do not fit the memory (one_pass): k_fgp_L
// writes L for every voxel; k_fgp_dual reads L at the voxel and its +x, +y, +z
// neighbours and updates the voxel's own six duals in place (no voxel reads
// another's in this pass).  A thread a voxel, 32x8 tiles, no registers kept
// between planes: twice the warps of k_fgp_step.  Bound by HBM and memory latency (2.6 to
// 3.2 TB/s at 512^3), in L2 by latency.
template <typename T, typename TF>
__global__ void __launch_bounds__(FG_BX * FG_BY)
k_fgp_L(int M, int N, int Z, const TF* __restrict__ f, const T* __restrict__ r, const T* __restrict__ s,
        const T* __restrict__ t, float* __restrict__ L, float lambda)
{
    const int x = blockIdx.x * FG_BX + threadIdx.x, y = blockIdx.y * FG_BY + threadIdx.y, z = blockIdx.z;
    if (x >= M || y >= N) return;
    const long long MN = (long long)M * N, p = (long long)z * MN + (long long)y * M + x;
    L[p] = fgp_L<T, TF>(f, r, s, t, x, y, z, p, M, MN, lambda);
}

template <typename T>
__global__ void __launch_bounds__(FG_BX * FG_BY)
k_fgp_dual(int M, int N, int Z, const float* __restrict__ L, T* __restrict__ r, T* __restrict__ s, T* __restrict__ t,
           T* __restrict__ o, T* __restrict__ pd, T* __restrict__ q, float alpha12, float gam)
{
    const int x = blockIdx.x * FG_BX + threadIdx.x, y = blockIdx.y * FG_BY + threadIdx.y, z = blockIdx.z;
    if (x >= M || y >= N) return;
    const long long MN = (long long)M * N, p = (long long)z * MN + (long long)y * M + x;
    const bool e[3] = {x < M - 1, y < N - 1, z < Z - 1};
    const long long up[3] = {1, M, MN};
    T* const rst[3] = {r, s, t};
    T* const old[3] = {o, pd, q};
    const float Lc = __ldg(L + p);
    float v[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[a] = Store<T>::ldw(rst[a] + p);
        if (e[a]) v[a] = fa(v[a], fm(alpha12, fs(Lc, __ldg(L + p + up[a]))));
    }
    const float den = fmaxf(1.0f, __fsqrt_rn(fa(fa(fm(v[0], v[0]), fm(v[1], v[1])), fm(v[2], v[2]))));   // :78-86
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (e[a]) {
            const float on = fdv(v[a], den);
            Store<T>::st(rst[a] + p, fa(on, fm(gam, fs(on, Store<T>::ldw(old[a] + p)))));
            Store<T>::st(old[a] + p, on);
        }
}

// x* = f - lambda*div(o,p,q) (the final L_Pc, V63/host_FGP_Denoise_GPUx7.c:83);
// with FISTA fused: y = x* + gam*(x* - xprev), xprev = x* (V63/main_recon.cu:375-382).
template <typename T, bool FISTA>
__global__ void __launch_bounds__(FG_BX * FG_BY)
k_fgp_final(int M, int N, int Z, T* __restrict__ vol, const T* __restrict__ o, const T* __restrict__ pd,
            const T* __restrict__ q, float lambda, T* __restrict__ xprev, float gam, const float* __restrict__ gam_dev)
{
    if (FISTA && gam_dev) gam = *gam_dev;
    const int x = blockIdx.x * FG_BX + threadIdx.x, y = blockIdx.y * FG_BY + threadIdx.y;
    if (x >= M || y >= N) return;
    const long long MN = (long long)M * N;
    for (int z = blockIdx.z; z < Z; z += gridDim.z) {
        const long long p = (long long)z * MN + (long long)y * M + x;
        const float xs = fgp_L<T>(vol, o, pd, q, x, y, z, p, M, MN, lambda);
        if (FISTA) {
            const float xp = Store<T>::ldw(xprev + p);
            // the stored x_k is what the momentum step sees
            T xs_t;
            Store<T>::st(&xs_t, xs);
            const float xk = Store<T>::ldw(&xs_t);
            Store<T>::st(vol + p, fa(xk, fm(gam, fs(xk, xp))));
            xprev[p] = xs_t;
        } else {
            Store<T>::st(vol + p, xs);
        }
    }
}

// Refinement solver: the start d0 of the correction volume, the storage
// rounding of y_k - y~_k = (1+g)(x_k - x~_k) - g (x_(k-1) - x~_(k-1)), where
// x~ are the projectors' round-to-nearest copies of the FP32 iterates (the
// pass projects y~_k through the copy of x_k and A x~_(k-1)).  With d
// starting there, A (y~_k + d) is the projection of the FP32 y_k up to the
// rounding of that small difference, so the copies' rounding does not bias
// the fixed point.  T: the copies' type; TD: the correction's (T, or FP32).
// Zero for FP32 copies.
template <typename T, typename TD>
__device__ __forceinline__ float refine_d0(float xk, float xm, float gm)
{
    const float e = fs(fm(fa(1.0f, gm), fs(xk, Store<T>::rn(xk))), fm(gm, fs(xm, Store<T>::rn(xm))));
    return Store<TD>::rn(e);
}

// d = d0 in the tiled layout, one thread per tiled element (padding zero).
template <typename T, typename TD>
__global__ void __launch_bounds__(256)
k_refine_start(const DevGeom g, const float* __restrict__ xk, const float* __restrict__ xm,
               const float* __restrict__ gdev, TD* __restrict__ d)
{
    const float gm = *gdev;
    const long long n = tiled_count(g);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int w = (int)(t & 63);
        const long long tile = t >> 6;
        const int tx = (int)(tile % g.Mt);
        const long long r = tile / g.Mt;
        const int ty = (int)(r % g.Nt);
        const int k = (int)(r / g.Nt);
        const int i = tx * 8 + (w & 7), j = ty * 8 + (w >> 3);
        float v = 0.0f;
        if (i < g.M && j < g.N) {
            const long long p = ((long long)k * g.N + j) * g.M + i;
            v = refine_d0<T, TD>(xk[p], xm[p], gm);
        }
        Store<TD>::st(d + t, v);
    }
}

// The FP32 input of the prox, z = y_k + (d - d0), written over x_(k-1) (which is
// not needed after it).  d is read in the projectors' tiled layout.
template <typename T, typename TD>
__global__ void __launch_bounds__(256)
k_refine_sum(const DevGeom g, const float* __restrict__ xk, float* __restrict__ xm, const TD* __restrict__ d,
             const float* __restrict__ gdev)
{
    const float gm = *gdev;
    const long long MN = (long long)g.M * g.N, n = MN * g.Z;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(p % g.M), y = (int)((p / g.M) % g.N), z = (int)(p / MN);
        const float xkv = xk[p], xmv = xm[p];
        const float yk = fs(fm(fa(1.0f, gm), xkv), fm(gm, xmv));
        xm[p] = fa(yk, fs(Store<TD>::ld(d + tile_index(g, x, y, z)), refine_d0<T, TD>(xkv, xmv, gm)));
    }
}

// Refinement solver: x* = the prox f - lambda*div(o,p,q) of f = xm (FGP), or
// f itself; then the rotation x_(k-1) = x_k, x_k = x*, and the projectors'
// 16-bit copy of x* in the tiled layout (round to nearest).
template <typename T, bool FGP>
__global__ void __launch_bounds__(256)
k_refine_final(const DevGeom g, float* __restrict__ xk, float* __restrict__ xm, const T* __restrict__ o,
               const T* __restrict__ pd, const T* __restrict__ q, float lambda, T* __restrict__ xt)
{
    const int M = g.M;
    const long long MN = (long long)g.M * g.N, n = MN * g.Z;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(p % M), y = (int)((p / M) % g.N), z = (int)(p / MN);
        const float xs = FGP ? fgp_L<T, float>(xm, o, pd, q, x, y, z, p, M, MN, lambda) : xm[p];
        xm[p] = xk[p];
        xk[p] = xs;
        Store<T>::st(xt + tile_index(g, x, y, z), xs);
    }
}

__global__ void k_set_scalar(float* p, float v) { *p = v; }

template <typename T>
__global__ void __launch_bounds__(256)
k_momentum(long long n, T* __restrict__ y, T* __restrict__ xprev, const T* __restrict__ x, float gam,
           const float* __restrict__ gam_dev)
{
    if (gam_dev) gam = *gam_dev;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const float xv = Store<T>::ldw(x + p);
        const float xp = Store<T>::ldw(xprev + p);
        Store<T>::st(y + p, fa(xv, fm(gam, fs(xv, xp))));        // main_recon.cu:378
        Store<T>::st(xprev + p, xv);                              // :380
    }
}

static int grid_for(long long n, int threads)
{
    long long b = (n + threads - 1) / threads;
    if (b > 148LL * 64) b = 148LL * 64;
    return (int)(b < 1 ? 1 : b);
}

// t_k = (1 + sqrt(1 + 4 t^2))/2 in float (V63/host_FGP_Denoise_GPUx7.c:161)
static float next_t(float t) { return (1.0f + sqrtf(1.0f + 4.0f * t * t)) / 2.0f; }

// Whether the one-pass form is the faster one.  It needs tiles with work in them
// (a third of the warps and more registers than the two-pass form), and planes to march
// through; it gains most when the duals exceed the L2 cache, and halves the launches
// of a volume that is little else (16^3 158 / 136).  Two passes / one, us
// for 20 iterations: FP32 512x512x8 531 / 499, 2048x2048x1 1212 / 1434, x2 2725 / 2135,
// 1024x1024x2 490 / 579, x3 953 / 783, 16x512x512 2315 / 1731, 8x512x512 1513 / 1651,
// 512x9x512 719 / 819, 1024x2x1024 901 / 1264; BF16 2048x2048x1 840 / 1294, 16x512x512
// 1629 / 1855, 20x512x512 1899 / 1893, 1024x4x1024 1159 / 1478, 33x512x512 4070 / 3268.
static bool one_pass_faster(const Geometry& G, ctr_dtype dt)
{
    const double M = G.desc.nx, N = G.desc.ny, V = (double)G.nvox();
    const double fill = M * N / (std::ceil(M / FG_BX) * FG_BX * std::ceil(N / FG_BY) * FG_BY);
    const bool big = V * 9 * dtype_size(dt) > 100e6;
    if (V <= 32768) return true;
    if (big) return G.desc.nz >= 2 && fill >= 0.5;
    return (G.desc.nz >= 3 || V <= 600e3) && fill >= 0.6;
}

ctr_status reserve_fgp(Geometry& G, ctr_dtype dt, bool* one_pass)
{
    const size_t V = (size_t)G.nvox(), es = dtype_size(dt), nine = 9 * es * V, seven = (6 * es + sizeof(float)) * V;
    *one_pass = one_pass_faster(G, dt) && (G.fgp_bytes >= nine || !G.fgp_short);
    if (*one_pass) {
        const ctr_status r = ensure_fgp(&G, nine);
        if (r != CTR_ERR_OUT_OF_MEMORY) return r;
        clear_error();
        cudaGetLastError();
        G.fgp_short = true;   // (not tried again: every try would free and allocate)
        *one_pass = false;
    }
    return ensure_fgp(&G, seven);
}

// The inner iterations of the prox of f: duals from zero, the last projections
// o, p, q in D.  The geometry's workspace holds nine arrays of V duals, or six
// and L.
template <typename T, typename TF>
static ctr_status fgp_iterations(Geometry& G, const TF* f, float lambda, int iters, T* D[3], cudaStream_t st)
{
    const int M = G.desc.nx, N = G.desc.ny, Z = G.desc.nz;
    const long long V = G.nvox();
    bool one_pass;
    CTR_TRY(reserve_fgp(G, DT<T>::v, &one_pass));
    T* base = (T*)G.d_fgp;
    T* A[3][3];   // [set][r s t]
    for (int i = 0; i < 3; ++i)
        for (int a = 0; a < 3; ++a) A[i][a] = base + (size_t)(3 * i + a) * V;
    for (int a = 0; a < 3; ++a) D[a] = A[0][a];
    if (iters <= 0) {
        CTR_CUDA_TRY(cudaMemsetAsync(base, 0, 3 * (size_t)V * sizeof(T), st));
        return CTR_OK;
    }
    const float alpha12 = 1.0f / (lambda * 12.0f);                 // :166
    float t_k_1 = 1.0f, gam_prev = 0.0f;
    if (!one_pass) {   // o, p, q in set 0, r, s, t in set 1, then L
        float* L = (float*)((char*)G.d_fgp + 6 * (size_t)V * sizeof(T));
        const dim3 blk(FG_BX, FG_BY), grd((M + FG_BX - 1) / FG_BX, (N + FG_BY - 1) / FG_BY, Z);
        CTR_CUDA_TRY(cudaMemsetAsync(base, 0, 6 * (size_t)V * sizeof(T), st));
        for (int it = 0; it < iters; ++it) {
            const float t_k = next_t(t_k_1);
            k_fgp_L<T, TF><<<grd, blk, 0, st>>>(M, N, Z, f, A[1][0], A[1][1], A[1][2], L, lambda);
            k_fgp_dual<T><<<grd, blk, 0, st>>>(M, N, Z, L, A[1][0], A[1][1], A[1][2], A[0][0], A[0][1], A[0][2], alpha12,
                                               (t_k_1 - 1.0f) / t_k);
            t_k_1 = t_k;
        }
        CTR_CUDA_TRY(cudaGetLastError());
        return CTR_OK;
    }
    // z planes per block: long runs (each recomputes one plane of L) while the
    // blocks still fill the GPU six times (148 SMs x 4 blocks)
    const long long tiles = (long long)((M + FG_BX - 1) / FG_BX) * ((N + FG_BY - 1) / FG_BY);
    int zrun = 32;
    while (zrun > 4 && tiles * ((Z + zrun - 1) / zrun) < 148LL * 24) zrun >>= 1;
    zrun = std::max(zrun, (Z + 65534) / 65535);
    const dim3 blk(32, FG_BY + 1), grd((M + FG_BX - 1) / FG_BX, (N + FG_BY - 1) / FG_BY, (Z + zrun - 1) / zrun);
    for (int it = 0; it < iters; ++it) {
        const float t_k = next_t(t_k_1);
        const float gam = (t_k_1 - 1.0f) / t_k;
        FgpSet<T> d{};
        for (int a = 0; a < 3; ++a) {
            if (FgpSet<T>::REC) {   // o_k, o_(k-1), o_(k+1) rotate through the three sets
                d.r[a] = A[it % 3][a];
                d.r0[a] = it == 1 ? d.r[a] : A[(it + 2) % 3][a];   // g_1 = 0: o_0 = 0 was never written
                d.rn[a] = A[(it + 1) % 3][a];
                D[a] = d.rn[a];
            } else {
                d.r[a] = A[1 + it % 2][a];
                d.rn[a] = A[2 - it % 2][a];
                d.o[a] = A[0][a];
            }
        }
        if (it == 0) k_fgp_step<T, TF, true><<<grd, blk, 0, st>>>(M, N, Z, zrun, f, d, lambda, alpha12, gam, 0.0f);
        else k_fgp_step<T, TF, false><<<grd, blk, 0, st>>>(M, N, Z, zrun, f, d, lambda, alpha12, gam, gam_prev);
        t_k_1 = t_k;
        gam_prev = gam;
    }
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

static dim3 fgp_final_grid(int M, int N, int Z)
{
    return dim3((M + FG_BX - 1) / FG_BX, (N + FG_BY - 1) / FG_BY, std::min(Z, 65535));
}

ctr_status launch_fgp(Geometry& G, void* vol, ctr_dtype dt, float lambda, int iters, void* fista_y,
                      void* fista_xprev, float fista_gamma, cudaStream_t st, const float* gamma_dev)
{
    const int M = G.desc.nx, N = G.desc.ny, Z = G.desc.nz;
    if (fista_y && fista_y != vol) return set_error(CTR_ERR_INVALID_ARGUMENT, "fused FISTA output must alias the volume");
    const dim3 blk(FG_BX, FG_BY), grd = fgp_final_grid(M, N, Z);
    CTR_DISPATCH_DTYPE(dt, T, {
        T* D[3];
        CTR_TRY((fgp_iterations<T, T>(G, (const T*)vol, lambda, iters, D, st)));
        if (fista_y)
            k_fgp_final<T, true><<<grd, blk, 0, st>>>(M, N, Z, (T*)vol, D[0], D[1], D[2], lambda, (T*)fista_xprev,
                                                      fista_gamma, gamma_dev);
        else
            k_fgp_final<T, false><<<grd, blk, 0, st>>>(M, N, Z, (T*)vol, D[0], D[1], D[2], lambda, nullptr, 0.0f, nullptr);
    });
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

ctr_status launch_momentum(const Geometry& G, void* y, void* xprev, const void* x, ctr_dtype dt, float gam,
                           cudaStream_t st, const float* gamma_dev)
{
    const long long V = G.nvox();
    CTR_DISPATCH_DTYPE(dt, T, {
        k_momentum<T><<<grid_for(V, 256), 256, 0, st>>>(V, (T*)y, (T*)xprev, (const T*)x, gam, gamma_dev);
    });
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

ctr_status launch_refine_update(Geometry& G, float* xk, float* xm, const void* d_tiled, ctr_dtype ddt, void* xt_tiled,
                                ctr_dtype dt, float lam, int iters, const float* gdev, cudaStream_t st)
{
    const long long V = G.nvox();
    const bool fgp = lam > 0.f && iters >= 0;
    if (ddt != dt && ddt != CTR_F32) return set_error(CTR_ERR_INVALID_ARGUMENT, "correction type");
    bool one_pass;
    if (fgp) CTR_TRY(reserve_fgp(G, dt, &one_pass));   // before xm is written over
    const int nb = grid_for(V, 256);
    CTR_DISPATCH_DTYPE(dt, T, {
        if (ddt == CTR_F32) k_refine_sum<T, float><<<nb, 256, 0, st>>>(G.dg, xk, xm, (const float*)d_tiled, gdev);
        else k_refine_sum<T, T><<<nb, 256, 0, st>>>(G.dg, xk, xm, (const T*)d_tiled, gdev);
        T* D[3] = {nullptr, nullptr, nullptr};
        if (fgp) CTR_TRY((fgp_iterations<T, float>(G, xm, lam, iters, D, st)));
        if (fgp) k_refine_final<T, true><<<nb, 256, 0, st>>>(G.dg, xk, xm, D[0], D[1], D[2], lam, (T*)xt_tiled);
        else k_refine_final<T, false><<<nb, 256, 0, st>>>(G.dg, xk, xm, D[0], D[1], D[2], 0.f, (T*)xt_tiled);
    });
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

ctr_status launch_refine_start(Geometry& G, const float* xk, const float* xm, void* d_tiled, ctr_dtype ddt,
                               ctr_dtype dt, const float* gdev, cudaStream_t st)
{
    if (ddt != dt && ddt != CTR_F32) return set_error(CTR_ERR_INVALID_ARGUMENT, "correction type");
    const int nb = grid_for(tiled_count(G.dg), 256);
    CTR_DISPATCH_DTYPE(dt, T, {
        if (ddt == CTR_F32) k_refine_start<T, float><<<nb, 256, 0, st>>>(G.dg, xk, xm, gdev, (float*)d_tiled);
        else k_refine_start<T, T><<<nb, 256, 0, st>>>(G.dg, xk, xm, gdev, (T*)d_tiled);
    });
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

ctr_status launch_set_scalar(float* p, float v, cudaStream_t st)
{
    k_set_scalar<<<1, 1, 0, st>>>(p, v);
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

// ---------------------------------------------------------------- reductions

// Sum of part[0..n) in a fixed order: block b sums the contiguous segment
// [b*seg, (b+1)*seg) into out[b].  Repeated runs give identical bits.
__global__ void __launch_bounds__(1024) k_reduce(const double* __restrict__ part, long long n, long long seg,
                                                 double* __restrict__ out)
{
    __shared__ double sh[32];
    const long long lo = blockIdx.x * seg, hi = min(n, lo + seg);
    double v = 0.0;
    for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) v += part[i];
    const double t = block_sum(v, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = t;
}

// Needs 1024 doubles of scratch after part[n].
ctr_status launch_reduce(const double* partial, size_t n, double* out, cudaStream_t st)
{
    if (n > 16384) {
        double* mid = const_cast<double*>(partial) + n;
        const long long seg = ((long long)n + 1023) / 1024;
        k_reduce<<<1024, 1024, 0, st>>>(partial, (long long)n, seg, mid);
        k_reduce<<<1, 1024, 0, st>>>(mid, 1024, 1024, out);
    } else {
        k_reduce<<<1, 1024, 0, st>>>(partial, (long long)n, (long long)n, out);
    }
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

template <int OP>   // 0: a*b, 1: (a-b)^2 in float
__global__ void __launch_bounds__(256)
k_pairsum(const float* __restrict__ a, const float* __restrict__ b, long long n, double* __restrict__ part)
{
    __shared__ double sh[8];
    double v = 0.0;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        if (OP == 0) v += (double)a[i] * (double)b[i];
        else {
            const float e = fs(a[i], b[i]);
            v += (double)fm(e, e);
        }
    }
    const double t = block_sum(v, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

ctr_status launch_dot(const float* a, const float* b, long long n, double* partial, size_t cap, double* out,
                      cudaStream_t st)
{
    int nb = grid_for(n, 256);
    if ((size_t)nb > cap) nb = (int)cap;
    k_pairsum<0><<<nb, 256, 0, st>>>(a, b, n, partial);
    CTR_CUDA_TRY(cudaGetLastError());
    return launch_reduce(partial, nb, out, st);
}

ctr_status launch_l2(const float* a, const float* b, long long n, double* partial, size_t cap, double* out,
                     cudaStream_t st)
{
    int nb = grid_for(n, 256);
    if ((size_t)nb > cap) nb = (int)cap;
    k_pairsum<1><<<nb, 256, 0, st>>>(a, b, n, partial);
    CTR_CUDA_TRY(cudaGetLastError());
    return launch_reduce(partial, nb, out, st);
}

// TV_norm_kernel (V63/kernel_tool_functions.cu:39-65) with an FP64 block sum.
template <typename T>
__global__ void __launch_bounds__(256)
k_tv(int M, int N, int Z, const T* __restrict__ d, double* __restrict__ part)
{
    __shared__ double sh[8];
    const long long MN = (long long)M * N, n = MN * Z;
    double acc = 0.0;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const int x = (int)(i % M), y = (int)((i / M) % N), z = (int)(i / MN);
        const float c = Store<T>::ld(d + i);
        const float dj = x < M - 1 ? fs(c, Store<T>::ld(d + i + 1)) : 0.f;
        const float dk = y < N - 1 ? fs(c, Store<T>::ld(d + i + M)) : 0.f;
        const float dl = z < Z - 1 ? fs(c, Store<T>::ld(d + i + MN)) : 0.f;
        float tv = 0.0f;
        const bool bx = x < M - 1, by = y < N - 1, bz = z < Z - 1;
        if (bx && by && bz) tv = __fsqrt_rn(fa(fa(fm(dj, dj), fm(dk, dk)), fm(dl, dl)));
        else if (!bx && by && bz) tv = __fsqrt_rn(fa(fm(dk, dk), fm(dl, dl)));
        else if (bx && !by && bz) tv = __fsqrt_rn(fa(fm(dj, dj), fm(dl, dl)));
        else if (bx && by && !bz) tv = __fsqrt_rn(fa(fm(dj, dj), fm(dk, dk)));
        else if (!bx && !by && bz) tv = fabsf(dl);
        else if (!bx && by && !bz) tv = fabsf(dk);
        else if (bx && !by && !bz) tv = fabsf(dj);
        acc += (double)tv;
    }
    const double t = block_sum(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

ctr_status launch_tv(const Geometry& G, const void* vol, ctr_dtype dt, double* partial, size_t cap, double* out,
                     cudaStream_t st)
{
    const long long V = G.nvox();
    int nb = grid_for(V, 256);
    if ((size_t)nb > cap) nb = (int)cap;
    CTR_DISPATCH_DTYPE(dt, T, { k_tv<T><<<nb, 256, 0, st>>>(G.desc.nx, G.desc.ny, G.desc.nz, (const T*)vol, partial); });
    CTR_CUDA_TRY(cudaGetLastError());
    return launch_reduce(partial, nb, out, st);
}

template <typename S, typename D>
__global__ void k_convert(const S* __restrict__ s, D* __restrict__ d, long long n)
{
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += (long long)gridDim.x * 256)
        Store<D>::st(d + i, Store<S>::ld(s + i));
}

ctr_status launch_convert(const void* src, ctr_dtype sdt, void* dst, ctr_dtype ddt, long long n, cudaStream_t st)
{
    const int nb = grid_for(n, 256);
    CTR_DISPATCH_DTYPE(sdt, S, {
        CTR_DISPATCH_DTYPE(ddt, D, { k_convert<S, D><<<nb, 256, 0, st>>>((const S*)src, (D*)dst, n); });
    });
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

}  // namespace ctr
