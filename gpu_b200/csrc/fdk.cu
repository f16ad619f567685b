// fdk.cu -- FDK reconstruction and ellipsoid phantom utilities.
//
// FDK restates Reconstruction_FDK (V63/host_FDK.cpp:4-57):
//   1. cosine pre-weight, kernel_FDK_projection_adjust (V63/FDK/kernel_FDK.cu:1-14);
//   2. ramp filter.  The reference zero-pads each row to 2R, runs a cuFFT C2C,
//      multiplies by |k|*F_step*0.5 and inverts (V63/FDK/FFT_1d_GPU.h:241-287),
//      i.e. a linear convolution with h[n] = (1/2R) sum_k H[k] cos(pi k n / R),
//      |n| < R, h computed once in FP64 on the host.  Rows of up to
//      kFftMost / 2 values are weighted and filtered in one kernel by an FFT in
//      shared memory (k_ramp_fft); longer ones by a register-tiled Toeplitz
//      product (k_fdk_weight, k_ramp);
//   3. voxel-driven bilinear backprojection, kernel_FDK_reconstruction
//      (V63/FDK/kernel_FDK.cu:16-62), with a batch of views per launch held in
//      registers (each view's update is still applied with the reference's
//      float/double steps, so the sum is the reference's to the bit).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "ctr_device.cuh"

namespace ctr {

__global__ void k_fdk_weight(const DevGeom g, const float* __restrict__ in, float* __restrict__ out)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y;
    const int w = blockIdx.z;
    if (u >= g.R) return;
    const long long p = ((long long)w * g.ZP + v) * g.R + u;
    const float x1 = g.dso;
    const float dd = fs(g.dso, g.dod);
    const float x2 = fdv(fm(fa(g.ymin, fm((float)u, g.du)), g.dso), dd);
    const float x3 = fdv(fm(fa(g.zmin, fm((float)v, g.dv)), g.dso), dd);
    out[p] = fdv(fm(in[p], g.dso), __fsqrt_rn(fa(fa(fm(x1, x1), fm(x2, x2)), fm(x3, x3))));
}

// Toeplitz row convolution out[r][j] = sum_m in[r][m] * h[j - m + R - 1].
// Block tile: 32 rows x 128 outputs; a thread owns 8 rows x 4 consecutive
// outputs and slides a 4-tap register window along m.
static constexpr int RP_COLS = 128, RP_ROWS = 32, RP_MC = 32, RP_TR = 8;
__global__ void __launch_bounds__(128)
k_ramp(const float* __restrict__ in, float* __restrict__ out, const float* __restrict__ h, int R, long long nrows)
{
    __shared__ float sg[RP_ROWS][RP_MC + 1];
    __shared__ float sh[RP_COLS + RP_MC + 4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j0 = blockIdx.x * RP_COLS;
    const long long r0 = (long long)blockIdx.y * RP_ROWS;
    const int jt = j0 + 4 * lane;          // first of this thread's 4 outputs
    float acc[RP_TR][4];
#pragma unroll
    for (int a = 0; a < RP_TR; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
    for (int m0 = 0; m0 < R; m0 += RP_MC) {
        __syncthreads();
        for (int t = threadIdx.x; t < RP_ROWS * RP_MC; t += 128) {
            const int rr = t / RP_MC, mm = t % RP_MC;
            const long long row = r0 + rr;
            sg[rr][mm] = (row < nrows && m0 + mm < R) ? in[row * R + m0 + mm] : 0.f;
        }
        // taps h[j - m + R - 1] for j in [j0, j0+128), m in [m0, m0+MC):
        // index e = j - m + R - 1 - (j0 - m0 - MC + 1 + R - 1) in [0, 128+MC-1)
        const int ebase = j0 - m0 - RP_MC + 1 + R - 1;
        for (int t = threadIdx.x; t < RP_COLS + RP_MC + 4; t += 128) {
            const int e = ebase + t;
            sh[t] = (e >= 0 && e < 2 * R - 1) ? h[e] : 0.f;
        }
        __syncthreads();
        // for output jt+b and m = m0+mm the tap is sh[jt + b - j0 - mm + MC - 1]
        const int hb = 4 * lane + RP_MC - 1;
        float w0 = sh[hb + 0], w1 = sh[hb + 1], w2 = sh[hb + 2], w3 = sh[hb + 3];
#pragma unroll 8
        for (int mm = 0; mm < RP_MC; ++mm) {
#pragma unroll
            for (int a = 0; a < RP_TR; ++a) {
                const float gv = sg[warp * RP_TR + a][mm];
                acc[a][0] = fmaf(gv, w0, acc[a][0]);
                acc[a][1] = fmaf(gv, w1, acc[a][1]);
                acc[a][2] = fmaf(gv, w2, acc[a][2]);
                acc[a][3] = fmaf(gv, w3, acc[a][3]);
            }
            // slide: next m needs taps one lower
            w3 = w2; w2 = w1; w1 = w0;
            w0 = sh[hb - mm - 1 >= 0 ? hb - mm - 1 : 0];
        }
    }
#pragma unroll
    for (int a = 0; a < RP_TR; ++a) {
        const long long row = r0 + warp * RP_TR + a;
        if (row >= nrows) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (jt + b < R) out[row * R + jt + b] = acc[a][b];
    }
}

// ---- weight and ramp of a detector row by FFT
//
// A row of R values is n = a power of two >= 2R - 1 real points, transformed in
// FP64 as n/2 complex ones (even + i odd points): Stockham passes of radix 8
// (radix 4 or 2 last), 8 points a thread, exchanged through one padded
// shared-memory buffer.  The first pass reads the row (weighted on the way with
// k_fdk_weight's operations, zero beyond R); the inverse's first pass separates
// the two interleaved spectra, multiplies by the taps' spectrum (real: the taps
// are even) and joins them again; its last pass writes the row.  Short rows
// share a block.  The length is a template parameter: with the passes unrolled and
// their addresses folded a row of 1024 takes 60 % of the time.
//
// FP64 because the ramp removes what a smooth row is made of, low frequencies:
// an FP32 transform's error follows the row's largest values and is several
// times the direct sum's.  A row alone because two rows as the real and
// imaginary part of one transform share their rounding error and every NaN.  A
// row with a non-finite value is summed directly (its transform would turn one
// Inf into NaN everywhere), with k_ramp's operations.
//
// Bound by shared memory (8 exchanges of 16 KB for 1024 values; the LSU data pipe
// at 92 %), 24 warps an SM.  256 views x 768 rows of 1024: 2.34 ms, weight
// included (4.0 ms with the length as an argument); FP32 pairs of rows 3.10 ms; the
// Toeplitz product and the weight pass 10.3 ms.  360 x 64 rows of 64: 15, 31 and 27 us.
static constexpr int kFftMost = 8192;     // 512 threads, 74 KB of shared memory

__device__ __forceinline__ int fft_pad(int i) { return i + (i >> 3); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// i*a (inverse) or -i*a (forward)
template <bool INV> __device__ __forceinline__ double2 crot(double2 a)
{
    return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}
__device__ __forceinline__ void fft2(double2& a, double2& b)
{
    const double2 t = csub(a, b);
    a = cadd(a, b);
    b = t;
}
template <bool INV> __device__ __forceinline__ void fft4(double2* v)   // in order
{
    const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = crot<INV>(csub(v[1], v[3]));
    v[0] = cadd(a, c);
    v[1] = cadd(b, d);
    v[2] = csub(a, c);
    v[3] = csub(b, d);
}
template <bool INV> __device__ __forceinline__ void fft8(double2* v)   // in order
{
    const double h = 0.70710678118654752440;
    double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    fft4<INV>(e);
    fft4<INV>(o);
    // o1 exp(-+i pi/4) and o3 exp(-+3i pi/4)
    const double2 r1 = crot<INV>(o[1]), r3 = crot<INV>(o[3]);
    o[1] = make_double2(h * (o[1].x + r1.x), h * (o[1].y + r1.y));
    o[2] = crot<INV>(o[2]);
    o[3] = make_double2(h * (r3.x - o[3].x), h * (r3.y - o[3].y));
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        v[t] = cadd(e[t], o[t]);
        v[t + 4] = csub(e[t], o[t]);
    }
}

// One pass of radix RX over n points whose sub-transforms have length ns:
// thread index j of n / RX holds points j + m n/RX; the results go to
// (j/ns) ns RX + j%ns + m ns.  tw[t] = exp(-2 pi i t / n).
template <int RX, bool INV>
__device__ __forceinline__ void fft_radix(double2* v, int j, int ns, int n, const double2* __restrict__ tw)
{
    if (ns > 1) {
        double2 w[8];   // powers of the butterfly's root: one load
        w[1] = __ldg(tw + (j & (ns - 1)) * (n / (ns * RX)));
        if (INV) w[1].y = -w[1].y;
#pragma unroll
        for (int m = 2; m < RX; ++m) w[m] = cmul(w[m >> 1], w[m - (m >> 1)]);
#pragma unroll
        for (int m = 1; m < RX; ++m) v[m] = cmul(v[m], w[m]);
    }
    if (RX == 8) fft8<INV>(v);
    else if (RX == 4) fft4<INV>(v);
    else fft2(v[0], v[1]);
}

// The passes of one direction over the 8 points of thread j of a row.  get(i)
// yields point i of the first pass, put(i, v) takes point i of the last; in
// between the points go through sh.  The forward's get does not read sh, the
// inverse's put does not write it.  The sub-transform lengths are 1, 8, 64, ...; a
// last pass of radix 2 or 4 does 4 or 2 butterflies a thread.
template <bool INV, int LOG2N, typename G, typename P>
__device__ __forceinline__ void fft_passes(double2* sh, int j, const double2* __restrict__ tw, G get, P put)
{
    constexpr int n = 1 << LOG2N, T = n >> 3;
    double2 v[8];
#pragma unroll
    for (int done = 0; done < LOG2N; done += 3) {   // levels of the transform
        const int ns = 1 << done;
        const bool first = done == 0;
        const int lr = min(3, LOG2N - done);
        const bool last = done + lr == LOG2N;
        const bool reads = INV || !first, writes = !INV || !last;   // of sh
        if (reads) __syncthreads();   // the previous pass's stores
        if (lr == 3) {
#pragma unroll
            for (int m = 0; m < 8; ++m) v[m] = first ? get(j + m * T) : sh[fft_pad(j + m * T)];
            fft_radix<8, INV>(v, j, ns, n, tw);
        } else {   // never the first pass: n >= 8
            if (lr == 2) {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = sh[fft_pad(j + (q >> 2) * T + (q & 3) * 2 * T)];
                fft_radix<4, INV>(v, j, ns, n, tw);
                fft_radix<4, INV>(v + 4, j + T, ns, n, tw);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = sh[fft_pad(j + (q >> 1) * T + (q & 1) * 4 * T)];
#pragma unroll
                for (int h = 0; h < 4; ++h) fft_radix<2, INV>(v + 2 * h, j + h * T, ns, n, tw);
            }
        }
        if (reads && writes) __syncthreads();   // every load done
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int jj = j + (q >> lr) * T, m = q & ((1 << lr) - 1);
            const int at = ((jj & ~(ns - 1)) << lr) + (jj & (ns - 1)) + m * ns;
            if (last) put(at, v[q]);
            else sh[fft_pad(at)] = v[q];
        }
    }
}

// Tables of k_ramp_fft (fft_tables): N = n/2 roots exp(-2 pi i t / N); per k
// of N the pair exp(-2 pi i k / n), (H[k] +- H[N-k]) / 2N; the weights' roots
// [v][u]; R taps.
struct FftTables {
    const double2* tw;
    const double2* un;
    const float* root;
    const float* taps;
};

// nrows rows of R values (row % ZP is the detector row): out = ramp(weight * in).
// A block takes fft_rows rows of N/8 threads.
constexpr int fft_rows(int log2N) { return log2N < 10 ? 1024 >> log2N : 1; }
constexpr int fft_threads(int log2N) { return fft_rows(log2N) << (log2N - 3); }   // 128, 256, 512
template <int LOG2N>
__global__ void __launch_bounds__(fft_threads(LOG2N), 6 * 128 / fft_threads(LOG2N))
k_ramp_fft(const float* __restrict__ in, float* __restrict__ out, const FftTables tb, float dso, int R, int ZP,
           long long nrows)
{
    constexpr int N = 1 << LOG2N, T = N >> 3;
    extern __shared__ double2 fsh[];
    __shared__ int bad[fft_rows(LOG2N)];   // rows with a non-finite value
    const int rl = threadIdx.x / T, j = threadIdx.x % T;
    const long long row = (long long)blockIdx.x * fft_rows(LOG2N) + rl;
    const bool live = row < nrows;
    double2* const sh = fsh + (size_t)rl * (N + T);
    const float* __restrict__ a = in + (live ? row : 0) * R;
    const float* __restrict__ rt = tb.root + (live ? row % ZP : 0) * R;
    if (j == 0) bad[rl] = 0;
    __syncthreads();
    auto value = [&](int i) { return fdv(fm(__ldg(a + i), dso), __ldg(rt + i)); };   // kernel_FDK.cu:1-14
    bool off = false;
    fft_passes<false, LOG2N>(sh, j, tb.tw, [&](int i) {
        float x = 0.0f, y = 0.0f;
        if (live && 2 * i < R) x = value(2 * i);
        if (live && 2 * i + 1 < R) y = value(2 * i + 1);
        off |= !(fabsf(x) <= 3.402823466e38f) || !(fabsf(y) <= 3.402823466e38f);
        return make_double2((double)x, (double)y);
    }, [&](int i, double2 v) { sh[fft_pad(i)] = v; });
    if (off) bad[rl] = 1;
    // Z = E + iO, the spectra of the even and the odd points; with the taps'
    // X[k] = E + W O, X[k+N] = E - W O become H[k] X[k], H[N-k] X[k+N]
    float* __restrict__ o = out + (live ? row : 0) * R;
    fft_passes<true, LOG2N>(sh, j, tb.tw, [&](int k) {
        const double2 z = sh[fft_pad(k)], y = sh[fft_pad((N - k) & (N - 1))];
        const double2 w = __ldg(tb.un + 2 * k), h = __ldg(tb.un + 2 * k + 1);
        const double2 e = make_double2(0.5 * (z.x + y.x), 0.5 * (z.y - y.y));
        const double2 od = make_double2(0.5 * (z.y + y.y), 0.5 * (y.x - z.x));
        const double2 wo = cmul(w, od), we = cmul(make_double2(w.x, -w.y), e);
        return make_double2(fma(h.x, z.x, h.y * (wo.x - we.y)), fma(h.x, z.y, h.y * (wo.y + we.x)));
    }, [&](int i, double2 v) {
        if (!live || bad[rl]) return;
        if (2 * i < R) o[2 * i] = (float)v.x;
        if (2 * i + 1 < R) o[2 * i + 1] = (float)v.y;
    });
    if (live && bad[rl])
        for (int u = j; u < R; u += T) {
            float acc = 0.0f;
            for (int m = 0; m < R; ++m) acc = fmaf(value(m), __ldg(tb.taps + abs(u - m)), acc);
            o[u] = acc;
        }
}

static constexpr int FB_BX = 32, FB_BY = 4;

// floor(x) and (int)floor(x) for 0 <= x < 2^22 without conversion
// instructions (the backprojection is bound by the pipe that executes them):
// adding 1.5*2^23 rounds x to an integer m held in the low mantissa bits, and
// m - 1 when m > x.  Both results are exact, so they equal the reference's
// an = floor(ksi) and (float)an.
__device__ __forceinline__ float floor_small(float x, int& n)
{
    const float C = 12582912.0f;   // 1.5 * 2^23
    const float t = __fadd_rn(x, C);
    float r = __fsub_rn(t, C);
    n = __float_as_int(t) - 0x4B400000;
    if (r > x) {
        r = __fsub_rn(r, 1.0f);
        n -= 1;
    }
    return r;
}
// x / d, correctly rounded, from r = 1/d correctly rounded: one multiplication
// and two fused multiply-adds (Markstein's division; Brisebarre, Muller and
// Raina, IEEE Trans. Computers 53(8), 2004, for a divisor known in advance).
// The remainder must not underflow; the launcher checks the geometry's scale
// (RCP) and the divisions are written out otherwise.  Compared with x / d on
// 1.2e9 pairs of random mantissas: no difference.
template <bool RCP> __device__ __forceinline__ float div_by(float x, float d, float r)
{
    if (!RCP) return fdv(x, d);
    const float q = fm(x, r);
    return __fmaf_rn(__fmaf_rn(-d, q, x), r, q);
}

// FULL: a full circle (us_rate*Nviews == 360).  Three divisions per voxel and
// view (by the voxel column's distance, DSO and the row pitch) by div_by, what
// does not depend on z once per K voxels of a column.  Bound by issue; 32 views into
// 512^3: 7.3 ms (13.6 ms with IEEE divide sequences and 4 voxels a thread).
template <bool FULL, bool RCP, int K>
__global__ void __launch_bounds__(FB_BX * FB_BY)
k_fdk_bp(const __grid_constant__ DevGeom g, float* __restrict__ vol, const float* __restrict__ proj, int view0, int nview)
{
    const int i = blockIdx.x * FB_BX + (threadIdx.x % FB_BX);
    const int j = blockIdx.y * FB_BY + (threadIdx.x / FB_BX);
    const int k0 = blockIdx.z * K;
    if (i >= g.M || j >= g.N) return;
    const long long MN = (long long)g.M * g.N;
    const int R = g.R, ZP = g.ZP;
    const float DSO = g.dso, SDD = fs(g.dso, g.dod), Rf = (float)R, ZPf = (float)ZP;
    const float r_dso = __frcp_rn(DSO), r_du = __frcp_rn(g.du), r_dv = __frcp_rn(g.dv);
    // kernel_FDK.cu:86-88
    const float x = fa(fa(g.bx, fm(g.vx, 0.5f)), fm((float)i, g.vx));
    const float y = fa(fa(g.by, fm(g.vy, 0.5f)), fm((float)j, g.vy));
    float acc[K], dz[K];
#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
        const int k = min(k0 + kk, g.Z - 1);
        acc[kk] = vol[(long long)k * MN + (long long)j * g.M + i];
        dz[kk] = fm(DSO, fa(fa(g.bz, fm(g.vz, 0.5f)), fm((float)k, g.vz)));
    }
    for (int w = 0; w < nview; ++w) {
        const float2 scv = g.trig_fdk[view0 + w];
        const float sn = scv.x, cs = scv.y;
        const float t = fa(fm(x, cs), fm(y, sn));
        const float s = fa(fm(-x, sn), fm(y, cs));
        const float ds = fs(DSO, s), r_ds = __frcp_rn(ds);
        const float temp1 = fdv(fm(DSO, DSO), fm(ds, ds));
        float p = div_by<RCP>(fm(DSO, t), ds, r_ds);
        p = div_by<RCP>(fs(div_by<RCP>(fm(p, SDD), DSO, r_dso), g.ymin), g.du, r_du);
        const bool in_u = (0 <= p) && (fa(p, 1.0f) < Rf);
        int bn;
        const float bn0 = fs(p, floor_small(in_u ? p : 0.0f, bn)), bn1 = fs(1.0f, bn0);
        const float* __restrict__ pv = proj + (long long)w * R * ZP + bn;
#pragma unroll
        for (int kk = 0; kk < K; ++kk) {
            float ksi = div_by<RCP>(dz[kk], ds, r_ds);
            ksi = div_by<RCP>(fs(div_by<RCP>(fm(ksi, SDD), DSO, r_dso), g.zmin), g.dv, r_dv);
            float temp2 = 0.0f;
            if ((0 <= ksi) && (fa(ksi, 1.0f) < ZPf) && in_u) {
                int an;
                const float an0 = fs(ksi, floor_small(ksi, an)), an1 = fs(1.0f, an0);   // ksi - an, an = floor(ksi)
                const float* q0 = pv + R * an;
                const float* q1 = q0 + R;
                const float t00 = fm(fm(an1, bn1), __ldg(q0));
                const float t01 = fm(fm(an1, bn0), __ldg(q0 + 1));
                const float t10 = fm(fm(an0, bn1), __ldg(q1));
                const float t11 = fm(fm(an0, bn0), __ldg(q1 + 1));
                temp2 = fa(fa(fa(t00, t01), t10), t11);
            }
            // vol += temp1*temp2*(us_rate*PI/180.0f)*360.0/(us_rate*Nviews)  (float*float*float, then double)
            const float fprod = fm(fm(temp1, temp2), g.fdk_ang);
            if (FULL) {
                // a full circle: (double)fprod*360.0 is exact
                // (24 + 6 significant bits) and dividing it by 360 gives fprod back; and
                // the FP64 sum of two floats rounded to float is their float sum (when
                // the FP64 sum is inexact the smaller term is below 2^-28 of the larger,
                // far under half a float ulp), so the update is one float add
                acc[kk] = fa(acc[kk], fprod);
            } else {
                const double dv = __ddiv_rn(__dmul_rn((double)fprod, 360.0), (double)g.fdk_usn);
                acc[kk] = (float)__dadd_rn((double)acc[kk], dv);
            }
        }
    }
#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
        const int k = k0 + kk;
        if (k < g.Z) vol[(long long)k * MN + (long long)j * g.M + i] = acc[kk];
    }
}

// h[n + R - 1], |n| < R, of the reference's padded-DFT ramp (FP64, as the oracle).
static void ramp_taps(const ctr_geometry_desc& d, std::vector<double>& taps)
{
    const int R = d.nu, P = 2 * R;
    const float DSO = d.dso, DOD = d.dod;
    const float F_max = (float)(1.0 / 2.0 / (double)(d.du * DSO / (DSO - DOD)));   // FFT_1d_GPU.h:246
    const float F_step = F_max / (float)(P / 2);
    std::vector<float> H(P);
    for (int i = 0; i < P; ++i) {
        const int k = (i >= P / 2) ? i - P : i;
        float hv = (float)std::abs(k) * F_step;
        hv *= 0.5f;
        H[i] = hv;
    }
    taps.assign(2 * R - 1, 0.0);
    std::vector<double> cosine(P);
    for (int m = 0; m < P; ++m) cosine[m] = std::cos(2.0 * M_PI * (double)m / (double)P);
    for (int n = 0; n <= R - 1; ++n) {
        double acc = 0.0;
        for (int i = 0, m = 0; i < P; ++i, m = m + n < P ? m + n : m + n - P) acc += (double)H[i] * cosine[m];   // m = i n mod P
        taps[R - 1 + n] = taps[R - 1 - n] = acc / (double)P;
    }
}

// The tables of k_ramp_fft, one allocation (G.d_ramp).
static size_t fft_points(int R)
{
    size_t n = 16;
    while (n < 2 * (size_t)R - 1) n <<= 1;
    return n;
}
static FftTables fft_table_pointers(const Geometry& G, size_t N)
{
    FftTables t;
    t.tw = reinterpret_cast<const double2*>(G.d_ramp);
    t.un = t.tw + N;
    t.root = reinterpret_cast<const float*>(t.un + 2 * N);
    t.taps = t.root + (size_t)G.dg.R * G.dg.ZP;
    return t;
}
static ctr_status fft_tables(Geometry& G, const std::vector<double>& taps)
{
    const DevGeom& g = G.dg;
    const int R = g.R, ZP = g.ZP;
    const size_t n = fft_points(R), N = n / 2;
    std::vector<double> c(n), s(n), d(6 * N), H(N + 1);   // cos, sin(2 pi t / n); the FP64 tables; the spectrum / N
    for (size_t t = 0; t < n; ++t) {
        const double a = 2.0 * M_PI * (double)t / (double)n;
        c[t] = std::cos(a);
        s[t] = std::sin(a);
    }
    for (size_t k = 0; k <= N; ++k) {
        double acc = taps[R - 1];
        for (int m = 1; m < R; ++m) acc += 2.0 * taps[R - 1 + m] * c[(k * (size_t)m) & (n - 1)];
        H[k] = acc / (double)N;
    }
    for (size_t k = 0; k < N; ++k) {
        d[2 * k] = c[2 * k];
        d[2 * k + 1] = -s[2 * k];
        double* un = d.data() + 2 * N + 4 * k;
        un[0] = c[k];
        un[1] = -s[k];
        un[2] = 0.5 * (H[k] + H[N - k]);
        un[3] = 0.5 * (H[k] - H[N - k]);
    }
    // the weights' roots with k_fdk_weight's operations (float, each rounded), and the taps
    std::vector<float> f((size_t)R * ZP + R);
    const float dd = g.dso - g.dod, x1x1 = g.dso * g.dso;
    std::vector<float> x2x2(R);
    for (int u = 0; u < R; ++u) {
        const float x2 = (g.ymin + (float)u * g.du) * g.dso / dd;
        x2x2[u] = x2 * x2;
        f[(size_t)R * ZP + u] = (float)taps[R - 1 + u];
    }
    for (int v = 0; v < ZP; ++v) {
        const float x3 = (g.zmin + (float)v * g.dv) * g.dso / dd, x3x3 = x3 * x3;
        for (int u = 0; u < R; ++u) f[(size_t)v * R + u] = std::sqrt((x1x1 + x2x2[u]) + x3x3);
    }
    const size_t db = d.size() * sizeof(double), fb = f.size() * sizeof(float);
    CTR_CUDA_TRY(cudaMalloc(&G.d_ramp, db + fb));
    CTR_CUDA_TRY(cudaMemcpy(G.d_ramp, d.data(), db, cudaMemcpyHostToDevice));
    CTR_CUDA_TRY(cudaMemcpy((char*)G.d_ramp + db, f.data(), fb, cudaMemcpyHostToDevice));
    return CTR_OK;
}

ctr_status launch_fdk(Geometry& G, const float* sino, float* vol, cudaStream_t st)
{
    const DevGeom& g = G.dg;
    const int nv = g.nviews;
    const long long P = G.npix();
    const size_t n = fft_points(g.R);
    const bool fft = n <= (size_t)kFftMost;
    if (!G.d_ramp) {
        std::vector<double> taps;
        ramp_taps(G.desc, taps);
        if (fft) {
            CTR_TRY(fft_tables(G, taps));
        } else {
            const std::vector<float> h(taps.begin(), taps.end());
            CTR_CUDA_TRY(cudaMalloc(&G.d_ramp, h.size() * sizeof(float)));
            CTR_CUDA_TRY(cudaMemcpy(G.d_ramp, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
        }
    }
    const size_t need = (size_t)P * nv * (fft ? 1 : 2);
    if (G.fdk_cap < need) {
        if (G.d_fdk) cudaFree(G.d_fdk);
        G.d_fdk = nullptr;
        G.fdk_cap = 0;
        CTR_CUDA_TRY(cudaMalloc(&G.d_fdk, need * sizeof(float)));
        G.fdk_cap = need;
    }
    float* fsino = G.d_fdk;
    const long long nrows = (long long)nv * g.ZP;
    if (fft) {
        const size_t N = n / 2;
        const FftTables tb = fft_table_pointers(G, N);
        auto launch = [&](auto log2N) -> cudaError_t {
            constexpr int L = decltype(log2N)::value, rows = fft_rows(L);
            constexpr size_t smem = (size_t)rows * ((1 << L) + (1 << L >> 3)) * sizeof(double2);
            const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(&k_ramp_fft<L>),
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            k_ramp_fft<L><<<(unsigned)((nrows + rows - 1) / rows), fft_threads(L), smem, st>>>(sino, fsino, tb, g.dso, g.R,
                                                                                             g.ZP, nrows);
            return cudaGetLastError();
        };
        cudaError_t e = cudaErrorInvalidValue;
        switch (N) {
        case 8: e = launch(std::integral_constant<int, 3>()); break;
        case 16: e = launch(std::integral_constant<int, 4>()); break;
        case 32: e = launch(std::integral_constant<int, 5>()); break;
        case 64: e = launch(std::integral_constant<int, 6>()); break;
        case 128: e = launch(std::integral_constant<int, 7>()); break;
        case 256: e = launch(std::integral_constant<int, 8>()); break;
        case 512: e = launch(std::integral_constant<int, 9>()); break;
        case 1024: e = launch(std::integral_constant<int, 10>()); break;
        case 2048: e = launch(std::integral_constant<int, 11>()); break;
        case 4096: e = launch(std::integral_constant<int, 12>()); break;
        }
        CTR_CUDA_TRY(e);
    } else {
        float* wsino = G.d_fdk + (size_t)P * nv;
        for (int v0 = 0; v0 < nv; v0 += 65535) {
            const int cnt = std::min(65535, nv - v0);
            k_fdk_weight<<<dim3((g.R + 127) / 128, g.ZP, cnt), 128, 0, st>>>(g, sino + (size_t)P * v0, wsino + (size_t)P * v0);
        }
        for (long long r0 = 0; r0 < nrows; r0 += 65535LL * RP_ROWS) {
            const long long cnt = std::min<long long>(65535LL * RP_ROWS, nrows - r0);
            dim3 grd((g.R + RP_COLS - 1) / RP_COLS, (unsigned)((cnt + RP_ROWS - 1) / RP_ROWS));
            k_ramp<<<grd, 128, 0, st>>>(wsino + r0 * g.R, fsino + r0 * g.R, G.d_ramp, g.R, cnt);
        }
    }
    CTR_CUDA_TRY(cudaGetLastError());
    return launch_fdk_bp(G, fsino, 0, nv, vol, st);
}

// In-place exchange of x and y in every z slice of a square (nx == ny) volume.
__global__ void k_swap_xy(int n, int Z, float* __restrict__ vol)
{
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, k = blockIdx.z;
    if (i >= n || j >= n || i >= j) return;
    float* sl = vol + (long long)k * n * n;
    const float a = sl[(long long)j * n + i];
    sl[(long long)j * n + i] = sl[(long long)i * n + j];
    sl[(long long)i * n + j] = a;
}

ctr_status launch_swap_xy(const Geometry& G, float* vol, cudaStream_t st)
{
    const int n = G.desc.nx, Z = G.desc.nz;
    k_swap_xy<<<dim3((n + 31) / 32, (n + 7) / 8, Z), dim3(32, 8), 0, st>>>(n, Z, vol);
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

ctr_status launch_fdk_bp(const Geometry& G, const float* fsino, int view0, int nview, float* vol, cudaStream_t st)
{
    const DevGeom& g = G.dg;
    const long long P = G.npix();
    // 8 voxels a thread, or 4 while that leaves the GPU short of blocks (148 SMs x
    // 4) and gives more of them.  4 / 8, ms, 180 views: 64^3 (256 blocks of 8) 0.326 /
    // 0.417, 256^2 x 8 (512) 0.312 / 0.355, 64^2 x 4 0.213 / 0.196; above, 8 voxels share
    // more of the in-plane work
    const dim3 tiles((g.M + FB_BX - 1) / FB_BX, (g.N + FB_BY - 1) / FB_BY);
    const bool wide = (long long)tiles.x * tiles.y * ((g.Z + 7) / 8) >= 148 * 4 || g.Z <= 4;
    const dim3 grd(tiles.x, tiles.y, wide ? (g.Z + 7) / 8 : (g.Z + 3) / 4);
    // div_by: lengths far from the ends of the float range
    auto plain = [](float v) { return std::fabs(v) > 1e-9f && std::fabs(v) < 1e9f; };
    const bool rcp = plain(g.dso) && plain(g.dsod) && plain(g.du) && plain(g.dv) && plain(g.vx) && plain(g.vy) && plain(g.vz);
    const int VB = 32;
    for (int w = 0; w < nview; w += VB) {
        const float* f = fsino + (size_t)P * w;
        const int n = std::min(VB, nview - w);
        auto launch = [&](auto full, auto known) {
            constexpr bool FULL = decltype(full)::value, RCP = decltype(known)::value;
            if (wide) k_fdk_bp<FULL, RCP, 8><<<grd, FB_BX * FB_BY, 0, st>>>(g, vol, f, view0 + w, n);
            else k_fdk_bp<FULL, RCP, 4><<<grd, FB_BX * FB_BY, 0, st>>>(g, vol, f, view0 + w, n);
        };
        if (!rcp) {
            if (g.fdk_full) launch(std::true_type(), std::false_type());
            else launch(std::false_type(), std::false_type());
        } else {
            if (g.fdk_full) launch(std::true_type(), std::true_type());
            else launch(std::false_type(), std::true_type());
        }
    }
    CTR_CUDA_TRY(cudaGetLastError());
    return CTR_OK;
}

// ---------------------------------------------------------------- phantoms
// Per ellipsoid: centre(3), rotation R (row major, 9), semi-axes(3), mu.
struct Ell { double c[3], R[9], ax[3], mu; };

__global__ void k_phantom(const DevGeom g, const Ell* __restrict__ e, int n, float* __restrict__ vol, double bx,
                          double by, double bz)
{
    const long long MN = (long long)g.M * g.N, V = MN * g.Z;
    for (long long q = blockIdx.x * 256LL + threadIdx.x; q < V; q += (long long)gridDim.x * 256) {
        const int i = (int)(q % g.M), j = (int)((q / g.M) % g.N), k = (int)(q / MN);
        const double p0 = __dadd_rn(bx, __dmul_rn((double)g.vx, (double)i + 0.5));
        const double p1 = __dadd_rn(by, __dmul_rn((double)g.vy, (double)j + 0.5));
        const double p2 = __dadd_rn(bz, __dmul_rn((double)g.vz, (double)k + 0.5));
        double acc = 0.0;
        for (int a = 0; a < n; ++a) {
            const Ell& E = e[a];
            const double d0 = __dsub_rn(p0, E.c[0]), d1 = __dsub_rn(p1, E.c[1]), d2 = __dsub_rn(p2, E.c[2]);
            double r2 = 0.0;
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const double l = __ddiv_rn(__dadd_rn(__dadd_rn(__dmul_rn(E.R[b], d0), __dmul_rn(E.R[3 + b], d1)),
                                                     __dmul_rn(E.R[6 + b], d2)),
                                           E.ax[b]);
                r2 = __dadd_rn(r2, __dmul_rn(l, l));
            }
            if (r2 <= 1.0) acc = __dadd_rn(acc, E.mu);
        }
        vol[q] = (float)__dadd_rn((double)vol[q], acc);
    }
}

static void euler_zxz(const double* e, double Rm[9])
{
    const double cp = std::cos(e[0]), sp = std::sin(e[0]), ct = std::cos(e[1]), st = std::sin(e[1]),
                 cs = std::cos(e[2]), ss = std::sin(e[2]);
    Rm[0] = cp * cs - sp * ct * ss; Rm[1] = -cp * ss - sp * ct * cs; Rm[2] = sp * st;
    Rm[3] = sp * cs + cp * ct * ss; Rm[4] = -sp * ss + cp * ct * cs; Rm[5] = -cp * st;
    Rm[6] = st * ss;                Rm[7] = st * cs;                 Rm[8] = ct;
}

ctr_status launch_phantom(const Geometry& G, const double* params, int n, float* vol, cudaStream_t st)
{
    std::vector<Ell> h(n);
    for (int a = 0; a < n; ++a) {
        const double* q = params + 10 * a;
        for (int b = 0; b < 3; ++b) { h[a].c[b] = q[b]; h[a].ax[b] = q[3 + b]; }
        euler_zxz(q + 6, h[a].R);
        h[a].mu = q[9];
    }
    Ell* d = nullptr;
    CTR_CUDA_TRY(cudaMalloc(&d, sizeof(Ell) * (n > 0 ? n : 1)));
    cudaError_t e = cudaMemcpyAsync(d, h.data(), sizeof(Ell) * n, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        const ctr_geometry_desc& D = G.desc;
        const double bx = -(double)D.vx * ((double)D.nx / 2.0 + (double)D.m_offset);
        const double by = -(double)D.vy * ((double)D.ny / 2.0);
        const double bz = -(double)D.vz * ((double)D.nz / 2.0);
        k_phantom<<<148 * 16, 256, 0, st>>>(G.dg, d, n, vol, bx, by, bz);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    CTR_CUDA_TRY(e);
    return CTR_OK;
}

}  // namespace ctr
