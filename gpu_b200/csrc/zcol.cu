// zcol.cu -- the z-column copy of a volume and the projection on it.
#include "zcol_fp.cuh"

namespace ctr {

// Linear [z][y][x] -> z-columns [y][x][z]: 32x32 (x, z) tiles through shared
// memory, one y per grid layer.  Values are moved, not converted.
static constexpr int ZT = 32, ZT_ROWS = 8;
template <typename T>
__global__ void __launch_bounds__(ZT * ZT_ROWS)
k_to_zcol(int M, int N, int Z, int zs, const T* __restrict__ src, T* __restrict__ dst)
{
    __shared__ T t[ZT][ZT + 1];
    const int i0 = blockIdx.x * ZT, k0 = blockIdx.y * ZT, j = blockIdx.z;
    const int a = threadIdx.x % ZT, r = threadIdx.x / ZT;
#pragma unroll
    for (int q = r; q < ZT; q += ZT_ROWS)
        if (i0 + a < M && k0 + q < Z) t[q][a] = src[((long long)(k0 + q) * N + j) * M + i0 + a];
    __syncthreads();
#pragma unroll
    for (int q = r; q < ZT; q += ZT_ROWS)
        if (i0 + q < M && k0 + a < Z) dst[((long long)j * M + i0 + q) * zs + k0 + a] = t[a][q];
}

size_t forward_zcol_bytes(const Geometry& G, ctr_dtype vdt)
{
    const size_t es = dtype_size(vdt);
    return (size_t)G.dg.M * G.dg.N * zcol_stride(G.dg, es) * es;
}

// Whether the rows that meet the volume fill the blocks' row lanes.  The path's
// time over the general projector's, per row that meets the volume, is about
// c_list x (rows of the blocks) + c_walk x (lanes of the warps with such rows):
// the lists are built for every block, the warps walk for their rows.  With 4
// columns a block c = 0.16, 0.56, with longer lists 0.52, 0.2 (an idle warp costs
// more there: 2 of 8 warps walk 64 rows).  General / here, ms, 512^2 x rows
// voxels and rows, 1024 columns, 4.6e9 steps: 4 rows 4.2 / 28.6, 16 rows 4.2 / 7.2, 24
// 4.2 / 4.8, 32 4.2 / 3.7, 40 4.2 / 4.6, 48 4.2 / 3.8, 64 4.2 / 2.9, 72 (of 64
// slices) 4.2 / 4.3, 96 4.3 / 3.7; 1024^2, 2048 columns: 32 rows 4.3 / 11.1, 64
// 8.3 / 10.2, 96 12.4 / 10.9, 128 16.4 / 11.5, 160 20.3 / 21.2, 192 24.3 / 21.5; 512^2 x
// 4 slices under 64 rows 0.65 / 4.3.
static bool zf_rows_fill(const Geometry& G)
{
    const DevGeom& g = G.dg;
    const int wc = zf_columns(g), per = 32 * (ZF_WARPS / wc);
    const double blocks = (double)((g.ZP + per - 1) / per) * per, lanes = (double)((G.rows_in + 31) / 32) * 32;
    const double cost = wc == 4 ? 0.16 * blocks + 0.56 * lanes : 0.52 * blocks + 0.2 * lanes;
    return cost <= 0.97 * G.rows_in;
}

// Where the z-column path is the faster one (ms here / on the linear volume),
// its cost counted in rays times x and y planes ("steps"):
// * a call pays for its lists and copy, and the first one maps the scratch
//   (0.9 ms for 37 MB, 3.7 ms for 512 MB), which it should win back: 4.5e9 steps,
//   and 120 a voxel.  426x424x288, 5 views (1.1e9) 0.93 / 0.83; 301x259x211, 60
//   views (4.2e9) 2.95 / 3.10, but a first call 3.95 / 3.17; 256^3, 64 views
//   (4.8e9) 3.39 / 4.61; 512^3, 32 views (2.6e10) 15.8 / 24.5;
// * short rays do not repay a list: 480 x and y planes (200x180x150, 60 views
//   1.12 / 1.06);
// * with 16-bit voxels and the reference's sums a step converts two voxels and
//   gains less: 415x383x299 2.49 / 2.33; 496x532x514 5.95 / 7.09;
// * a detector column's list is built once for all the rows of a block, and its
//   rows are the lanes of the warps: see zf_rows_fill;
// * the scratch is no more than the pool keeps between calls (columns of a few
//   voxels are padded to many times their size).
bool forward_zcol_fits(const Geometry& G, ctr_dtype vdt, int nview)
{
    const DevGeom& g = G.dg;
    if (g.entry64 || g.N > 65535 || (g.Z + ZT - 1) / ZT > 65535 || zf_smem(g, 2) > ZF_SMEM ||
        (long long)g.M * g.N * zcol_stride(g, 2) > 2147483647LL || !zf_rows_fill(G) ||
        forward_zcol_bytes(G, vdt) > pool_kept_bytes(G))
        return false;
    const double steps = (double)nview * (double)G.npix() * (g.M + g.N);
    return g.M + g.N >= (vdt == CTR_F32 || g.fast_sums ? 480 : 900) && steps >= 4.5e9 && steps >= 120.0 * (double)G.nvox();
}

ctr_status forward_zcol(const Geometry& G, const void* vol, ctr_dtype vdt, void* scratch, void* out, ctr_dtype out_dt,
                        int view0, int nview, cudaStream_t st)
{
    const DevGeom& g = G.dg;
    const int zs = zcol_stride(g, dtype_size(vdt));
    const dim3 grid((g.M + ZT - 1) / ZT, (g.Z + ZT - 1) / ZT, g.N);
    if (dtype_size(vdt) == 4)
        k_to_zcol<uint32_t><<<grid, ZT * ZT_ROWS, 0, st>>>(g.M, g.N, g.Z, zs, (const uint32_t*)vol, (uint32_t*)scratch);
    else
        k_to_zcol<uint16_t><<<grid, ZT * ZT_ROWS, 0, st>>>(g.M, g.N, g.Z, zs, (const uint16_t*)vol, (uint16_t*)scratch);
    CTR_CUDA_TRY(cudaGetLastError());
    const size_t view_bytes = (size_t)G.npix() * dtype_size(out_dt);
    for (int c = 0; c < nview; c += 65535) {
        const int n = std::min(65535, nview - c);
        void* o = (char*)out + (size_t)c * view_bytes;
        cudaError_t e = cudaErrorInvalidValue;
        if (vdt == CTR_F32) e = launch_zcol_f32(G, scratch, vol, view0 + c, n, o, out_dt, st);
        else if (vdt == CTR_BF16) e = launch_zcol_bf16(G, scratch, vol, view0 + c, n, o, out_dt, st);
        else if (vdt == CTR_F16) e = launch_zcol_f16(G, scratch, vol, view0 + c, n, o, out_dt, st);
        CTR_CUDA_TRY(e);
    }
    return CTR_OK;
}

}  // namespace ctr
