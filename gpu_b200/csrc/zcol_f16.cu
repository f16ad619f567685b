// zcol_f16.cu -- the z-column projector's kernels for __half volumes (zcol_fp.cuh).
#include "zcol_fp.cuh"

namespace ctr {

cudaError_t launch_zcol_f16(const Geometry& G, const void* vol, const void* lin, int view0, int nview,
                            void* out, ctr_dtype out_dt, cudaStream_t st)
{
    return launch_zcol_t<__half>(G, vol, lin, view0, nview, out, out_dt, st);
}

}  // namespace ctr
