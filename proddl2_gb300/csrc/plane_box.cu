// The plane stage on box grids (sizes per axis at run time): launches of
// plane_lines_kernel<0, ..>.
#include "plane_lines.cuh"

namespace fftdock {

template <bool QUAD>
static cudaError_t launch(const BatchArgs& a, const float2* twy, const float2* twz, cudaStream_t s) {
    const int nx = a.box.n[0], ny = a.box.n[1], nz = a.box.n[2];
    PlanePlan pl{};
    if (!plane_plan(ny, nz, pl)) return cudaErrorInvalidValue;
    const size_t sm = plane_lines_smem(ny, nz);
    cudaError_t e = cudaFuncSetAttribute((const void*)plane_lines_kernel<0, QUAD>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    const int nxp = QUAD ? (nx + 3) / 4 * 4 : nx;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nxp, a.n_rot);
    cfg.blockDim = dim3(kPlaneThreads);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (QUAD) {
        // clusters of 4 CTAs along x (the planes of one x-quad)
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 4;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, plane_lines_kernel<0, QUAD>, (const float2*)(QUAD ? a.g2t : a.g2), twy, twz, pl,
                              nx, nxp, a.PP, a.cand_v, a.cand_i, a.dbg_corr);
}

cudaError_t box_plane(const BatchArgs& a, const float2* twy, const float2* twz, bool quad, cudaStream_t s) {
    return quad ? launch<true>(a, twy, twz, s) : launch<false>(a, twy, twz, s);
}

cudaError_t box_plane_load() {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, (const void*)plane_lines_kernel<0, false>);
}

}  // namespace fftdock
