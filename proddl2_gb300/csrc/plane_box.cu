// The plane stage on box grids (sizes per axis at run time): launches of
// plane_lines_kernel<0, ..>.
#include "plane_lines.cuh"

namespace fftdock {

constexpr int kThreads = 256;

template <int MODE> static cudaError_t launch(const BatchArgs& a, const float2* twy, const float2* twz, cudaStream_t s) {
    const int nx = a.box.n[0], ny = a.box.n[1], nz = a.box.n[2];
    PlanePlan pl{};
    if (!plane_plan(ny, nz, pl)) return cudaErrorInvalidValue;
    constexpr bool quad = MODE != kPlanePlanes;
    const int nxp = quad ? (nx + 3) / 4 * 4 : nx;
    return launch_planes<MODE>(&plane_lines_kernel<0, MODE, kThreads>, dim3(MODE == kPlaneQuadCluster ? nxp : nx, a.n_rot),
                               kThreads, plane_lines_smem(ny, nz), s, (const float2*)(quad ? a.g2t : a.g2), twy, twz, pl,
                               nx, nxp, a.PP, a.cand_v, a.cand_i, a.dbg_corr);
}

cudaError_t box_plane(const BatchArgs& a, const float2* twy, const float2* twz, bool quad, cudaStream_t s) {
    if (!quad) return launch<kPlanePlanes>(a, twy, twz, s);
    return plane_quad_mode(a.box.n[1], a.box.n[2]) == kPlaneQuad ? launch<kPlaneQuad>(a, twy, twz, s)
                                                                 : launch<kPlaneQuadCluster>(a, twy, twz, s);
}

cudaError_t box_plane_load() {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, (const void*)plane_lines_kernel<0, kPlanePlanes, kThreads>);
}

}  // namespace fftdock
