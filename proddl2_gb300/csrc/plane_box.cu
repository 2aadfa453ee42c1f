// The plane stage on box grids (sizes per axis at run time): launches of
// plane_lines_kernel<0, ..>.
#include "plane_lines.cuh"

namespace fftdock {

// Threads per plane: 256, or 64 on small planes, whose passes have too few
// butterflies for more.  Plane stage, ms per 1000 rotations, 64 | 256 threads, from
// planes and (/) from x-quads: 8^3 0.26 | 0.42 / 0.15 | 0.29, 12 x 13 x 26 0.46 | 0.70 /
// 0.30 | 0.60, 12 x 24 x 26 0.33 | 0.49 / 0.21 | 0.42.  A lone rotation takes the same
// time up to about 400 values, then longer the longer the lines: 64 x 8 and 32 x 30
// 14 | 12 and 16 | 14 us, 169 x 26 51 | 14 us, which loses with 1000 rotations too
// (1.18 | 0.69 ms).
constexpr int kThreads = 256, kSmallThreads = 64;
constexpr int kSmallPlane = 400;  // complex values (ny hz)
static_assert(kSmallPlane <= 5400, "clusters start on larger planes");

template <int MODE, int NT> static cudaError_t launch(const BatchArgs& a, const float2* twy, const float2* twz, cudaStream_t s) {
    const int nx = a.box.n[0], ny = a.box.n[1], nz = a.box.n[2];
    PlanePlan pl{};
    if (!plane_plan(ny, nz, pl)) return cudaErrorInvalidValue;
    constexpr bool quad = MODE != kPlanePlanes;
    const int nxp = quad ? (nx + 3) / 4 * 4 : nx;
    return launch_planes<MODE>(&plane_lines_kernel<0, MODE, NT>, dim3(MODE == kPlaneQuadCluster ? nxp : nx, a.n_rot),
                               NT, plane_lines_smem(ny, nz), s, (const float2*)(quad ? a.g2t : a.g2), twy, twz, pl,
                               nx, nxp, a.PP, a.cand_v, a.cand_i, a.dbg_corr);
}

cudaError_t box_plane(const BatchArgs& a, const float2* twy, const float2* twz, bool quad, cudaStream_t s) {
    const int ny = a.box.n[1], nz = a.box.n[2];
    const bool small = ny * (nz / 2 + 1) <= kSmallPlane;
    if (!quad)
        return small ? launch<kPlanePlanes, kSmallThreads>(a, twy, twz, s) : launch<kPlanePlanes, kThreads>(a, twy, twz, s);
    if (plane_quad_mode(ny, nz) == kPlaneQuadCluster) return launch<kPlaneQuadCluster, kThreads>(a, twy, twz, s);
    return small ? launch<kPlaneQuad, kSmallThreads>(a, twy, twz, s) : launch<kPlaneQuad, kThreads>(a, twy, twz, s);
}

cudaError_t box_plane_load() {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, (const void*)plane_lines_kernel<0, kPlanePlanes, kThreads>);
    return e != cudaSuccess ? e : cudaFuncGetAttributes(&fa, (const void*)plane_lines_kernel<0, kPlanePlanes, kSmallThreads>);
}

}  // namespace fftdock
