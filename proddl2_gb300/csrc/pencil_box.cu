// The FFT form of the pencil stage on box grids (sizes per axis at run time):
// the choice of the kernel, and the unpaired one.
#include "pencil_lines.cuh"

namespace fftdock {

int box_pencil_classes(const int dims[3], int K, bool paired) {
    // two classes where the y size is even and the doubled line buffers fit;
    // with many terms an x bin holds too few entries to share their sums
    if ((K > 1 && !paired) || dims[1] % 2 != 0) return 1;
    return pencil_lines_smem_box(dims[0], dims[1], dims[2], K, 2, paired) <= kPencilMaxSmem ? 2 : 1;
}

cudaError_t box_pencil(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz, cudaStream_t s) {
    if (!a.lig_w32) return box_pencil_plain(a, twx, twy, twz, s);
    // two 256-thread CTAs per SM where their shared memory fits
    const int nx = a.box.n[0], ny = a.box.n[1], nz = a.box.n[2];
    const size_t sm = pencil_lines_smem_box(nx, ny, nz, a.K, a.qc, true) +
                      pencil_stage_bytes(nx, a.K, a.qc, a.n_ent, true);
    return a.qc == 1 || sm <= kPencilMaxSmem / 2 - 1024 ? box_pencil_paired(a, twx, twy, twz, s)
                                                        : box_pencil_paired_wide(a, twx, twy, twz, s);
}

cudaError_t box_pencil_plain(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz,
                             cudaStream_t s) {
    return a.qc == 2 ? launch_box_pencil<false, 2, kPencilThreads>(a, twx, twy, twz, s)
                     : launch_box_pencil<false, 1, kPencilThreads>(a, twx, twy, twz, s);
}

cudaError_t box_pencil_load() {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, (const void*)pencil_lines_kernel<0, float2, false, 1, kPencilThreads, 2>);
}

}  // namespace fftdock
