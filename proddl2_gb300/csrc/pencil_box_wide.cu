// Box grids, ljComp: one 512-thread CTA per SM.
#include "pencil_lines.cuh"

namespace fftdock {

cudaError_t box_pencil_paired_wide(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz,
                                   cudaStream_t s) {
    return launch_box_pencil<true, 2, kPencilWideThreads>(a, twx, twy, twz, s);
}

}  // namespace fftdock
