// Box grids, ljComp: two 256-thread CTAs per SM.
#include "pencil_lines.cuh"

namespace fftdock {

cudaError_t box_pencil_paired(const BatchArgs& a, const float2* twx, const float2* twy, const float2* twz,
                              cudaStream_t s) {
    return a.qc == 2 ? launch_box_pencil<true, 2, kPencilThreads>(a, twx, twy, twz, s)
                     : launch_box_pencil<true, 1, kPencilThreads>(a, twx, twy, twz, s);
}

}  // namespace fftdock
