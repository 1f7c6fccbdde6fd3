// FP64 stage kernel in the reference's operation order on 8x8 tiles: the fused
// RK stage of qpair_kernel.cuh, built with -fmad=false so that no multiply-add
// is contracted.  Same bits per value as the scalar stage kernel of
// kernels_f64.cu; grids off the tiles run the forms of kernels_f64exactany.cu.
#include "launch.h"
#include "qpair_kernel.cuh"

namespace bolt {

cudaError_t launch_qpair_f64exact(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                                  cudaStream_t st) {
    return launch_qpair<double, true, QG_TILES>(a, bgk, recon, grid, smem, st);
}

}  // namespace bolt
