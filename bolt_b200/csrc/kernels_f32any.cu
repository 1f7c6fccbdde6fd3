// FP32 stage kernels on any grid (partial tiles and chunks, currents): the
// QG_ANY and QG_CURRENTS forms of qpair_kernel.cuh.
#include "launch.h"
#include "qpair_kernel.cuh"

namespace bolt {

cudaError_t launch_qpair_f32_any(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                            cudaStream_t st) {
    return launch_qpair_any<float, false>(a, bgk, recon, grid, smem, st);
}

}  // namespace bolt
