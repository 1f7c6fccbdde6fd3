// FP64 stage kernels in the reference's operation order on any grid: the QG_ANY
// and QG_CURRENTS forms of qpair_kernel.cuh, built with -fmad=false.
#include "launch.h"
#include "qpair_kernel.cuh"

namespace bolt {

cudaError_t launch_qpair_f64exact_any(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                            cudaStream_t st) {
    return launch_qpair_any<double, true>(a, bgk, recon, grid, smem, st);
}

}  // namespace bolt
