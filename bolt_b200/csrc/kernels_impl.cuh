// kernels_impl.cuh - instantiation switchboard shared by kernels_f64.cu and
// kernels_f32.cu.  Define BOLT_T, BOLT_EXACT and BOLT_SUFFIX before including.
#pragma once

#include "launch.h"
#include "fvm_kernels.cuh"
#include "pstage_kernel.cuh"
#include "line_kernel.cuh"
#include "asl_kernels.cuh"

namespace bolt {

#define BOLT_CAT2(a, b) a##b
#define BOLT_CAT(a, b) BOLT_CAT2(a, b)

template <int RECON, int TQ1, int TQ2, bool Q2, bool BGK>
static cudaError_t qlaunch(const QStageArgs& a, dim3 grid, size_t smem, cudaStream_t st) {
    auto k = qstage_kernel<BOLT_T, BOLT_EXACT, RECON, TQ1, TQ2, Q2, BGK>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    k<<<grid, NTHREADS, smem, st>>>(a);
    return cudaGetLastError();
}

template <int RECON>
static cudaError_t qdispatch(const QStageArgs& a, int tiling, int bgk, dim3 grid, size_t smem,
                             cudaStream_t st) {
    if (tiling == TILING_2D)
        return bgk ? qlaunch<RECON, 8, 8, true, true>(a, grid, smem, st)
                   : qlaunch<RECON, 8, 8, true, false>(a, grid, smem, st);
    if (tiling == TILING_1D)
        return bgk ? qlaunch<RECON, 64, 1, false, true>(a, grid, smem, st)
                   : qlaunch<RECON, 64, 1, false, false>(a, grid, smem, st);
    return bgk ? qlaunch<RECON, 64, 1, true, true>(a, grid, smem, st)
               : qlaunch<RECON, 64, 1, true, false>(a, grid, smem, st);
}

cudaError_t BOLT_CAT(launch_qstage_, BOLT_SUFFIX)(const QStageArgs& a, int recon, int tiling,
                                                  int bgk, dim3 grid, size_t smem,
                                                  cudaStream_t st) {
    switch (recon) {
        case BOLT_RECON_PC: return qdispatch<BOLT_RECON_PC>(a, tiling, bgk, grid, smem, st);
        case BOLT_RECON_MINMOD: return qdispatch<BOLT_RECON_MINMOD>(a, tiling, bgk, grid, smem, st);
        case BOLT_RECON_PPM: return qdispatch<BOLT_RECON_PPM>(a, tiling, bgk, grid, smem, st);
        default: return qdispatch<BOLT_RECON_WENO5>(a, tiling, bgk, grid, smem, st);
    }
}

template <int RECON, bool BGK>
static void (*pick_line(int r))(QStageArgs) {
    switch (r) {
        case 1: return line_kernel<BOLT_T, BOLT_EXACT, RECON, BGK, 1>;
        case 2: return line_kernel<BOLT_T, BOLT_EXACT, RECON, BGK, 2>;
        default: return line_kernel<BOLT_T, BOLT_EXACT, RECON, BGK, 4>;
    }
}

static void (*pick_line(int recon, int bgk, int r))(QStageArgs) {
    switch (recon) {
        case BOLT_RECON_PC: return bgk ? pick_line<BOLT_RECON_PC, true>(r)
                                       : pick_line<BOLT_RECON_PC, false>(r);
        case BOLT_RECON_MINMOD: return bgk ? pick_line<BOLT_RECON_MINMOD, true>(r)
                                           : pick_line<BOLT_RECON_MINMOD, false>(r);
        case BOLT_RECON_PPM: return bgk ? pick_line<BOLT_RECON_PPM, true>(r)
                                        : pick_line<BOLT_RECON_PPM, false>(r);
        default: return bgk ? pick_line<BOLT_RECON_WENO5, true>(r)
                            : pick_line<BOLT_RECON_WENO5, false>(r);
    }
}

cudaError_t BOLT_CAT(launch_line_, BOLT_SUFFIX)(const QStageArgs& a, int recon, int bgk,
                                                const LineShape& shape, cudaStream_t st) {
    const dim3 grid((a.Nq1 + shape.r - 1) / shape.r, a.Ns * a.nsplit);
    pick_line(recon, bgk, shape.r)<<<grid, shape.threads + (bgk ? 32 : 0), 0, st>>>(a);
    return cudaGetLastError();
}

// CTAs of the line kernel that an SM holds (0: unknown)
int BOLT_CAT(line_resident_, BOLT_SUFFIX)(int recon, int bgk, const LineShape& shape) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pick_line(recon, bgk, shape.r),
                                                      shape.threads + (bgk ? 32 : 0), 0) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <int RECON>
static cudaError_t plaunch(const PStageArgs& a, dim3 grid, int threads, size_t smem,
                           cudaStream_t st) {
    auto k = pstage_kernel<BOLT_T, BOLT_EXACT, RECON>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    // all of the SM's shared memory: it holds the blocks of more CTAs than the
    // default split of it with L1 does (12 of 64^2 x 32^2 FP32)
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    k<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t BOLT_CAT(launch_pstage_, BOLT_SUFFIX)(const PStageArgs& a, int recon, dim3 grid,
                                                  int threads, size_t smem, cudaStream_t st) {
    switch (recon) {
        case BOLT_RECON_PC: return plaunch<BOLT_RECON_PC>(a, grid, threads, smem, st);
        case BOLT_RECON_MINMOD: return plaunch<BOLT_RECON_MINMOD>(a, grid, threads, smem, st);
        case BOLT_RECON_PPM: return plaunch<BOLT_RECON_PPM>(a, grid, threads, smem, st);
        default: return plaunch<BOLT_RECON_WENO5>(a, grid, threads, smem, st);
    }
}

cudaError_t BOLT_CAT(launch_moment_, BOLT_SUFFIX)(const void* f, int mid, double* out, int Ns,
                                                  int Np1, int Np2, int Np3, int Nq1g, int Nq2g,
                                                  const SpeciesGrid& sg, cudaStream_t st) {
    dim3 grid(Nq1g * Nq2g, Ns);
    auto k = Np1 * Np2 * Np3 > 256 ? moment_kernel<BOLT_T, true> : moment_kernel<BOLT_T, false>;
    k<<<grid, 256, 0, st>>>(static_cast<const BOLT_T*>(f), mid, out, Ns, Np1,
                             Np2, Np3, Nq1g, Nq2g, sg);
    return cudaGetLastError();
}

cudaError_t BOLT_CAT(launch_moments5_, BOLT_SUFFIX)(const void* f, double* part, int Ns, int Np1,
                                                    int Np2, int Np3, int Nq1, int Nq2, int Ng,
                                                    const SpeciesGrid& sg, cudaStream_t st) {
    dim3 grid(Nq1 * Nq2, Ns);
    moments5_kernel<BOLT_T><<<grid, 256, 0, st>>>(static_cast<const BOLT_T*>(f), part, Ns, Np1,
                                                  Np2, Np3, Nq1, Nq2, Ng, sg);
    return cudaGetLastError();
}

cudaError_t BOLT_CAT(launch_ghost_, BOLT_SUFFIX)(void* f, const void* dl, const void* dr,
                                                 const void* db, const void* dt, int Nq1, int Nq2,
                                                 int Ng, int Ns, int Np, int Np1, int Np2,
                                                 int per1, int per2, int dir1, int dir2,
                                                 int mir1, int mir2, int ext1, int ext2,
                                                 const SpeciesGrid& sg, const GhostShear& sh,
                                                 cudaStream_t st) {
    const long long Nq1g = Nq1 + 2 * Ng;
    const long long ncells = 2LL * Ng * Nq1g + 2LL * Ng * Nq2;
    if (ncells == 0) return cudaSuccess;
    // one CTA per ghost cell (grid-stride beyond 16 CTAs per SM), its threads
    // over the cell's (species, p) block
    const long long rowlen = (long long)Ns * Np;
    const long long blocks = ncells < 148 * 16 ? ncells : 148 * 16;
    const int threads = rowlen >= 2048 ? 256 : (rowlen >= 512 ? 128 : 64);
    ghost_kernel<BOLT_T><<<(unsigned)blocks, threads, 0, st>>>(
        static_cast<BOLT_T*>(f), static_cast<const BOLT_T*>(dl), static_cast<const BOLT_T*>(dr),
        static_cast<const BOLT_T*>(db), static_cast<const BOLT_T*>(dt), Nq1, Nq2, Ng, Ns, Np, Np1,
        Np2, per1, per2, dir1, dir2, mir1, mir2, ext1, ext2, sg, sh, ncells);
    return cudaGetLastError();
}

cudaError_t BOLT_CAT(launch_asl_q_, BOLT_SUFFIX)(const AslArgs& a, int* flag, cudaStream_t st) {
    constexpr int R = AslRows<BOLT_T>::R;
    const long long total = (long long)((a.Nq2 + R - 1) / R) * a.Ns * a.Np;   // threads
    if (total == 0) return cudaSuccess;
    // 32-bit element offsets when the ghosted array has fewer than 2^31 elements
    const long long elems = (long long)(a.Nq2 + 2 * a.Ng) * (a.Nq1 + 2 * a.Ng) * a.Ns * a.Np;
    if (elems < (1LL << 31))
        asl_q_kernel<BOLT_T, int><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a, flag);
    else
        asl_q_kernel<BOLT_T, long long><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a, flag);
    return cudaGetLastError();
}

cudaError_t BOLT_CAT(launch_asl_src_, BOLT_SUFFIX)(const QStageArgs& a, const void* in,
                                                   const void* base, void* out, double c,
                                                   int mode, int* flag, double* mom_out,
                                                   cudaStream_t st) {
    dim3 grid(a.Nq1 * a.Nq2, a.Ns);
    asl_src_kernel<BOLT_T><<<grid, 256, 0, st>>>(a, in, base, out, c, mode, flag, mom_out);
    return cudaGetLastError();
}

cudaError_t BOLT_CAT(launch_asl_source_, BOLT_SUFFIX)(const QStageArgs& a, const void* in,
                                                      void* out, double dt, int* flag,
                                                      cudaStream_t st) {
    auto k = asl_source_kernel<BOLT_T>;
    const unsigned smem = asl_source_smem(a.Np, a.Np1 + a.Np2 + a.Np3, sizeof(BOLT_T));
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<dim3(a.Nq1 * a.Nq2, a.Ns), 256, smem, st>>>(a, in, out, dt, flag);
    return cudaGetLastError();
}

}  // namespace bolt
