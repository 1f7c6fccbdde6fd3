// launch.h - host-side launchers of the FVM kernels, one set per dtype.
// Implemented in kernels_f64.cu (FP64, reference operation order, no FMA
// contraction) and kernels_f32.cu (FP32 fast path).
#pragma once

#include <cuda_runtime.h>

#include "fvm_args.h"

namespace bolt {

enum Tiling { TILING_2D = 0, TILING_1D = 1, TILING_1D_Q2 = 2 };

struct TileShape {
    int tq1, tq2, q2;
};

inline TileShape tile_shape(int tiling) {
    switch (tiling) {
        case TILING_2D: return {8, 8, 1};
        case TILING_1D: return {64, 1, 0};
        default: return {64, 1, 1};
    }
}

// bytes of dynamic shared memory of the q-stage kernel
inline size_t qstage_smem(int tiling, size_t elem, int bgk, int bgk_direct, int ntab) {
    TileShape t = tile_shape(tiling);
    return qstage_layout(t.tq1, t.tq2, t.q2, (int)elem, bgk, bgk_direct, ntab).total;
}

// bytes of dynamic shared memory of the paired kernel (elem: 4 FP32, 8 FP64)
// (any: the form for any grid)
inline size_t qpair_smem(int ntab, int bgk, size_t elem, int any = 0) {
    return qpair_layout(ntab, bgk, (unsigned)elem, any).total;
}

// p-split of the q-stage grid (q-tiles x species x splits): the split that
// minimises (waves, rounded up) x (chunks per CTA + ~2 chunks of prologue), a
// wave being the GPU's SMs x the stage kernel's resident CTAs per SM (from its
// shared memory, at most 2).  Shared by the context and the allocation-free
// entry point.
struct PSplit {
    int nsplit, chunks_per_split;
};

inline PSplit choose_psplit(int nchunks, long long base_ctas, int sms, size_t smem_per_cta) {
    long long per_sm = 233472LL / (long long)(smem_per_cta + 1024);
    per_sm = per_sm < 1 ? 1 : (per_sm > 2 ? 2 : per_sm);
    const long long wave = (long long)(sms > 0 ? sms : 1) * per_sm;
    double best = 1e300;
    int best_cps = nchunks;
    for (int n = 1; n <= nchunks && n <= 64; ++n) {
        const int cps = (nchunks + n - 1) / n;
        const int ne = (nchunks + cps - 1) / cps;
        const long long waves = (base_ctas * ne + wave - 1) / wave;
        const double cost = (double)waves * (cps + 2.0);
        if (cost < best - 1e-9) {
            best = cost;
            best_cps = cps;
        }
    }
    return PSplit{(nchunks + best_cps - 1) / best_cps, best_cps};
}

// Launch shape of the 1D1V q-stage (line_kernel): q-cells per thread, p-threads
// per CTA, p-chunks of 32 per CTA.  R grows while the threads still fill about
// two warps per scheduler; the p-range of a q-cell is split over CTAs only while
// there are fewer than two CTAs per SM (each split is one more slot for the next
// stage's prologue to sum).
struct LineShape {
    int r, threads, chunks_per_split;
};

constexpr int kLineMaxR = 4;

inline LineShape choose_line(int Nq1, int Ns, int Np, int sms) {
    LineShape L;
    const long long cells = (long long)Nq1 * Ns * Np;
    L.r = 1;
    while (L.r < kLineMaxR && cells / (2 * L.r) >= (long long)sms * 256) L.r *= 2;
    L.threads = Np >= LINE_THREADS ? LINE_THREADS : (Np + 31) / 32 * 32;
    const int chunks = (Np + PW - 1) / PW, per_cta = L.threads / PW;
    const long long ctas = (long long)((Nq1 + L.r - 1) / L.r) * Ns;
    long long splits = (2LL * sms + ctas - 1) / ctas;
    const long long most = (chunks + per_cta - 1) / per_cta;
    if (splits > most) splits = most;
    L.chunks_per_split = (int)((chunks + splits - 1) / splits);
    return L;
}

// Whether the line kernel takes a 1D1V stage.  Larger grids fill the GPU with the
// scalar kernel's 64-cell tiles, which read f through shared memory; eight cells
// per thread were up to 1.8 times as slow as they are.  A CTA covers a whole row of
// p up to LINE_THREADS; there the line kernel's time goes by waves of CTAs
// (`resident` per SM), while the tiles' hardly grows in this range.  RK2 step with the
// source, FP32, tiles 29-33 us: one wave of four cells per thread 25 us, two 35-37 us; one
// wave of one or two cells 16-21 us, two 25-29 us, three 35-41 us.  FP64, tiles 37-45 us: the
// same waves 25, 37-41, 16-20, 29 and 37-41 us.  Without the source, tiles 16 us (FP64
// 21 us): up to three waves 12-16 us, four 18-21 us.  Longer rows keep to the line
// kernel: tiles 41-65 us, line 25-45 us.
inline bool line_fits(const LineShape& L, int Nq1, int Ns, int Np, int bgk, size_t elem,
                      int resident, int sms) {
    const long long lanes = (long long)Nq1 * Ns * ((Np + PW - 1) / PW * PW);
    if (lanes >= (long long)sms * 256 * 2 * kLineMaxR) return false;
    if (Np > LINE_THREADS || resident < 1) return true;
    const long long ctas = (long long)((Nq1 + L.r - 1) / L.r) * Ns;
    const long long waves = (ctas + (long long)resident * sms - 1) / ((long long)resident * sms);
    if (!bgk) return waves <= 3;
    return waves <= (elem == 4 ? 2 : 3) - (L.r == 4 ? 1 : 0);
}

// SM count of the current device (148 on B200 if the query fails)
inline int current_sm_count() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// p-blocks the p-stage takes: four blocks of values and the p-cell centres
// within 200 KB (6,250 FP64 or 12,600 FP32 p-cells)
inline bool pstage_fits(int Np, size_t elem, int ntab) {
    return ((4 * (size_t)Np * elem + 7) & ~(size_t)7) + (size_t)ntab * sizeof(double) <=
           200 * 1024;
}

// Launch shape of the p-stage kernel: threads per CTA (one q-cell) and the
// pieces each p-line is walked in.
struct PShape {
    int threads, seg[3];
    size_t smem;
};

// A thread's work on one axis is rounds x (piece + 3): a piece costs its cells
// and about three more for the walker's start; `pairs`: a thread walks two pieces
// side by side (seg counts the pairs).  The shape minimises thread-time
// of a CTA, scaled up while the SM holds fewer than 24 warps of this launch
// (latency not hidden): 2D blocks take the fewest threads that still fill the
// SM, small q-grids take as many threads as shorten the walk.  The three cells, the 24
// warps and the 1.5 per value are a model; registers, which admit fewer CTAs than
// shared memory does (64 each: two of 416 threads, not three), are not in it.
inline PShape choose_pshape(int n1, int n2, int n3, size_t elem, bool pairs, long long ctas,
                            int sms) {
    const int n[3] = {n1, n2, n3};
    const int Np = n1 * n2 * n3;
    const int lanes = pairs ? 2 : 1;
    PShape best;
    best.smem = 2 * (size_t)pstage_pitch(n1) * n2 * n3 * elem + (size_t)(n1 + n2 + n3) * 8;
    best.threads = 32;
    double best_cost = 1e300;
    const long long by_smem = 233472LL / (long long)(best.smem + 1024 + 640);
    for (int t = 32; t <= PTHREADS_MAX; t += 32) {
        if (t > 32 && t > Np) break;
        long long resident = by_smem < 1 ? 1 : by_smem;
        if (resident > 2048 / t) resident = 2048 / t;
        if (resident > 32) resident = 32;
        const long long have = (ctas + sms - 1) / sms;
        if (resident > have) resident = have;
        double cost = 1.5 * ((Np + t - 1) / t);
        int seg[3] = {1, 1, 1};
        for (int ax = 0; ax < 3; ++ax) {
            if (n[ax] == 1) continue;
            double c_best = 1e300;
            for (int s = 1; s <= n[ax]; ++s) {
                const int len = (n[ax] + lanes * s - 1) / (lanes * s);
                if (s > 1 && lanes * (s - 1) * len >= n[ax]) continue;
                const double c = (double)(((long long)Np / n[ax] * s + t - 1) / t) * (len + 3.0);
                if (c < c_best - 1e-9) {
                    c_best = c;
                    seg[ax] = s;
                }
            }
            cost += c_best;
        }
        const double warps = (double)resident * t / 32.0;
        const double total = cost * t * (warps < 24.0 ? 24.0 / warps : 1.0);
        if (total < best_cost - 1e-9) {
            best_cost = total;
            best.threads = t;
            for (int ax = 0; ax < 3; ++ax) best.seg[ax] = seg[ax];
        }
    }
    return best;
}

#define BOLT_DECLARE_LAUNCHERS(SUFFIX, T)                                                   \
    cudaError_t launch_qstage_##SUFFIX(const QStageArgs& a, int recon, int tiling, int bgk, \
                                       dim3 grid, size_t smem, cudaStream_t st);            \
    cudaError_t launch_line_##SUFFIX(const QStageArgs& a, int recon, int bgk,               \
                                     const LineShape& shape, cudaStream_t st);              \
    int line_resident_##SUFFIX(int recon, int bgk, const LineShape& shape);                 \
    cudaError_t launch_pstage_##SUFFIX(const PStageArgs& a, int recon, dim3 grid,           \
                                       int threads, size_t smem, cudaStream_t st);          \
    cudaError_t launch_moment_##SUFFIX(const void* f, int mid, double* out, int Ns,          \
                                       int Np1, int Np2, int Np3, int Nq1g, int Nq2g,        \
                                       const SpeciesGrid& sg, cudaStream_t st);             \
    cudaError_t launch_moments5_##SUFFIX(const void* f, double* part, int Ns, int Np1,       \
                                         int Np2, int Np3, int Nq1, int Nq2, int Ng,         \
                                         const SpeciesGrid& sg, cudaStream_t st);           \
    cudaError_t launch_ghost_##SUFFIX(void* f, const void* dl, const void* dr,               \
                                      const void* db, const void* dt, int Nq1, int Nq2,      \
                                      int Ng, int Ns, int Np, int Np1, int Np2, int per1,    \
                                      int per2, int dir1, int dir2, int mir1, int mir2,      \
                                      int ext1, int ext2, const SpeciesGrid& sg,             \
                                      const GhostShear& sh, cudaStream_t st);

// electrostatic field solve of one df/dt argument (poisson.cu)
struct PoissonArgs {
    const double* part;       // density partial sums [Ns][Nq2][Nq1] (moments5 split 0)
    double2* rho_hat;         // Nq2 x Nq1 complex work
    double2* e_hat;           // 2 x Nq2 x Nq1 complex work (E1, E2)
    double* cell;             // (6, Nq2g, Nq1g) cell-centred fields; E1, E2 written
    int Nq1, Nq2, Ng, Ns;
    double dq1, dq2, eps;
    double charge[kMaxSpecies], measure[kMaxSpecies];
    double mom_scale;         // the moments' factor: initial_mu on polar2D, else 1
};
int poisson_plans_create(int Nq1, int Nq2, int* fwd, int* inv);
void poisson_plans_destroy(int fwd, int inv);
cudaError_t launch_poisson(const PoissonArgs& a, int fwd, int inv, cudaStream_t st,
                           long long* launches);

BOLT_DECLARE_LAUNCHERS(f64, double)
BOLT_DECLARE_LAUNCHERS(f32, float)

// advective semi-Lagrangian step in q (asl_kernels.cuh): the interpolation of
// the interior at the feet of the characteristics, and the BGK source
cudaError_t launch_asl_q_f64(const AslArgs& a, int* flag, cudaStream_t st);
cudaError_t launch_asl_q_f32(const AslArgs& a, int* flag, cudaStream_t st);
cudaError_t launch_asl_src_f64(const QStageArgs& a, const void* in, const void* base, void* out,
                               double c, int mode, int* flag, double* mom_out, cudaStream_t st);
cudaError_t launch_asl_src_f32(const QStageArgs& a, const void* in, const void* base, void* out,
                               double c, int mode, int* flag, double* mom_out, cudaStream_t st);

// the whole RK2 step of the source, the p-block in shared memory
cudaError_t launch_asl_source_f64(const QStageArgs& a, const void* in, void* out, double dt,
                                  int* flag, cudaStream_t st);
cudaError_t launch_asl_source_f32(const QStageArgs& a, const void* in, void* out, double dt,
                                  int* flag, cudaStream_t st);

// paired q-stage (8x8 tiling, fused combine, TMA in and out): FP32, and FP64
// with FMA contraction and Newton-refined reciprocals (BOLT_F64_FAST)
cudaError_t launch_qpair_f32(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                             cudaStream_t st);
cudaError_t launch_qpair_f64(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                             cudaStream_t st);

// the same FP64 stage in the reference's operation order (BOLT_F64)
cudaError_t launch_qpair_f64exact(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                                  cudaStream_t st);

// any grid: partial tiles and chunks, and (a.want_j) currents; FP64 in the
// reference's operation order (both FP64 forms)
cudaError_t launch_qpair_f32_any(const QStageArgs& a, int bgk, int recon, dim3 grid, size_t smem,
                                 cudaStream_t st);
cudaError_t launch_qpair_f64exact_any(const QStageArgs& a, int bgk, int recon, dim3 grid,
                                      size_t smem, cudaStream_t st);

// FDTD sequence (FP64): prepare -> halo -> E -> halo -> B -> to_cell
cudaError_t launch_fdtd(const FieldArgs& a, cudaStream_t st, long long* launches);
cudaError_t launch_fdtd_part(const FieldArgs& a, int part, cudaStream_t st, long long* launches);
cudaError_t launch_field_halo(const FieldArgs& a, cudaStream_t st);

}  // namespace bolt
