// fdtd_kernels.cuh - Yee-grid FDTD kernels (FP64), included by kernels_f64.cu only.
#pragma once

#include "fvm_common.cuh"
#include "fvm_args.h"

namespace bolt {

// ---------------------------------------------------------------------------
// Yee-grid FDTD (fdtd_explicit.py:9-177, fields.py:527-647).  Field arrays are
// [6][Nq2g][Nq1g] FP64; af.shift(a,0,0,s1,s2) neighbours wrap over the ghosted
// extent like the reference's circular shifts.
// ---------------------------------------------------------------------------
// one cluster (the portable size) of large CTAs updates a whole field grid of up
// to kFieldClusterCells (ghosts included); on larger ones its eight SMs run out
// and a launch per pass over the whole GPU is faster.  An update of 64^2 cells: 15 us
// by the cluster, 27 us by launches; 120^2: 27 and 30 us; 128^2: 32 us each way;
// 200^2: 46 and 31 us; 250^2: 76 and 28 us.
constexpr int kFieldCluster = 8, kFieldThreads = 1024;
constexpr int kFieldClusterCells = 1 << 14;

// all threads of the cluster, their global memory accesses before it visible
// after it (not the .aligned form: the passes before it end in loops whose threads
// leave at different times)
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\t"
                 "barrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ int wrapi(int x, int n) { return ((x % n) + n) % n; }
// the circular neighbours of x in 0 .. n - 1
__device__ __forceinline__ int up(int x, int n) { return x + 1 == n ? 0 : x + 1; }
__device__ __forceinline__ int down(int x, int n) { return x == 0 ? n - 1 : x - 1; }

// a/b from r = 1/b (the spacings and eps are the same for every cell), an infinite
// quotient as the division gives it
__device__ __forceinline__ double field_div(double a, double b, double r) {
    const double q = a * r;
    return fabs(q) < INFINITY ? fma(fma(-b, q, a), r, q) : q;
}

// J from partial sums (or the caller's J); copy of the cell-centred E before the update
__device__ __forceinline__ void fdtd_prepare(const FieldArgs& a, int first, int step) {
    const int n = a.Nq1g * a.Nq2g;
    for (int t = first; t < n; t += step) {
        const int g1 = t % a.Nq1g, g2 = t / a.Nq1g;
        const int i = g1 - a.Ng, j = g2 - a.Ng;
        for (int c = 0; c < 3; ++c) {
            double v = 0.0;
            if (a.j_given) {
                v = a.j_given[c * n + t];
            } else if (i >= 0 && i < a.Nq1 && j >= 0 && j < a.Nq2) {
                // per species: charge * moment, the moment sum * measure
                // (times initial_mu on the polar2D grid); then the species sum
                for (int s = 0; s < a.Ns; ++s) {
                    double sum = 0.0;
#pragma unroll 4
                    for (int sp = 0; sp < a.nsplit; ++sp)
                        sum += a.jpart[(((long long)sp * 3 + c) * a.Ns + s) * a.Nq2 * a.Nq1
                                       + (long long)j * a.Nq1 + i];
                    const double mom = sum * a.measure[s];
                    v += a.charge[s] * (a.mom_scale * mom);
                }
            }
            a.J[c * n + t] = v;
            a.ebefore[c * n + t] = a.cell[c * n + t];
        }
    }
}

// periodic refresh of the 6 Yee components' halos (communicate_fields); the
// ghosts of an external axis (a block's cut), corners included, are the
// caller's: it exchanges them with the neighbouring blocks afterwards
__device__ __forceinline__ void fdtd_halo(const FieldArgs& a, int first, int step) {
    const int n = a.Nq1g * a.Nq2g;
    for (int t = first; t < n; t += step) {
        const int g1 = t % a.Nq1g, g2 = t / a.Nq1g;
        const int i = g1 - a.Ng, j = g2 - a.Ng;
        const bool in1 = i >= 0 && i < a.Nq1, in2 = j >= 0 && j < a.Nq2;
        if (in1 && in2) continue;
        if ((!in1 && a.ext1) || (!in2 && a.ext2)) continue;
        const int si = wrapi(i, a.Nq1) + a.Ng, sj = wrapi(j, a.Nq2) + a.Ng;
        for (int c = 0; c < 6; ++c) a.yee[c * n + t] = a.yee[c * n + sj * a.Nq1g + si];
    }
}

// E += (dt/(mu eps)) curl B - J dt / eps   (fdtd_explicit.py:29-66)
__device__ __forceinline__ void fdtd_e(const FieldArgs& a, int first, int step) {
    const int n = a.Nq1g * a.Nq2g;
    const double* B1 = a.yee + 3 * n;
    const double* B2 = a.yee + 4 * n;
    const double* B3 = a.yee + 5 * n;
    const double cf = a.dt / (a.mu * a.eps);
    const double r1 = 1.0 / a.dq1, r2 = 1.0 / a.dq2, re = 1.0 / a.eps;
    for (int t = first; t < n; t += step) {
        const int g1 = t % a.Nq1g, g2 = t / a.Nq1g;
        const int p1 = g2 * a.Nq1g + up(g1, a.Nq1g);     // shift(.., -1, 0)
        const int p2 = up(g2, a.Nq2g) * a.Nq1g + g1;     // shift(.., 0, -1)
        const double curl1 = field_div(B3[p2] - B3[t], a.dq2, r2);
        const double curl2 = field_div(-(B3[p1] - B3[t]), a.dq1, r1);
        const double curl3 = field_div(B2[p1] - B2[t], a.dq1, r1) -
                             field_div(B1[p2] - B1[t], a.dq2, r2);
        a.yee[0 * n + t] = a.yee[0 * n + t] +
                           (cf * curl1 - field_div(a.J[0 * n + t] * a.dt, a.eps, re));
        a.yee[1 * n + t] = a.yee[1 * n + t] +
                           (cf * curl2 - field_div(a.J[1 * n + t] * a.dt, a.eps, re));
        a.yee[2 * n + t] = a.yee[2 * n + t] +
                           (cf * curl3 - field_div(a.J[2 * n + t] * a.dt, a.eps, re));
    }
}

// B -= dt curl E   (fdtd_explicit.py:100-129)
__device__ __forceinline__ void fdtd_b(const FieldArgs& a, int first, int step) {
    const int n = a.Nq1g * a.Nq2g;
    const double* E1 = a.yee;
    const double* E2 = a.yee + n;
    const double* E3 = a.yee + 2 * n;
    const double r1 = 1.0 / a.dq1, r2 = 1.0 / a.dq2;
    for (int t = first; t < n; t += step) {
        const int g1 = t % a.Nq1g, g2 = t / a.Nq1g;
        const int m1 = g2 * a.Nq1g + down(g1, a.Nq1g);     // shift(.., 1, 0)
        const int m2 = down(g2, a.Nq2g) * a.Nq1g + g1;     // shift(.., 0, 1)
        const double curl1 = field_div(E3[t] - E3[m2], a.dq2, r2);
        const double curl2 = field_div(-(E3[t] - E3[m1]), a.dq1, r1);
        const double curl3 = field_div(E2[t] - E2[m1], a.dq1, r1) -
                             field_div(E1[t] - E1[m2], a.dq2, r2);
        a.yee[3 * n + t] = a.yee[3 * n + t] + -a.dt * curl1;
        a.yee[4 * n + t] = a.yee[4 * n + t] + -a.dt * curl2;
        a.yee[5 * n + t] = a.yee[5 * n + t] + -a.dt * curl3;
    }
}

// Yee -> cell centres; E becomes the average of the old and new values
// (the reference's three cell-centred arrays alias one object, so its
// E_at_n_plus_half write lands in the array that get_fields returns)
__device__ __forceinline__ void fdtd_to_cell(const FieldArgs& a, int first, int step) {
    const int n = a.Nq1g * a.Nq2g;
    const double* y = a.yee;
    for (int t = first; t < n; t += step) {
        const int g1 = t % a.Nq1g, g2 = t / a.Nq1g;
        const int p1 = g2 * a.Nq1g + up(g1, a.Nq1g);
        const int p2 = up(g2, a.Nq2g) * a.Nq1g + g1;
        const int p12 = up(g2, a.Nq2g) * a.Nq1g + up(g1, a.Nq1g);
        const double e1 = 0.5 * (y[0 * n + t] + y[0 * n + p1]);
        const double e2 = 0.5 * (y[1 * n + t] + y[1 * n + p2]);
        const double e3 = y[2 * n + t];
        a.cell[0 * n + t] = 0.5 * (a.ebefore[0 * n + t] + e1);
        a.cell[1 * n + t] = 0.5 * (a.ebefore[1 * n + t] + e2);
        a.cell[2 * n + t] = 0.5 * (a.ebefore[2 * n + t] + e3);
        a.cell[3 * n + t] = 0.5 * (y[3 * n + t] + y[3 * n + p2]);
        a.cell[4 * n + t] = 0.5 * (y[4 * n + t] + y[4 * n + p1]);
        a.cell[5 * n + t] = 0.25 * (((y[5 * n + t] + y[5 * n + p2]) + y[5 * n + p1]) + y[5 * n + p12]);
    }
}

__global__ void fdtd_prepare_kernel(FieldArgs a) {
    fdtd_prepare(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void fdtd_halo_kernel(FieldArgs a) {
    fdtd_halo(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void fdtd_e_kernel(FieldArgs a) {
    fdtd_e(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void fdtd_b_kernel(FieldArgs a) {
    fdtd_b(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void fdtd_to_cell_kernel(FieldArgs a) {
    fdtd_to_cell(a, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// The whole update as one cluster of CTAs: the same passes in the same order,
// the cluster barrier (release / acquire) between them instead of a launch each.
// What bounds it: the latency of the passes.  64^2 cells: six launches were 36 us
// of a 312 us step (FP32, 64^2 x 32^2), 301 us with this one; the kernel itself
// 26 us with IEEE divisions and index remainders, 20 us with reciprocals.
__global__ void __cluster_dims__(kFieldCluster, 1, 1) __launch_bounds__(kFieldThreads)
fdtd_step_kernel(FieldArgs a) {
    const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    fdtd_prepare(a, first, step);
    fdtd_halo(a, first, step);
    cluster_barrier();
    fdtd_e(a, first, step);
    cluster_barrier();
    fdtd_halo(a, first, step);
    cluster_barrier();
    fdtd_b(a, first, step);
    cluster_barrier();
    fdtd_to_cell(a, first, step);
}

}  // namespace bolt
