// line_kernel.cuh - q-stage of 1D1V grids (sm_100a): one q2 cell, periodic in
// q2, one cell along p2 and p3.
//
// The same stage as qstage_kernel (df_dt_fvm.py:56-97 q-part and source, stage
// update of fvm_operator.py:26,33 / integrators.py:15-28, FP64 moments of the
// output) with the same operations per value; the q2 faces of a single periodic
// cell are equal, so their difference is exactly zero and is left out.
//
// These grids are small (8,192 cells in the smallest use) and a launch is one
// chain of latencies, so the work is cut for parallelism: a thread owns one p
// and R consecutive q-cells, loads their R + 6 values at once and walks R + 1
// faces in registers; nothing is staged in shared memory.  R is the largest of
// 1, 2, 4 that still fills the GPU (fewer faces computed twice).  The
// Maxwellian's parameters are worked out by one extra warp while the others
// load and reconstruct.
//
// What bounds it: the latency of one chain of loads, faces, exponential and
// reduction, then the host.  64 x 128 FP64 cells, RK2 and a density diagnostic per
// step: 49 us with 64-cell tiles (four CTAs, each walking its tile's faces one
// after another, 18 us a stage), 34 us here (33 us of it host time).
#pragma once

#include "fvm_kernels.cuh"

namespace bolt {

template <typename T, bool EXACT, int RECON, bool BGK, int R>
__global__ void __launch_bounds__(LINE_THREADS + 32)
line_kernel(const __grid_constant__ QStageArgs a) {
    __shared__ double qc[R][6];              // Maxwellian of the cells, 1 / (2 kB T)
    __shared__ double red[LINE_THREADS / 32][R][3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nt = blockDim.x - (BGK ? 32 : 0), nwarp = nt >> 5;
    const int Ng = a.Ng, Nq1 = a.Nq1, Np = a.Np;
    const int i0 = blockIdx.x * R;
    const int s = blockIdx.y / a.nsplit, split = blockIdx.y % a.nsplit;
    const int pb = split * a.chunks_per_split * PW;
    const int pe = min(Np, pb + a.chunks_per_split * PW);
    const long long rowstride = (long long)a.Ns * Np;
    const long long colstride = rowstride * a.Nq1g;
    const long long row0 = (long long)Ng * colstride + (long long)s * Np;
    const T* fs = static_cast<const T*>(a.fs) + row0;
    const T* base1 = static_cast<const T*>(a.base1);
    const T* base2 = static_cast<const T*>(a.base2);
    T* out1 = static_cast<T*>(a.out1);
    T* out2 = static_cast<T*>(a.out2);
    const T* tau_arr = static_cast<const T*>(a.tau_arr);
    const T c1 = T(a.c1), c2 = T(a.c2);
    const T inv_dq1 = T(1.0 / a.dq1);
    // (an infinite collision time: 0 and 0, which divide to 0)
    const double tau = isinf(a.tau) ? 0.0 : a.tau;
    const T inv_tau = T(1.0 / a.tau);
    const double p1s = a.sg.p1_start[s], dp1 = a.sg.dp1[s];
    const double V2 = a.sg.p2_start[s] + 0.5 * a.sg.dp2[s];
    const double V3 = a.sg.p3_start[s] + 0.5 * a.sg.dp3[s];
    const double mneg = -a.sg.mass[s];
    const bool want_mom = a.mom_out != nullptr;
    const bool border = a.periodic1 || a.periodic2 || a.peer_left || a.peer_right;
    const int ncell = min(R, Nq1 - i0);

    // column of each window cell; a stencil reaching past the array wraps
    // around it (af.shift), as it does for N_ghost < 3
    auto col = [&](int i) {
        int g = i + Ng;
        if (g < 0 || g >= a.Nq1g) g = ((g % a.Nq1g) + a.Nq1g) % a.Nq1g;
        return (long long)g * rowstride;
    };
    // q1 part of df/dt of the thread's cells at p, and their values
    T d[R], fc[R];
    auto faces = [&](int p) {
        const T v1 = T(p1s + (0.5 + p) * dp1);
        const bool right = v1 > T(0);
        const int first = i0 - (right ? 3 : 2);
        T y[R + 5];
#pragma unroll
        for (int t = 0; t < R + 5; ++t) y[t] = fs[col(first + t) + p];
        Weno5Side<T> S;
        S.set(right);
        FaceWalker<RECON, EXACT, T> W;
        T Fp = v1 * W.first(y[0], y[1], y[2], y[3], y[4], right, S);
#pragma unroll
        for (int c = 0; c < R; ++c) {
            const T Fn = v1 * W.next(y[c + 1], y[c + 2], y[c + 3], y[c + 4], y[c + 5], right, S);
            if constexpr (EXACT) d[c] = div_by(-(Fn - Fp), a.dq1, inv_dq1);
            else d[c] = (Fp - Fn) * inv_dq1;
            fc[c] = right ? y[c + 3] : y[c + 2];
            Fp = Fn;
        }
    };
    int p = pb + tid;
    if (BGK && warp == nwarp) {
        p = pe;                              // the parameter warp has no p
        if (lane < ncell) {
            bgk_cell_params(a, s, i0 + lane, 0, qc[lane]);
            qc[lane][5] = 1.0 / qc[lane][4];
        }
    }
    if (p < pe) faces(p);
    if (BGK) __syncthreads();

    double macc[R][3];
#pragma unroll
    for (int c = 0; c < R; ++c) macc[c][0] = macc[c][1] = macc[c][2] = 0.0;
    bool bad = false;
    while (p < pe) {
        const double V1 = p1s + (0.5 + p) * dp1;
        const double vsq = (V1 * V1 + V2 * V2) + V3 * V3;
#pragma unroll
        for (int c = 0; c < R; ++c) {
            if (c >= ncell) break;
            const long long g = row0 + (long long)(i0 + c + Ng) * rowstride + p;
            T kk = d[c];
            if (BGK) {
                // f0 of collision_operator.py:52-65
                const double* qq = qc[c];
                const double dv = V1 - qq[1];
                double fmb = qq[0] * exp(div_by(mneg * (dv * dv), qq[4], qq[5]));
                if (a.p_dim >= 2) {
                    const double d2 = V2 - qq[2];
                    fmb = fmb * exp(div_by(mneg * (d2 * d2), qq[4], qq[5]));
                }
                if (a.p_dim == 3) {
                    const double d3 = V3 - qq[3];
                    fmb = fmb * exp(div_by(mneg * (d3 * d3), qq[4], qq[5]));
                }
                if constexpr (EXACT) {
                    const double x = -(double(fc[c]) - fmb);
                    kk = kk + (tau_arr ? x / double(tau_arr[g]) : div_by(x, tau, inv_tau));
                } else {
                    const T itau = tau_arr ? T(1) / tau_arr[g] : inv_tau;
                    kk = kk + (T(fmb) - fc[c]) * itau;
                }
            }
            const T o1 = base1 ? base1[g] + kk * c1 : kk;
            if (out2) out2[g] = base2[g] + kk * c2;
            out1[g] = o1;
            const int ii = i0 + c;
            if (border) {
                write_ghost_images(out1, o1, ii, 0, s, p, Ng, Nq1, 1, a.Nq1g, a.Nq2g,
                                   a.periodic1, a.periodic2, rowstride, colstride, Np);
                if (a.peer_left && ii < Ng)
                    static_cast<T*>(a.peer_left)[g + (long long)Nq1 * rowstride] = o1;
                if (a.peer_right && ii >= Nq1 - Ng)
                    static_cast<T*>(a.peer_right)[g - (long long)Nq1 * rowstride] = o1;
            }
            bad |= !isfinite(o1);
            if (want_mom) {
                const double o = double(o1);
                macc[c][0] += o;
                macc[c][1] += o * V1;
                macc[c][2] += (0.5 * o) * vsq;
            }
        }
        p += nt;
        if (p < pe) faces(p);
    }
    if (bad && a.flag) atomicOr(a.flag, 1);
    if (!want_mom) return;
    if (warp < nwarp) {
#pragma unroll
        for (int c = 0; c < R; ++c)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double v = warp_sum(macc[c][q]);
                if (lane == 0) red[warp][c][q] = v;
            }
    }
    __syncthreads();
    if (tid < ncell) {
        double m0 = 0.0, m1 = 0.0, m4 = 0.0;
        for (int w = 0; w < nwarp; ++w) {
            m0 += red[w][tid][0];
            m1 += red[w][tid][1];
            m4 += red[w][tid][2];
        }
        const double mom[kNumMom] = {m0, m1, V2 * m0, V3 * m0, m4};
#pragma unroll
        for (int q = 0; q < kNumMom; ++q)
            a.mom_out[(((long long)split * kNumMom + q) * a.Ns + s) * Nq1 + i0 + tid] = mom[q];
    }
}

}  // namespace bolt
