// pstage_kernel.cuh - p-stage of a df/dt evaluation with fields (sm_100a).
//
//   k = k_q + (-((d1 + d2) + d3)),  d_a = (F_a(right) - F_a(left)) * (1/dp_a)
//
// (df_dt_fvm.py:245-323) with circular neighbours along each p axis and C_p
// from the cell-centred fields (advection_terms.py:147-188), then the RK
// combine and the FP64 moments of out1 (full sums: nsplit = 1).
//
// One CTA per (interior q-cell, species) holds the p-block in shared memory,
// rows of p1 at an odd pitch.  A thread walks a piece of one p-line: the
// acceleration C_a does not vary along its own axis, so a whole line has one
// upwind side, consecutive faces share the walker's smoothness indicators and
// four of five window values, and a face is computed once (plus one per
// piece).  The axes run one after another, each adding its divergence to an
// accumulator block in the reference's order ((d1 + d2) + d3); a last pass
// reads k_q and the bases in 16-byte vectors and combines.  Lanes walk
// neighbouring lines: axis 1 reads at the odd pitch and axes 2, 3 read
// consecutive p1, both without bank conflicts.
//
// What bounds it: instruction issue (shared-memory loads, indices and the face
// arithmetic), not memory.  64^2 x 32^2 cells, WENO5: a stage took 88 us in FP32 and
// 150 us in FP64 with every face worked out from scratch by one thread per cell,
// here 41 us and 85 us.  A minmod RK2 step of 32^2 x 20^3 FP32 cells went from
// 967 us to 283 us.
//
// FP32 threads walk two pieces of a line side by side as an f32x2 pair, except
// for WENO5: its walkers carry enough state that the pair's second set of
// pointers and the longer pieces cost more than the paired arithmetic saves (41 us
// a stage by single pieces, 44 us by pairs; minmod 105 us by single pieces, 94 us
// by pairs).
#pragma once

#include <type_traits>

#include "fvm_kernels.cuh"

namespace bolt {

// q / n and q % n for 0 <= q < 2^24 with n >= 1, from a float reciprocal
// and one correction step
struct PDiv {
    int n;
    float inv;
    __device__ __forceinline__ explicit PDiv(int nn) : n(nn), inv(1.0f / float(nn)) {}
    __device__ __forceinline__ int div(int q, int* rem) const {
        int d = __float2int_rz(float(q) * inv);
        int r = q - d * n;
        if (r < 0) { --d; r += n; }
        else if (r >= n) { ++d; r -= n; }
        *rem = r;
        return d;
    }
};

// 16-byte vectors of f and single values, as arrays of T
template <typename T, int VN> struct PVec;
template <> struct PVec<float, 4> {
    __device__ static void load(const float* p, float (&v)[4]) {
        const float4 u = *reinterpret_cast<const float4*>(p);
        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
    }
    __device__ static void store(float* p, const float (&v)[4]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <> struct PVec<double, 2> {
    __device__ static void load(const double* p, double (&v)[2]) {
        const double2 u = *reinterpret_cast<const double2*>(p);
        v[0] = u.x; v[1] = u.y;
    }
    __device__ static void store(double* p, const double (&v)[2]) {
        *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    }
};
template <typename T> struct PVec<T, 1> {
    __device__ static void load(const T* p, T (&v)[1]) { v[0] = *p; }
    __device__ static void store(T* p, const T (&v)[1]) { *p = v[0]; }
};

// Electrostatic E1 of cell ii of a periodic q-line: the FFT solve of fft.py:9-78
// is a circular convolution of the charge density with the Green's function G
// (sum_j G_j = 0), so E1_ii = sum_j G_{ii-j} (rho_j - rho_ii), a sum of small
// terms.  This thread's share of the sum.
__device__ __forceinline__ double line_field_part(const PStageArgs& a, int ii) {
    const int n = a.Nq1;
    auto rho = [&](int j) {
        double r = 0.0;
        for (int s = 0; s < a.Ns; ++s)
            r += a.sg.charge[s] * (a.mom_scale * (a.measure[s] * a.density[s * n + j]));
        return r;
    };
    const double own = rho(ii);
    double e = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x)
        e = fma(a.green[ii >= j ? ii - j : ii - j + n], rho(j) - own, e);
    return e;
}

// the periodic images of a q-cell's p-values c .. c + VN - 1 (as
// write_ghost_images, VN values at a time)
template <typename T, int VN>
__device__ __forceinline__ void store_images(const PStageArgs& a, T* out, const T (&v)[VN],
                                             int ii, int jj, long long sp, long long rowstride,
                                             long long colstride) {
    const int n1 = a.periodic1 ? (a.Ng + a.Nq1 - 1) / a.Nq1 : 0;
    const int n2 = a.periodic2 ? (a.Ng + a.Nq2 - 1) / a.Nq2 : 0;
    for (int t1 = -n1; t1 <= n1; ++t1) {
        const int g1 = ii + a.Ng + t1 * a.Nq1;
        if (g1 < 0 || g1 >= a.Nq1g) continue;
        for (int t2 = -n2; t2 <= n2; ++t2) {
            const int g2 = jj + a.Ng + t2 * a.Nq2;
            if (g2 < 0 || g2 >= a.Nq2g || (t1 == 0 && t2 == 0)) continue;
            PVec<T, VN>::store(out + g2 * colstride + g1 * rowstride + sp, v);
        }
    }
}

// the stage combine of one q-cell, VN consecutive p per step
template <typename T, int VN>
__device__ __forceinline__ bool pstage_combine(const PStageArgs& a, const T* fb, const T* acc,
                                               const double* vg, int pitch, int ii, int jj,
                                               int s, double (&macc)[kNumMom]) {
    const int tid = threadIdx.x, nt = blockDim.x;
    const int n1 = a.Np1, n2 = a.Np2;
    const long long rowstride = (long long)a.Ns * a.Np;
    const long long colstride = rowstride * a.Nq1g;
    const long long sp0 = (long long)s * a.Np;
    const long long cbase = (long long)(jj + a.Ng) * colstride +
                            (long long)(ii + a.Ng) * rowstride + sp0;
    T* out1 = static_cast<T*>(a.out1) + cbase;
    T* out2 = a.out2 ? static_cast<T*>(a.out2) + cbase : nullptr;
    const T* kq = static_cast<const T*>(a.kq) + cbase;
    // a base that is the stage input is the block already in shared memory
    const bool f1 = a.base1 == a.fs, f2 = a.base2 == a.fs;
    const T* base1 = a.base1 ? static_cast<const T*>(a.base1) + cbase : nullptr;
    const T* base2 = a.base2 ? static_cast<const T*>(a.base2) + cbase : nullptr;
    const T c1 = T(a.c1), c2 = T(a.c2);
    const bool ghost_cell = (a.periodic1 && (ii < a.Ng || ii >= a.Nq1 - a.Ng)) ||
                            (a.periodic2 && (jj < a.Ng || jj >= a.Nq2 - a.Ng));
    const double dp1 = a.sg.dp1[s];
    bool bad = false;
    constexpr int U = 2;                     // vectors whose loads are in flight together
    PCellWalk w(tid * VN, nt * VN, n1, n2);
    for (int c0 = tid * VN; c0 < a.Np; c0 += U * nt * VN) {
        T k[U][VN], b1[U][VN], b2[U][VN];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * nt * VN;
            if (c >= a.Np) break;
            PVec<T, VN>::load(kq + c, k[u]);
            if (base1 && !f1) PVec<T, VN>::load(base1 + c, b1[u]);
            if (out2 && !f2) PVec<T, VN>::load(base2 + c, b2[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * nt * VN;
            if (c >= a.Np) break;
            const int row = w.i3 * n2 + w.i2;
            const int q = row * pitch + w.i1;
            T o1[VN], o2[VN];
#pragma unroll
            for (int t = 0; t < VN; ++t) {
                if (f1) b1[u][t] = fb[q + t];
                if (f2) b2[u][t] = fb[q + t];
                const T kk = k[u][t] + (-acc[q + t]);
                o1[t] = base1 ? b1[u][t] + kk * c1 : kk;
                o2[t] = b2[u][t] + kk * c2;
                bad |= !isfinite(o1[t]);
            }
            PVec<T, VN>::store(out1 + c, o1);
            if (out2) PVec<T, VN>::store(out2 + c, o2);
            if (ghost_cell)
                store_images<T, VN>(a, static_cast<T*>(a.out1), o1, ii, jj, sp0 + c, rowstride,
                                    colstride);
            if (a.mom_out) {
                double ov[VN];
#pragma unroll
                for (int t = 0; t < VN; ++t) ov[t] = double(o1[t]);
                add_moment_run<VN>(ov, vg[w.i1], dp1, vg[n1 + w.i2], vg[n1 + n2 + w.i3], macc);
            }
            w.advance();
        }
    }
    return bad;
}

// Lane value and face walker of a p-line: FP64 walks one piece per thread with
// the reference-order faces, FP32 one (WENO5) or an f32x2 pair of pieces of the
// same line with the walkers of the paired q-stage kernel (twice the face value).
template <int RECON, typename T> struct PWalk;
template <int RECON> struct PWalk<RECON, double> {
    typedef double P;
    typedef Weno5Side<double> Side;
    FaceWalker<RECON, true, double> w;
    __device__ __forceinline__ P first(const P (&y)[5], bool right, const Side& S) {
        return w.first(y[0], y[1], y[2], y[3], y[4], right, S);
    }
    __device__ __forceinline__ P next(P y0, P y1, P y2, P y3, P y4, bool right, const Side& S) {
        return w.next(y0, y1, y2, y3, y4, right, S);
    }
    __device__ __forceinline__ static double scale(double C) { return C; }
};
template <int RECON> struct PWalk<RECON, float> {
    static constexpr bool WENO = RECON == BOLT_RECON_WENO5;
    typedef typename std::conditional<WENO, float, float2>::type P;
    typedef Weno5PairT<float, P> Side;
    typename std::conditional<
        RECON == BOLT_RECON_MINMOD, MinmodPairWalkerT<float>,
        typename std::conditional<
            RECON == BOLT_RECON_PPM, PpmPairWalkerT<float>,
            typename std::conditional<RECON == BOLT_RECON_PC, ConstPairWalkerT<float>,
                                      Weno5PairWalkerT<float, P, true>>::type>::type>::type w;
    __device__ __forceinline__ P first(const P (&y)[5], bool, const Side& S) {
        return w.first(y[0], y[1], y[2], y[3], y[4], S);
    }
    __device__ __forceinline__ P next(P y0, P y1, P y2, P y3, P y4, bool, const Side& S) {
        return w.next(y0, y1, y2, y3, y4, S);
    }
    __device__ __forceinline__ static float scale(float C) { return 0.5f * C; }
};

// the next value of a circular line of n elements: m the index of *p
template <typename T>
__device__ __forceinline__ T line_next(const T*& p, int& m, int n, int stride) {
    const T v = *p;
    p += stride;
    if (++m == n) {
        m = 0;
        p -= n * stride;
    }
    return v;
}

template <typename T, bool EXACT, int RECON>
__global__ void __launch_bounds__(PTHREADS_MAX, sizeof(T) == 4 ? 2 : 1)
pstage_kernel(const __grid_constant__ PStageArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int n1 = a.Np1, n2 = a.Np2, n3 = a.Np3;
    const int pitch = pstage_pitch(n1), block = pitch * n2 * n3;
    double* vg = reinterpret_cast<double*>(smem_raw);        // p-cell centres, p1 | p2 | p3
    T* fb = reinterpret_cast<T*>(vg + (n1 + n2 + n3));       // [n3][n2][pitch]
    T* acc = fb + block;                                     // divergence sum, same layout
    __shared__ double red[PTHREADS_MAX / 32][kNumMom];
    __shared__ double field[PTHREADS_MAX / 32];

    const int tid = threadIdx.x, nt = blockDim.x;
    const int ii = blockIdx.x % a.Nq1, jj = blockIdx.x / a.Nq1, s = blockIdx.y;
    const long long rowstride = (long long)a.Ns * a.Np;
    const long long colstride = rowstride * a.Nq1g;
    const T* fs = static_cast<const T*>(a.fs) + (long long)(jj + a.Ng) * colstride +
                  (long long)(ii + a.Ng) * rowstride + (long long)s * a.Np;
    constexpr int VW = 16 / (int)sizeof(T);
    if (a.vec) {
        PCellWalk w(tid * VW, nt * VW, n1, n2);
        for (int c = tid * VW; c < a.Np; c += nt * VW) {
            T v[VW];
            PVec<T, VW>::load(fs + c, v);
            T* d = fb + (w.i3 * n2 + w.i2) * pitch + w.i1;
#pragma unroll
            for (int t = 0; t < VW; ++t) d[t] = v[t];
            w.advance();
        }
    } else {
        PCellWalk w(tid, nt, n1, n2);
        for (int c = tid; c < a.Np; c += nt) {
            fb[(w.i3 * n2 + w.i2) * pitch + w.i1] = fs[c];
            w.advance();
        }
    }
    for (int q = tid; q < n1 + n2 + n3; q += nt) {
        if (q < n1) vg[q] = a.sg.p1_start[s] + (0.5 + q) * a.sg.dp1[s];
        else if (q < n1 + n2) vg[q] = a.sg.p2_start[s] + (0.5 + (q - n1)) * a.sg.dp2[s];
        else vg[q] = a.sg.p3_start[s] + (0.5 + (q - n1 - n2)) * a.sg.dp3[s];
    }
    const long long plane_g = (long long)a.Nq2g * a.Nq1g;
    const long long qg = (long long)(jj + a.Ng) * a.Nq1g + (ii + a.Ng);
    double E1 = a.cell[0 * plane_g + qg], E2 = a.cell[1 * plane_g + qg];
    const double E3 = a.cell[2 * plane_g + qg], B1 = a.cell[3 * plane_g + qg];
    const double B2 = a.cell[4 * plane_g + qg], B3 = a.cell[5 * plane_g + qg];
    const double em = a.sg.charge[s] / a.sg.mass[s];
    const PDiv D1(n1), D2(n2);
    if (a.green) {
        const double e = warp_sum(line_field_part(a, ii));
        if ((tid & 31) == 0) field[tid >> 5] = e;
    }
    __syncthreads();
    if (a.green) {
        double e = 0.0;
        for (int w = 0; w < nt / 32; ++w) e += field[w];
        E1 = e / a.eps;
        E2 = 0.0;
        if (s == 0)                          // the cell and its periodic images
            for (int t = tid; t < a.Nq2g; t += nt)
                for (int g = (ii + a.Ng) % a.Nq1; g < a.Nq1g; g += a.Nq1) {
                    a.cell_out[(long long)t * a.Nq1g + g] = E1;
                    a.cell_out[plane_g + (long long)t * a.Nq1g + g] = E2;
                }
    }

    // a single-cell axis contributes exactly zero; `term` keeps one axis alone
    typedef PWalk<RECON, T> Walk;
    typedef typename Walk::P P;
    constexpr int LN = LaneOf<P>::n;         // pieces a thread walks side by side
    bool first = true;
#pragma unroll 1
    for (int ax = 0; ax < 3; ++ax) {
        const int n = ax == 0 ? n1 : (ax == 1 ? n2 : n3);
        if (n == 1 || (a.term && a.term != ax + 1)) continue;
        const int lines = a.Np / n, seg = a.seg[ax], items = lines * seg;
        const int len = (n + LN * seg - 1) / (LN * seg);
        const int stride = ax == 0 ? 1 : (ax == 1 ? pitch : n2 * pitch);
        const T inv = T(1.0 / (ax == 0 ? a.sg.dp1[s] : (ax == 1 ? a.sg.dp2[s] : a.sg.dp3[s])));
        const PDiv DL(lines);
        for (int it = tid; it < items; it += nt) {
            // pieces sg and sg + seg of the line
            int line, base;
            const int sg = DL.div(it, &line);
            const int b = sg * len, e = min(n, b + len);
            if (b >= e) continue;
            // the line's first element and its acceleration
            double Cd;
            if (ax == 0) {
                int i2;
                const int i3 = D2.div(line, &i2);
                base = line * pitch;
                Cd = em * ((E1 + vg[n1 + i2] * B3) - vg[n1 + n2 + i3] * B2);
            } else {
                int i1;
                const int i = D1.div(line, &i1);
                base = i1 + i * (ax == 1 ? n2 * pitch : pitch);
                Cd = ax == 1 ? em * ((E2 + vg[n1 + n2 + i] * B1) - vg[i1] * B3)
                             : em * ((E3 + vg[i1] * B2) - vg[n1 + i] * B1);
            }
            const T C = T(Cd);
            const bool right = C > T(0);
            // window of the left face of cell i: cells i - 3 .. i + 1 (upwind from
            // the left), or i - 2 .. i + 2, circular
            const T* p[LN];
            int m[LN], cell[LN];
#pragma unroll
            for (int h = 0; h < LN; ++h) {
                cell[h] = b + h * seg * len;
                m[h] = cell[h] + (right ? -3 : -2);
                while (m[h] < 0) m[h] += n;
                while (m[h] >= n) m[h] -= n;          // an empty second piece
                p[h] = fb + base + m[h] * stride;
            }
            auto take = [&]() {
                P v;
#pragma unroll
                for (int h = 0; h < LN; ++h) comp(v, h) = line_next(p[h], m[h], n, stride);
                return v;
            };
            typename Walk::Side S;
            S.set(right);
            Walk W;
            P y[5];
#pragma unroll
            for (int t = 0; t < 5; ++t) y[t] = take();
            const P vC = LaneOf<P>::splat(Walk::scale(C));
            P Fprev = mul2(vC, W.first(y, right, S));
            T* al = acc + base + b * stride;
            const int other = seg * len * stride;     // from one piece's cell to the other's
            int left = e - b, left2 = n - cell[LN - 1];
            // pairs: five faces per round, the window rotates through its registers
            // (32^2 x 20^3 minmod: 281 us per RK2 step against 284 us unrolled by 4)
            constexpr int U = LN == 1 ? 1 : 5, ROUNDS = LN == 1 ? 4 : 1;
#pragma unroll ROUNDS
            while (left > 0) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (left <= 0) break;
                    const P v = take();
                    P Fn;
                    if constexpr (U == 1) {
                        y[0] = y[1]; y[1] = y[2]; y[2] = y[3]; y[3] = y[4]; y[4] = v;
                        Fn = W.next(y[0], y[1], y[2], y[3], y[4], right, S);
                    } else {
                        y[u] = v;
                        Fn = W.next(y[(u + 1) % 5], y[(u + 2) % 5], y[(u + 3) % 5],
                                    y[(u + 4) % 5], y[u], right, S);
                    }
                    Fn = mul2(vC, Fn);
                    P d = mul2(sub2(Fn, Fprev), LaneOf<P>::splat(inv));
                    Fprev = Fn;
#pragma unroll
                    for (int h = 0; h < LN; ++h) {
                        if (h && left2 <= 0) break;
                        T* q = al + h * other;
                        *q = first ? comp(d, h) : *q + comp(d, h);
                    }
                    al += stride;
                    --left;
                    --left2;
                }
            }
        }
        first = false;
        __syncthreads();
    }
    if (first) {                             // no active axis (or term of a single-cell axis)
        for (int c = tid; c < block; c += nt) acc[c] = T(0);
        __syncthreads();
    }
    if (a.term) {
        // one p-flux divergence (df_dt_fvm.py:325-335 term_to_return)
        T* out = static_cast<T*>(a.out1) + (fs - static_cast<const T*>(a.fs));
        PCellWalk w(tid, nt, n1, n2);
        for (int c = tid; c < a.Np; c += nt) {
            out[c] = acc[(w.i3 * n2 + w.i2) * pitch + w.i1];
            w.advance();
        }
        return;
    }
    double macc[kNumMom] = {0, 0, 0, 0, 0};
    const bool bad = a.vec ? pstage_combine<T, VW>(a, fb, acc, vg, pitch, ii, jj, s, macc)
                           : pstage_combine<T, 1>(a, fb, acc, vg, pitch, ii, jj, s, macc);
    if (bad && a.flag) atomicOr(a.flag, 1);
    if (a.mom_out) {
        const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
        for (int q = 0; q < kNumMom; ++q) {
            const double v = warp_sum(macc[q]);
            if (lane == 0) red[warp][q] = v;
        }
        __syncthreads();
        if (tid < kNumMom) {
            double v = 0.0;
            for (int w = 0; w < nt / 32; ++w) v += red[w][tid];
            const long long plane = (long long)a.Nq2 * a.Nq1;
            a.mom_out[((long long)tid * a.Ns + s) * plane + (long long)jj * a.Nq1 + ii] = v;
        }
    }
}

}  // namespace bolt
