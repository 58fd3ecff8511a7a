// FP64 pair arithmetic of the direct sum and the FP64 near field.
//
// The GPU's FP64 pipe issues 2 multiply-adds per clock and SM (64 times fewer
// than FP32), so an FP64 pair kernel is bound by the number of FP64
// instructions per pair and by nothing else.  For multipole orders <= 2 and
// field orders <= 2 the field is therefore written with dot products instead
// of the Cartesian tensor: with the source polynomials
//   A_0 = Mc_0, A_1(R) = sum_{|s|=1} Mc_s R^s + tr, A_2(R) = sum_{|s|=2} Mc_s R^s
// (tr = Mc_xx + Mc_yy + Mc_zz) and d g_j / d R_a = R_a g_{j+1},
//   F_0    = S_0,                  S_k = sum_i g_{i+k} A_i
//   F_a    = R_a S_1 + V0_a,       Vk_a = sum_i g_{i+k} dA_i / dR_a
//   F_ab   = delta_ab S_1 + R_a U_b + R_b U_a + W_ab,  U_a = V1_a + R_a S_2 / 2,
//   W_ab   = g_2 d^2 A_2 / dR_a dR_b.
// The diagonal is summed as halves, R_a U_a + W_aa / 2, beside one sum of S_1
// for all three (finish_f64).
// Quadrupole sources come as "near rows" (near_rows below): the off-diagonal
// second moments halved (exact) and tr as an extra row, so that with
// h = grad A_2 / 2 the terms are A_2 = R . h and 2 g_2 h.  FP64 instructions
// per undamped pair (m = 2): 47 at f = 1 and 74 at f = 2, against 126 and
// about 240 of the tensor recursion and full contraction (which orders above
// 2 keep, pair.cuh).
#pragma once

#include "pair.cuh"

namespace fmm {

// Whether (m, f) takes the dot-product form (and, for m = 2, near rows).
__host__ __device__ constexpr bool near_rows(int m, int f) { return m <= 2 && f <= 2; }
// Rows of source coefficients per particle.
__host__ __device__ constexpr int near_row_count(int m, int f) { return nT(m) + (m == 2 && f <= 2 ? 1 : 0); }

// Accumulators of the field: its components and, with the diagonal in halves,
// the sum of S_1.
__host__ __device__ constexpr int acc_count(int m, int f) { return nT(f) + (near_rows(m, f) && f == 2 ? 1 : 0); }

// The field's components from the accumulators (of any part of the sum).
template <int M, int F>
__device__ __forceinline__ void finish_f64(const double* acc, double* fld) {
#pragma unroll
    for (int f = 0; f < nT(F); ++f) fld[f] = acc[f];
    if constexpr (acc_count(M, F) > nT(F)) {
        constexpr double w = M == 0 ? 1.0 : 2.0;
        fld[4] = fma(w, acc[4], acc[10]);
        fld[7] = fma(w, acc[7], acc[10]);
        fld[9] = fma(w, acc[9], acc[10]);
    }
}

// Beyond these the damped numerators round to the undamped ones for every
// order up to 6: e^-u q_6(u) / 11!! < 2^-62 from u = (a r)^3 = 60 (AMOEBA),
// e^-x P_6(x) / 11!! < 2^-59 from x = a r = 60 (Thole), and e^-s s^(11/2) / 11!!
// < 2^-63 from s = a r^2 = 60 (erf).
constexpr float kFarDamp = 60.0f;

// g_0..g_N of radial_g_ir in FP64.  A pair beyond the damping range, tested in
// FP32 (off the FP64 pipe), takes the undamped chain.
template <int N>
__device__ __forceinline__ void radial_g_f64(int damp, double r2, double ir, double a, double* g) {
    bool far = damp == DAMP_NONE;
    if (damp != DAMP_NONE) {
        const float af = f32_bits(a), r2f = f32_bits(r2);
        const float x = damp == DAMP_ERF ? af * r2f : af * sqrtf(r2f);
        far = (damp == DAMP_AMOEBA ? x * x * x : x) > kFarDamp * 1.001f;
    }
    if (far) {
        const double ir2 = ir * ir;
        g[0] = ir;
#pragma unroll
        for (int j = 1; j <= N; ++j) g[j] = -(double)(2 * j - 1) * g[j - 1] * ir2;
        if (damp == DAMP_AMOEBA) g[0] = 0.0;
    } else {
        radial_g_ir<N, double>(damp, r2, ir, a, g);
    }
}

// acc += field of the source rows mc at R from g (see the head of the file).
template <int M, int F>
__device__ __forceinline__ void contract_f64(double X, double Y, double Z, const double* g, const double* mc, int damp,
                                             double* acc) {
    static_assert(near_rows(M, F), "dot-product form");
    const double R[3] = {X, Y, Z};
    double A1 = 0.0, A2 = 0.0, h[3] = {0.0, 0.0, 0.0}, g2d = 0.0;
    if constexpr (M == 1) A1 = fma(mc[1], X, fma(mc[2], Y, mc[3] * Z));
    if constexpr (M == 2) {
        A1 = fma(mc[1], X, fma(mc[2], Y, fma(mc[3], Z, mc[10])));
        h[0] = fma(mc[4], X, fma(mc[5], Y, mc[6] * Z));
        h[1] = fma(mc[5], X, fma(mc[7], Y, mc[8] * Z));
        h[2] = fma(mc[6], X, fma(mc[8], Y, mc[9] * Z));
        A2 = fma(X, h[0], fma(Y, h[1], Z * h[2]));
        g2d = g[2] + g[2];
    }
    // AMOEBA: g_0 = 0, which leaves NaN of infinite charges and NaN
    if (damp != DAMP_AMOEBA || (__double2hiint(mc[0]) & 0x7ff00000) == 0x7ff00000) acc[0] = fma(mc[0], g[0], acc[0]);
    if constexpr (M >= 1) acc[0] = fma(A1, g[1], acc[0]);
    if constexpr (M >= 2) acc[0] = fma(A2, g[2], acc[0]);
    if constexpr (F >= 1) {
        double S1 = mc[0] * g[1];
        if constexpr (M >= 1) S1 = fma(A1, g[2], S1);
        if constexpr (M >= 2) S1 = fma(A2, g[3], S1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = fma(R[c], S1, acc[1 + c]);
            if constexpr (M >= 1) v = fma(mc[1 + c], g[1], v);
            if constexpr (M >= 2) v = fma(h[c], g2d, v);
            acc[1 + c] = v;
        }
        if constexpr (F == 2) {
            double S2 = mc[0] * g[2];
            if constexpr (M >= 1) S2 = fma(A1, g[3], S2);
            if constexpr (M >= 2) S2 = fma(A2, g[4], S2);
            const double S2h = M == 0 ? S2 : 0.5 * S2;
            double U[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if constexpr (M == 0) {
                    U[c] = R[c] * S2h;  // (charges: whole components)
                } else {
                    double v = mc[1 + c] * g[2];
                    if constexpr (M == 2) v = fma(h[c], g[3] + g[3], v);
                    U[c] = fma(R[c], S2h, v);
                }
            }
            acc[10] += S1;
            // components xx, xy, xz, yy, yz, zz
            constexpr int ca[6] = {0, 0, 0, 1, 1, 2}, cb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                double v = fma(R[ca[q]], U[cb[q]], acc[4 + q]);
                if (M > 0 && ca[q] != cb[q]) v = fma(R[cb[q]], U[ca[q]], v);
                if constexpr (M == 2) v = fma(mc[4 + q], ca[q] == cb[q] ? g[2] : g2d, v);
                acc[4 + q] = v;
            }
        }
    }
}

// Field of one source (rows mc) at displacement target - source, into acc_count
// accumulators.
template <int M, int F>
__device__ __forceinline__ void pair_field_f64(double dx, double dy, double dz, double a, int damp, const double* mc,
                                               double* acc) {
    if constexpr (near_rows(M, F)) {
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        double g[M + F + 1];
        radial_g_f64<M + F>(damp, r2, rsqrt_f64(r2), a, g);
        contract_f64<M, F>(dx, dy, dz, g, mc, damp, acc);
    } else {
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        double g[M + F + 1], T[nT(M + F)];
        radial_g_f64<M + F>(damp, r2, rsqrt_f64(r2), a, g);
        md_tensor<M + F, double>(dx, dy, dz, g, T);
        contract<M, F, double>(T, mc, acc);
    }
}

// Sum of the warp's NF values per lane over its lanes.  Each exchange halves
// the values a lane keeps (NF - 1 + few FP64 additions instead of 5 NF).
// Returns whether this lane holds a total: component *f, in a[0].
template <int NF>
__device__ __forceinline__ bool warp_totals(double (&a)[NF], int lane, int* f) {
    int lo = 0, hi = NF, n = NF, plain = 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const bool up = (lane & off) != 0;
        if (n == 1) {
            a[0] += __shfl_xor_sync(0xffffffffu, a[0], off);
            plain |= off;
        } else {
            const int h = (n + 1) / 2;
#pragma unroll
            for (int i = 0; i < (NF + 1) / 2; ++i) {
                if (i < h) {
                    const double b = i + h < n ? a[i + h < NF ? i + h : 0] : 0.0;
                    const double send = up ? a[i] : b, keep = up ? b : a[i];
                    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
            if (up)
                lo = min(lo + h, hi);
            else
                hi = min(lo + h, hi);
            n = h;
        }
    }
    *f = lo;
    return (lane & plain) == 0 && lo < hi;
}

}  // namespace fmm
