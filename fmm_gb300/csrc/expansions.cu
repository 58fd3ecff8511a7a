// Reference-mode M2L (FP64): the reference's own closed-form tensors with the
// int32 Cnij table (src/tensors_recursive.F90:29-135), L_f(i) += sum_s
// (-1)^(|s|+1) M'_s(j) T_{s+f}(c_i - c_j) (src/fmm.F90:826-882), with M'_s =
// M_s / s! the scaled moments of translate.cu.
//
// Up to order 2p = 10 no coefficient wraps: the closed form is the exact tensor
// up to rounding, and the reduced-basis M2L of the exact modes (m2l.cu,
// m2l_gemm.cu) gives the reference's result.  Above, the tensors are not
// harmonic; they are evaluated once per displacement group and multiplied over
// all Cartesian components (m2l_gemm.cu, m2l_tc64.cuh), or per pair where the
// groups hold a pair or two each (k_m2l_f64).  66,666 water molecules, p = 6
// (9.3e5 far pairs): 136.7 ms when every pair had its own closed form.
#include <algorithm>
#include <vector>

#include "internal.h"
#include "pair.cuh"

namespace fmm {

namespace {

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

constexpr int kMaxNPL = (nT(kMaxP) + 31) / 32;  // per-lane accumulators

__device__ __forceinline__ int pack_comp(int q) { return comp_x(q) | (comp_y(q) << 8) | (comp_z(q) << 16); }
__device__ __forceinline__ int cx_(int c) { return c & 0xff; }
__device__ __forceinline__ int cy_(int c) { return (c >> 8) & 0xff; }
__device__ __forceinline__ int cz_(int c) { return (c >> 16) & 0xff; }

__device__ __forceinline__ void fill_comp(int* sh, int nq) {
    for (int q = threadIdx.x; q < nq; q += blockDim.x) sh[q] = pack_comp(q);
}

// ---------------------------------------------------------------- M2L
// One warp per target node; sources of its far list in turn.  The tensor of
// orders <= 2p is built in shared memory, either by the Hermite recursion
// (exact) or by the reference's closed form with its Cnij table (ref mode,
// terms prepared on the host, evaluated in the reference's operation order).
__device__ __forceinline__ double ipow_rn(double x, int m) {
    unsigned nn = (unsigned)m;
    double y = (nn % 2) ? x : 1.0;
    while (nn >>= 1) {
        x = __dmul_rn(x, x);
        if (nn % 2) y = __dmul_rn(y, x);
    }
    return y;
}

// The tensor T_c(X, Y, Z) of every component c < nT(N) in the warp's shared
// memory: the reference's closed form with its Cnij table (ref) or the Hermite
// recursion (exact).  Returns TA or TB, whichever holds the result.
__device__ double* warp_tensor(double X, double Y, double Z, int N, int ref, const int* __restrict__ comp,
                               double* TA, double* TB, double* gsh, double* yp, double* zp, double* ir,
                               const int32_t* __restrict__ term_off, const uchar4* __restrict__ term_abc,
                               const double* __restrict__ term_c, int lane) {
    const int nqT = nT(N);
    double* T;
    if (ref) {
        const double R = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(X, X), __dmul_rn(Y, Y)), __dmul_rn(Z, Z)));
        if (lane < 3) {
            const double v = lane == 0 ? X : (lane == 1 ? Y : Z);
            double* pw = lane == 0 ? gsh : (lane == 1 ? yp : zp);
            const double u = __ddiv_rn(v, R);
            pw[0] = 1.0;
            for (int a = 1; a <= N; ++a) pw[a] = __dmul_rn(pw[a - 1], u);
        }
        for (int k = lane; k <= N; k += 32) ir[k] = __ddiv_rn(1.0, ipow_rn(R, k + 1));
        __syncwarp();
        for (int c = lane; c < nqT; c += 32) {
            double a = 0.0;
            for (int tt = term_off[c]; tt < term_off[c + 1]; ++tt) {
                const uchar4 e = term_abc[tt];
                const double Cx = __dmul_rn(term_c[3 * tt], gsh[e.x]);
                const double Cy = __dmul_rn(__dmul_rn(Cx, term_c[3 * tt + 1]), yp[e.y]);
                a = __dadd_rn(a, __dmul_rn(__dmul_rn(Cy, term_c[3 * tt + 2]), zp[e.z]));
            }
            TA[c] = __dmul_rn(a, ir[order_of(c)]);
        }
        __syncwarp();
        T = TA;
    } else {
        const double r2 = X * X + Y * Y + Z * Z;
        const double rinv = rsqrt(r2);
        const double rinv2 = rinv * rinv;
        if (lane <= N) {
            // g_j = (-1)^j (2j-1)!! r^-(2j+1)
            double v = rinv, c = 1.0;
            for (int jj = 1; jj <= lane; ++jj) {
                v *= rinv2;
                c *= -(double)(2 * jj - 1);
            }
            gsh[lane] = c * v;
        }
        __syncwarp();
        // level N holds only g_N; descend to level 0
        double* A = TA;
        double* B = TB;
        if (lane == 0) A[0] = gsh[N];
        __syncwarp();
        for (int lev = N - 1; lev >= 0; --lev) {
            const int lim = nT(N - lev);
            for (int c = lane; c < lim; c += 32) {
                double v;
                if (c == 0) {
                    v = gsh[lev];
                } else {
                    const int cc = comp[c];
                    const int tx = cx_(cc), ty = cy_(cc), tz = cz_(cc);
                    if (tx > 0) {
                        v = X * A[pidx(tx - 1, ty, tz)];
                        if (tx > 1) v += (double)(tx - 1) * A[pidx(tx - 2, ty, tz)];
                    } else if (ty > 0) {
                        v = Y * A[pidx(tx, ty - 1, tz)];
                        if (ty > 1) v += (double)(ty - 1) * A[pidx(tx, ty - 2, tz)];
                    } else {
                        v = Z * A[pidx(tx, ty, tz - 1)];
                        if (tz > 1) v += (double)(tz - 1) * A[pidx(tx, ty, tz - 2)];
                    }
                }
                B[c] = v;
            }
            __syncwarp();
            double* tmp = A;
            A = B;
            B = tmp;
        }
        T = A;
    }
    return T;
}

__global__ void k_m2l_f64(const TreeDev t, const double* __restrict__ mom, double* __restrict__ loc, int p, int ref,
                          const int32_t* __restrict__ term_off, const uchar4* __restrict__ term_abc,
                          const double* __restrict__ term_c) {
    extern __shared__ double smem[];
    const int nq = nT(p), N = 2 * p, nqT = nT(N);
    int* comp = reinterpret_cast<int*>(smem);
    double* base = smem + (nqT + 1) / 2 + 1;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per_warp = 2 * nqT + nq + 5 * (N + 1);
    double* TA = base + wib * per_warp;
    double* TB = TA + nqT;
    double* ms = TB + nqT;
    double* gsh = ms + nq;     // g_j, or x powers in ref mode
    double* yp = gsh + (N + 1);
    double* zp = yp + (N + 1);
    double* ir = zp + (N + 1);
    fill_comp(comp, nqT);
    __syncthreads();
    const int i = blockIdx.x * (blockDim.x >> 5) + wib;
    if (i >= t.num_nodes) return;
    const double cxi = t.cx[i], cyi = t.cy[i], czi = t.cz[i];
    const int q0 = t.far_off[i], q1 = t.far_off[i + 1];
    int fcomp[kMaxNPL];
#pragma unroll
    for (int r = 0; r < kMaxNPL; ++r) fcomp[r] = (lane + 32 * r < nq) ? comp[lane + 32 * r] : 0;
    double acc[kMaxNPL];
#pragma unroll
    for (int r = 0; r < kMaxNPL; ++r) acc[r] = 0.0;
    for (int q = q0; q < q1; ++q) {
        const int j = t.far_src[q];
        const double X = __dsub_rn(cxi, t.cx[j]);
        const double Y = __dsub_rn(cyi, t.cy[j]);
        const double Z = __dsub_rn(czi, t.cz[j]);
        for (int s = lane; s < nq; s += 32) {
            const double v = mom[(size_t)src_node(t, j) * nq + s];
            ms[s] = ((order_of(s) + 1) % 2) ? -v : v;  // (-1)^(|s|+1) M'_s
        }
        double* T = warp_tensor(X, Y, Z, N, ref, comp, TA, TB, gsh, yp, zp, ir, term_off, term_abc, term_c, lane);
        // contraction: L_f += sum_s ms_s T_{s+f}
#pragma unroll
        for (int r = 0; r < kMaxNPL; ++r) {
            if (lane + 32 * r < nq) {
                const int fx = cx_(fcomp[r]), fy = cy_(fcomp[r]), fz = cz_(fcomp[r]);
                double a = 0.0;
                for (int s = 0; s < nq; ++s) {
                    const int cs = comp[s];
                    a += ms[s] * T[pidx(cx_(cs) + fx, cy_(cs) + fy, cz_(cs) + fz)];
                }
                acc[r] += a;
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < kMaxNPL; ++r) {
        const int fq = lane + 32 * r;
        if (fq < nq) loc[(size_t)i * nq + fq] = acc[r];
    }
}


size_t comp_bytes(int nq) { return sizeof(double) * ((nq + 1) / 2 + 1); }

// Terms of the reference's closed-form tensors (src/tensors_recursive.F90:29-62)
// for all components of order <= N, with the int32 Cnij table of
// src/tensors_recursive.F90:64-93 (two's-complement wrap).
void build_ref_terms(int N, std::vector<int32_t>& off, std::vector<uchar4>& abc, std::vector<double>& coef) {
    const int maxo = N, d1 = maxo + 2, d0 = 2 * maxo + 3;
    std::vector<int32_t> C((size_t)d0 * d1 * d1, 0);
    auto at = [&](int nn, int ii, int jj) { return ((size_t)(nn - 1) * d1 + ii) * d1 + jj; };
    for (int nn = 1; nn <= d0; ++nn) C[at(nn, 0, 0)] = 1;
    for (int nn = 1; nn <= d0; ++nn) {
        if (nn % 2 == 0) continue;
        for (int ii = 1; ii <= maxo + 1; ++ii) {
            int k = (ii % 2 != 0) ? ii - 1 : ii;
            for (int jj = 0; jj <= ii; ++jj) {
                if ((ii + jj) % 2 != 0) continue;
                if (jj == 0) {
                    C[at(nn, ii, jj)] = C[at(nn, ii - 1, jj + 1)];
                } else if (jj != ii) {
                    uint32_t a = (uint32_t)(jj + 1) * (uint32_t)C[at(nn, ii - 1, jj + 1)];
                    uint32_t b = (uint32_t)(nn + k) * (uint32_t)C[at(nn, ii - 1, jj - 1)];
                    C[at(nn, ii, jj)] = (int32_t)(a - b);
                    k += 2;
                } else {
                    C[at(nn, ii, jj)] = (int32_t)(0u - (uint32_t)(nn + k) * (uint32_t)C[at(nn, ii - 1, jj - 1)]);
                }
            }
        }
    }
    off.assign(1, 0);
    abc.clear();
    coef.clear();
    for (int nn = 0; nn <= N; ++nn)
        for (int kx = nn; kx >= 0; --kx)
            for (int ky = nn - kx; ky >= 0; --ky) {
                const int kz = nn - kx - ky;
                for (int a = 0; a <= kx; ++a) {
                    const int32_t c1 = C[at(1, kx, a)];
                    if (c1 == 0) continue;
                    for (int b = 0; b <= ky; ++b) {
                        const int32_t c2 = C[at(a + kx + 1, ky, b)];
                        if (c2 == 0) continue;
                        for (int c = 0; c <= kz; ++c) {
                            const int32_t c3 = C[at(a + kx + b + ky + 1, kz, c)];
                            if (c3 == 0) continue;
                            abc.push_back(make_uchar4((unsigned char)a, (unsigned char)b, (unsigned char)c, 0));
                            coef.push_back((double)c1);
                            coef.push_back((double)c2);
                            coef.push_back((double)c3);
                        }
                    }
                }
                off.push_back((int32_t)abc.size());
            }
}

int set_smem(const void* fn, size_t bytes) {
    if (bytes > 48 * 1024) FMM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return FMM_OK;
}

}  // namespace

// Closed-form tensor terms of the reference at order N (ref mode), once per order.
int ensure_ref_terms(Workspace& ws, int N, cudaStream_t st) {
    if (ws.term_order == N) return FMM_OK;
    std::vector<int32_t> off;
    std::vector<uchar4> abc;
    std::vector<double> coef;
    build_ref_terms(N, off, abc, coef);
    FMM_TRY(ws.term_off.ensure(sizeof(int32_t) * off.size()));
    FMM_TRY(ws.term_abc.ensure(sizeof(uchar4) * std::max<size_t>(1, abc.size())));
    FMM_TRY(ws.term_c.ensure(sizeof(double) * std::max<size_t>(1, coef.size())));
    FMM_CUDA_TRY(cudaMemcpyAsync(ws.term_off.p, off.data(), sizeof(int32_t) * off.size(), cudaMemcpyHostToDevice, st));
    FMM_CUDA_TRY(cudaMemcpyAsync(ws.term_abc.p, abc.data(), sizeof(uchar4) * abc.size(), cudaMemcpyHostToDevice, st));
    FMM_CUDA_TRY(cudaMemcpyAsync(ws.term_c.p, coef.data(), sizeof(double) * coef.size(), cudaMemcpyHostToDevice, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    ws.term_order = N;
    return FMM_OK;
}

namespace {

// Whether the reference's int32 coefficients of order N are the exact ones:
// they reach 2^31 first at N = 11.
constexpr int kExactRefOrder = 10;

// Warp per displacement group: the closed-form tensor at the displacement in
// units of the coarser cell's half-width, the group's order and unit ratios.
__global__ void k_group_tensor_ref(int ng, const int32_t* __restrict__ gstart, const int32_t* __restrict__ svals,
                                   const int32_t* __restrict__ tgt, const TreeDev t, int p, int ldT,
                                   const int32_t* __restrict__ term_off, const uchar4* __restrict__ term_abc,
                                   const double* __restrict__ term_c, double* __restrict__ gT,
                                   int32_t* __restrict__ gq, float2* __restrict__ gab) {
    extern __shared__ double smem[];
    const int N = 2 * p, nqT = nT(N);
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* TA = smem + wib * (nqT + 4 * (N + 1));
    double* gsh = TA + nqT;
    double* yp = gsh + (N + 1);
    double* zp = yp + (N + 1);
    double* ir = zp + (N + 1);
    const int g = blockIdx.x * (blockDim.x >> 5) + wib;
    if (g >= ng) return;
    const int pos0 = svals[gstart[g]];
    const int i = tgt[pos0], j = t.far_src[pos0];
    const double hi = t.r[i], hj = t.r[j], hc = fmax(hi, hj);
    const double X = (t.cx[i] - t.cx[j]) / hc, Y = (t.cy[i] - t.cy[j]) / hc, Z = (t.cz[i] - t.cz[j]) / hc;
    const double* T = warp_tensor(X, Y, Z, N, 1, nullptr, TA, nullptr, gsh, yp, zp, ir, term_off, term_abc, term_c,
                                  lane);
    for (int c = lane; c < nqT; c += 32) gT[(size_t)g * ldT + c] = T[c];
    if (lane == 0) {
        gq[g] = p;
        gab[g] = make_float2((float)(hi / hc), (float)(hj / hc));
    }
}

}  // namespace

int launch_group_tensor_ref(Workspace& ws, const TreeDev& t, int ng, const int32_t* tgt, int p, int ldT,
                            cudaStream_t st) {
    const int N = 2 * p;
    FMM_TRY(ensure_ref_terms(ws, N, st));
    const size_t per_warp = sizeof(double) * (nT(N) + 4 * (N + 1));
    const int wpb = (int)std::max<size_t>(1, std::min<size_t>(4, (100 * 1024) / per_warp));
    FMM_TRY(set_smem((const void*)k_group_tensor_ref, wpb * per_warp));
    count_launches(1);
    k_group_tensor_ref<<<grid_for(ng, wpb), 32 * wpb, wpb * per_warp, st>>>(
        ng, ws.m2l_gstart.as<int32_t>(), ws.m2l_vals2.as<int32_t>(), tgt, t, p, ldT, ws.term_off.as<int32_t>(),
        ws.term_abc.as<uchar4>(), ws.term_c.as<double>(), ws.m2l_T.as<double>(), ws.m2l_gq.as<int32_t>(),
        ws.m2l_gab.as<float2>());
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

// M2L pair by pair on the CUDA cores (FP64), ref or exact tensors.
static int launch_m2l_pairwise(Workspace& ws, const TreeDev& t, int p, const Modes& md, cudaStream_t st) {
    const int nq = nT(p), N = 2 * p, nqT = nT(N);
    FMM_TRY(ws.loc.ensure(sizeof(double) * (size_t)t.num_nodes * nq));
    const int ref = md.coef_mode == 0 ? 1 : 0;
    if (ref) FMM_TRY(ensure_ref_terms(ws, N, st));
    const int per_warp = 2 * nqT + nq + 5 * (N + 1);
    int wpb = (int)std::max<size_t>(1, std::min<size_t>(4, (100 * 1024) / (sizeof(double) * per_warp)));
    const size_t sm = comp_bytes(nqT) + sizeof(double) * wpb * per_warp;
    FMM_TRY(set_smem((const void*)k_m2l_f64, sm));
    count_launches(1);
    k_m2l_f64<<<grid_for(t.num_nodes, wpb), 32 * wpb, sm, st>>>(t, ws.mom.as<double>(), ws.loc.as<double>(), p, ref,
                                                                ws.term_off.as<int32_t>(), ws.term_abc.as<uchar4>(),
                                                                ws.term_c.as<double>());
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int launch_m2l(Workspace& ws, const TreeDev& t, int p, const Modes& md, cudaStream_t st) {
    int rc;
    if (md.coef_mode != 0 || 2 * p <= kExactRefOrder) {
        rc = launch_m2l_reduced(ws, t, p, md.precision == 1 || md.precision == 3, md.coef_mode == 0 || t.nimg > 1, st);
    } else {
        FMM_TRY(ws.loc.ensure(sizeof(double) * (size_t)t.num_nodes * nT(p)));
        rc = launch_m2l_grouped(ws, t, p, false, st, true, true);
    }
    return rc == FMM_ENOTSUP ? launch_m2l_pairwise(ws, t, p, md, st) : rc;
}

// ---------------------------------------------------------------- periodic
// The lattice beyond the 27 explicit images (src/fmm.F90:884-952), for the
// root's local expansion.  Level multipoles, scaled like the cell moments
// (M'_t = M_t / t!): S_0 is the root's with its charge removed (the
// reference forces charge neutrality), and S_l = S_(l-1) plus the 26 copies
// of S_(l-1) shifted by H (3^(l-1) a), a != 0, in the reference's order of a.
// One block with a warp per copy (each copy's moments, then per component the
// sum over the copies in order): the levels are a serial chain, and so were the
// copies when one after another went through the block (14 us each, 18.5 ms for
// 50 levels at p = 5).
//
// The levels run in batches [l0, l1): the sum stops after the first level whose
// contribution is below the threshold (a cubic cell's after about six), and
// the kernels of the later batches return at once when *stop is set.
constexpr int kLatticeCopies = 26;

__global__ void __launch_bounds__(32 * kLatticeCopies) k_lattice_moments(int p, int l0, int l1,
                                                                         const int* __restrict__ stop,
                                                                         const double* __restrict__ root_mom,
                                                                         const Box9 H, double* __restrict__ S) {
    extern __shared__ double sh[];
    if (*stop) return;
    const int nq = nT(p), P1 = p + 1;
    double* src = sh;
    double* part = src + nq;                  // copies x nq
    double* e = part + kLatticeCopies * nq;   // scaled powers d^u / u! per copy and axis
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
        const double v = l0 > 0 ? S[(size_t)(l0 - 1) * nq + q] : (q == 0 ? 0.0 : root_mom[q]);
        src[q] = v;
        if (l0 == 0) S[q] = v;
    }
    double three_l = 1.0;
    for (int l = 1; l < l0; ++l) three_l *= 3.0;
    for (int l = max(l0, 1); l < l1; ++l) {
        three_l *= 3.0;  // 3^l, exact
        if (threadIdx.x < 3 * kLatticeCopies) {
            const int ax = threadIdx.x % 3;
            int k = threadIdx.x / 3;
            if (k >= 13) ++k;  // skip a = 0 (index 13 of the 27 in i,j,k order)
            const int ai = k / 9 - 1, aj = (k / 3) % 3 - 1, ak = k % 3 - 1;
            // d_aijk = matmul(H, a 3^l) / 3 (fmm.F90:920-923)
            const double v = __dadd_rn(__dadd_rn(__dmul_rn(H.h[ax], ai * three_l), __dmul_rn(H.h[3 + ax], aj * three_l)),
                                       __dmul_rn(H.h[6 + ax], ak * three_l));
            const double d = __ddiv_rn(v, 3.0);
            double pw = 1.0, fact = 1.0;
            for (int u = 0; u <= p; ++u) {
                e[threadIdx.x * P1 + u] = pw / fact;
                pw *= d;
                fact *= (double)(u + 1);
            }
        }
        __syncthreads();
        const int c = threadIdx.x >> 5;
        const double* ec = e + 3 * c * P1;
        for (int t = threadIdx.x & 31; t < nq; t += 32) {
            const int tx = comp_x(t), ty = comp_y(t), tz = comp_z(t), to = tx + ty + tz;
            double acc = 0.0;
            for (int so = 0; so <= to; ++so)
                for (int sx = min(so, tx); sx >= 0; --sx)
                    for (int sy = min(so - sx, ty); sy >= 0; --sy) {
                        const int sz = so - sx - sy;
                        if (sz > tz) continue;
                        acc += ec[tx - sx] * ec[P1 + ty - sy] * ec[2 * P1 + tz - sz] * src[pidx(sx, sy, sz)];
                    }
            part[c * nq + t] = acc;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < nq; q += blockDim.x) {
            double v = src[q];
            for (int k = 0; k < kLatticeCopies; ++k) v += part[k * nq + q];
            src[q] = v;
            S[(size_t)l * nq + q] = v;
        }
        // (the next level's powers touch neither src nor part)
    }
}

// Level l (1 .. L): the 702 copies of S_(l-1) at H (3^l a + 3^(l-1) b),
// a != 0 and b in {-1,0,1}^3, evaluated at the root centre like the
// reference's multipole_field call (tensors at R = the copy's position,
// src/fmm.F90:929-943).  Block (l-1, slice) sums a slice of the copies;
// partial sums go to C ((L x slices) x nq).  In exact mode the tensors are
// evaluated at R 2^-k (k ~ l log2 3, an exact scaling) and the moments and
// results rescaled by the matching powers of two, so the recursion's r^-(4p+1)
// does not underflow at the far levels; ref mode follows the reference's
// closed form unscaled.
constexpr int kLatticeSlices = 16;  // (the order of the copies' sum)

__global__ void k_lattice_m2l(int p, int l0, const int* __restrict__ stop, int ref, const double* __restrict__ S,
                              const Box9 H,
                              const int32_t* __restrict__ term_off, const uchar4* __restrict__ term_abc,
                              const double* __restrict__ term_c, double* __restrict__ C) {
    extern __shared__ double smem[];
    if (*stop) return;
    const int nq = nT(p), N = 2 * p, nqT = nT(N);
    int* comp = reinterpret_cast<int*>(smem);
    double* base = smem + (nqT + 1) / 2 + 1;
    const int nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per_warp = 2 * nqT + nq + 5 * (N + 1);
    double* red = base + nw * per_warp;  // nw x nq
    double* TA = base + wib * per_warp;
    double* TB = TA + nqT;
    double* ms = TB + nqT;
    double* gsh = ms + nq;
    double* yp = gsh + (N + 1);
    double* zp = yp + (N + 1);
    double* ir = zp + (N + 1);
    fill_comp(comp, nqT);
    const int l = l0 + blockIdx.x + 1, slice = blockIdx.y;
    const int ksc = ref ? 0 : (int)floor(l * 1.5849625007211563);  // log2(3)
    const double* Sl = S + (size_t)(l - 1) * nq;
    for (int s = lane; s < nq; s += 32) {
        const double v = Sl[s];
        ms[s] = ldexp(((order_of(s) + 1) % 2) ? -v : v, -ksc * order_of(s));  // (-1)^(|s|+1) M'_s 2^(-k|s|)
    }
    __syncthreads();
    double three_l = 1.0;
    for (int k = 0; k < l; ++k) three_l *= 3.0;
    const double three_lm = three_l / 3.0;
    int fcomp[kMaxNPL];
#pragma unroll
    for (int r = 0; r < kMaxNPL; ++r) fcomp[r] = (lane + 32 * r < nq) ? comp[lane + 32 * r] : 0;
    double acc[kMaxNPL];
#pragma unroll
    for (int r = 0; r < kMaxNPL; ++r) acc[r] = 0.0;
    for (int k = slice * nw + wib; k < 26 * 27; k += kLatticeSlices * nw) {
        int ka = k / 27, kb = k % 27;
        if (ka >= 13) ++ka;  // skip a = 0 (index 13 of the 27 in i,j,k order)
        const int ai = ka / 9 - 1, aj = (ka / 3) % 3 - 1, ak = ka % 3 - 1;
        const int bi = kb / 9 - 1, bj = (kb / 3) % 3 - 1, bk = kb % 3 - 1;
        double pos[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const double da = __dadd_rn(__dadd_rn(__dmul_rn(H.h[ax], ai * three_l), __dmul_rn(H.h[3 + ax], aj * three_l)),
                                        __dmul_rn(H.h[6 + ax], ak * three_l));
            const double db = __dadd_rn(__dadd_rn(__dmul_rn(H.h[ax], bi * three_lm), __dmul_rn(H.h[3 + ax], bj * three_lm)),
                                        __dmul_rn(H.h[6 + ax], bk * three_lm));
            pos[ax] = ldexp(__dadd_rn(da, db), -ksc);
        }
        double* T = warp_tensor(pos[0], pos[1], pos[2], N, ref, comp, TA, TB, gsh, yp, zp, ir, term_off, term_abc,
                                term_c, lane);
#pragma unroll
        for (int r = 0; r < kMaxNPL; ++r) {
            if (lane + 32 * r < nq) {
                const int fx = cx_(fcomp[r]), fy = cy_(fcomp[r]), fz = cz_(fcomp[r]);
                double a = 0.0;
                for (int s = 0; s < nq; ++s) {
                    const int cs = comp[s];
                    a += ms[s] * T[pidx(cx_(cs) + fx, cy_(cs) + fy, cz_(cs) + fz)];
                }
                acc[r] += a;
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < kMaxNPL; ++r)
        if (lane + 32 * r < nq) red[wib * nq + lane + 32 * r] = acc[r];
    __syncthreads();
    for (int f = threadIdx.x; f < nq; f += blockDim.x) {
        double v = 0.0;
        for (int w = 0; w < nw; ++w) v += red[w * nq + f];
        C[((size_t)(l - 1) * kLatticeSlices + slice) * nq + f] = ldexp(v, -ksc * (order_of(f) + 1));
    }
}

// Adds the levels' contributions to the root's local expansion in order and
// stops after the first level whose contribution (without its first
// component) has a norm below tol, as the reference does (fmm.F90:944-950);
// levels_used receives the number of levels added.
__global__ void k_lattice_apply(int nq, int l0, int l1, const double* __restrict__ C, double* __restrict__ loc_root,
                                double tol, int* levels_used, int* stop_flag) {
    __shared__ double lev[kMaxNPL * 32];
    __shared__ int stop;
    const int lane = threadIdx.x;
    if (*stop_flag) return;
    int used = l0;
    for (int l = l0; l < l1; ++l) {
        for (int f = lane; f < nq; f += 32) {
            double v = 0.0;
            for (int sl = 0; sl < kLatticeSlices; ++sl) v += C[((size_t)l * kLatticeSlices + sl) * nq + f];
            lev[f] = v;
            loc_root[f] += v;
        }
        __syncwarp();
        if (lane == 0) {
            // NORM2 as the scaled sum of squares
            double scale = 0.0, ssq = 1.0;
            for (int f = 1; f < nq; ++f) {
                const double v = lev[f];
                if (v != 0.0) {
                    const double ax = fabs(v);
                    if (scale < ax) {
                        const double t = scale / ax;
                        ssq = 1.0 + (ssq * t) * t;
                        scale = ax;
                    } else {
                        const double t = ax / scale;
                        ssq = ssq + t * t;
                    }
                }
            }
            stop = (scale * sqrt(ssq) < tol) ? 1 : 0;
        }
        __syncwarp();
        ++used;
        if (stop) break;
    }
    if (lane == 0) {
        *levels_used = used;
        *stop_flag = stop;
    }
}

// Surface term of the periodic sum (src/fmm.F90:954-979), on the field in
// sorted order: phi-column += 4 pi (D . x) / 3V + 2 pi tr(Q) / 3V and the
// order-1 columns += 4 pi D / 3V, with D and tr(Q) the root's dipole and
// quadrupole trace.  Ref mode keeps the reference's constant for pi and its
// cofactor expansion of the volume; exact mode the true ones.
__global__ void k_dipole_fix(int64_t n, int f, const double* __restrict__ sx, const double* __restrict__ sy,
                             const double* __restrict__ sz, const double* __restrict__ root_mom, const Box9 H,
                             int ref, double* __restrict__ fs) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    auto h = [&](int i, int j) { return H.h[(j - 1) * 3 + (i - 1)]; };  // h(i, j), column-major
    double vol;
    if (ref)
        vol = h(1, 1) * (h(2, 2) * h(3, 3) - h(2, 3) * h(3, 2)) - h(1, 2) * (h(2, 1) * h(3, 3) - h(2, 3) * h(3, 1)) +
              h(1, 3) * (h(1, 2) * h(3, 2) - h(2, 2) * h(3, 1));
    else
        vol = h(1, 1) * (h(2, 2) * h(3, 3) - h(2, 3) * h(3, 2)) - h(1, 2) * (h(2, 1) * h(3, 3) - h(2, 3) * h(3, 1)) +
              h(1, 3) * (h(2, 1) * h(3, 2) - h(2, 2) * h(3, 1));
    const double pi = ref ? 3.14159265359 : 3.141592653589793;
    const double dx = root_mom[1], dy = root_mom[2], dz = root_mom[3];
    // raw second moments are 2! times the scaled ones
    const double tr = 2.0 * root_mom[4] + 2.0 * root_mom[7] + 2.0 * root_mom[9];
    const double dot = dx * sx[k] + dy * sy[k] + dz * sz[k];
    fs[k] = fs[k] + 4.0 * pi * dot / (3.0 * vol) + 2.0 * pi * tr / (3.0 * vol);
    if (f >= 1) {
        const double c = 4.0 * pi / (3.0 * vol);
        fs[(size_t)1 * n + k] += c * dx;
        fs[(size_t)2 * n + k] += c * dy;
        fs[(size_t)3 * n + k] += c * dz;
    }
}

int launch_periodic_lattice(Workspace& ws, const TreeDev& t, int p, int f, const Modes& md, const Box9& H,
                            double* d_fs, int* d_levels, cudaStream_t st) {
    constexpr int L = 50;  // the reference's limit of levels
    const int nq = nT(p), N = 2 * p, nqT = nT(N);
    const int ref = md.coef_mode == 0 ? 1 : 0;
    if (ref) FMM_TRY(ensure_ref_terms(ws, N, st));
    FMM_TRY(ws.lattice.ensure(sizeof(double) * ((size_t)L * nq + (size_t)L * kLatticeSlices * nq) + sizeof(int)));
    double* S = ws.lattice.as<double>();
    double* C = S + (size_t)L * nq;
    int* stop = reinterpret_cast<int*>(C + (size_t)L * kLatticeSlices * nq);
    FMM_CUDA_TRY(cudaMemsetAsync(stop, 0, sizeof(int), st));
    const double* root_mom = ws.mom.as<double>();  // the root is node 0
    const size_t sm_mom = sizeof(double) * ((size_t)(1 + kLatticeCopies) * nq + 3 * kLatticeCopies * (p + 1));
    FMM_TRY(set_smem((const void*)k_lattice_moments, sm_mom));
    const int per_warp = 2 * nqT + nq + 5 * (N + 1);
    const int nw = (int)std::max<size_t>(1, std::min<size_t>(4, (100 * 1024) / (sizeof(double) * (per_warp + nq))));
    const size_t sm = comp_bytes(nqT) + sizeof(double) * nw * (per_warp + nq);
    FMM_TRY(set_smem((const void*)k_lattice_m2l, sm));
    // batches of levels: cubic cells stop within the first, skewed ones run all
    constexpr int kFirst = 8;
    for (int l0 = 0; l0 < L; l0 = l0 == 0 ? kFirst : L) {
        const int l1 = l0 == 0 ? kFirst : L;
        count_launches(3);
        k_lattice_moments<<<1, 32 * kLatticeCopies, sm_mom, st>>>(p, l0, l1, stop, root_mom, H, S);
        k_lattice_m2l<<<dim3(l1 - l0, kLatticeSlices), 32 * nw, sm, st>>>(p, l0, stop, ref, S, H,
                                                                           ws.term_off.as<int32_t>(),
                                                                           ws.term_abc.as<uchar4>(),
                                                                           ws.term_c.as<double>(), C);
        k_lattice_apply<<<1, 32, 0, st>>>(nq, l0, l1, C, ws.loc.as<double>(), 1.0e-8, d_levels, stop);
    }
    count_launches(1);
    k_dipole_fix<<<grid_for(t.n, 256), 256, 0, st>>>(t.n, f, ws.sx.as<double>(), ws.sy.as<double>(),
                                                      ws.sz.as<double>(), root_mom, H, ref, d_fs);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

}  // namespace fmm
